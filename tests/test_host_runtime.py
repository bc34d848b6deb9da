"""What the host side does around its launches, on a simulated CUDA runtime
(tests/hostsim): the order of streams, and arrays built and freed."""
import os
import subprocess
import sys

import pytest

import hostsim
from ctl_b200 import _lib as L


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return hostsim.build(str(tmp_path_factory.mktemp("hostsim")))


@pytest.fixture
def sim(library):
    s = hostsim.Sim(library)
    yield s
    s.close()


@pytest.mark.parametrize("answers", [[1000, 1 << 30], [1000] * 3 + [1 << 30], [1 << 30, 1000], [1 << 30]])
@pytest.mark.parametrize("views", [5, 40, 100])
def test_a_host_result_comes_from_one_loop_ordered_after_its_array(sim, answers, views):
    """Up-sampled projections into host memory, in chunks on two streams, while the free
    memory changes between any two looks at it: one loop serves the whole call, and no
    chunk reads cells that its stream is not ordered after."""
    v, _ = sim.volume()
    sim.clear()
    sim.free_answers(answers + [answers[-1]] * 20)
    assert sim.project(v, sim.settings(volume_upsampling=2), views=views, host=True) == L.OK
    launches = sim.projections()
    assert sum(p[1] for p in launches) == views
    assert {p[0] for p in launches} == {hostsim.GATHER if answers[0] == 1000 else hostsim.SEGMENTS_UP}
    assert all(p[4] in ("-", "ok") for p in launches)
    assert len({p[2] for p in launches}) == (2 if views >= 8 else 1)


@pytest.mark.parametrize("kw,loop,build", [({}, hostsim.SEGMENTS, "build_cells"),
                                           (dict(kernel=L.KERNEL_PAIRS), hostsim.PAIRS, "build_pairs"),
                                           (dict(volume_upsampling=2), hostsim.SEGMENTS_UP, "build_cells")])
@pytest.mark.parametrize("host", [False, True])
def test_an_array_whose_build_failed_is_not_kept(sim, kw, loop, build, host):
    """The launch that fills a derived array fails once, after its allocation: the call
    fails, or is served without the array where the gather loop can; the memory is given
    back, and the next call builds the array before it reads it."""
    v, _ = sim.volume()
    used = sim.memory_used()
    sim.clear()
    sim.fail(build)
    up = "volume_upsampling" in kw
    assert sim.project(v, sim.settings(**kw), host=host) == (L.OK if up else L.ERR_CUDA)
    assert {p[0] for p in sim.projections()} == ({hostsim.GATHER} if up else set())
    assert sim.memory_used() == used
    sim.clear()
    assert sim.project(v, sim.settings(**kw), host=host) == L.OK
    assert sim.record()[0].startswith(build) and sim.record()[0].endswith("done")
    assert {(p[0], p[4]) for p in sim.projections()} == {(loop, "ok")}
    assert sim.memory_used() > used


@pytest.mark.parametrize("reader", ["noalloc", "captured", "plan", "project", "stream"])
@pytest.mark.parametrize("upsampling", [1, 2])
def test_autotuning_leaves_arrays_that_captured_work_may_read(sim, reader, upsampling):
    """A no-allocation call, a call during capture of its stream and a plan leave launches
    behind that may be replayed for as long as the volume lives: autotuning, won by the
    gather loop, does not free the cells that they read.  After a plain call it does."""
    import ctypes as C
    v, _ = sim.volume()
    s = sim.settings(volume_upsampling=upsampling)
    assert sim.project(v, s) == L.OK  # builds the cells
    cells = sim.projections()[-1][3]
    if reader == "noalloc":
        assert sim.project(v, s, call="ctlcu_project_noalloc") == L.OK
        assert sim.projections()[-1][3:5] == (cells, "ok")
    elif reader == "captured":
        sim.lib.sim_capturing(1)
        assert sim.project(v, s) == L.OK
        sim.lib.sim_capturing(0)
        assert sim.projections()[-1][3] == cells
    elif reader == "stream":  # a plain call, still running on a stream of the caller's
        assert sim.project(v, s, stream=sim.lib.sim_stream()) == L.OK
        assert sim.projections()[-1][3:5] == (cells, "ok")
    elif reader == "plan":
        if upsampling != 1:
            pytest.skip("plans take volumes as they are")
        q = L.Request(v, sim.device(96), sim.device(256), 1, 1, 8, 8)
        plan = C.c_void_p()
        assert sim.lib.ctlcu_plan_create(sim.h, C.byref(q), 1, C.byref(s), C.byref(plan)) == L.OK
    for loop in (hostsim.SEGMENTS, hostsim.PAIRS):
        sim.lib.sim_mode_ms(loop, 9.0)
    sim.lib.sim_mode_ms(hostsim.GATHER, 1.0)
    loop = C.c_int()
    assert sim.lib.ctlcu_autotune(sim.h, v, C.byref(sim.settings()), sim.device(96), 1, 1, 8, 8, 0, C.byref(loop),
                                  None) == L.OK
    assert loop.value == L.KERNEL_GATHER
    freed = any(line == f"freed_array {cells}" for line in sim.record())
    assert freed == (reader in ("project", "stream")) and sim.count("freed_while_read") == 0
    sim.clear()
    assert sim.project(v, sim.settings(volume_upsampling=2), call="ctlcu_project_noalloc") == L.OK
    assert sim.projections()[0][4] == ("-" if freed else "ok")
    if reader == "plan":
        sim.lib.ctlcu_plan_destroy(plan)


@pytest.mark.parametrize("upsampling", [2, 3])
def test_an_upsampled_call_leaves_a_capture_elsewhere_alone(sim, upsampling):
    """While another thread captures a stream of its own in the global mode, cudaMalloc
    fails and ends that capture; an up-sampled call does not need it."""
    v, _ = sim.volume()
    sim.clear()
    sim.lib.sim_foreign_capture(1)
    assert sim.project(v, sim.settings(volume_upsampling=upsampling)) == L.OK
    assert sim.lib.sim_unsafe_calls() == 0
    assert {(p[0], p[4]) for p in sim.projections()} == {(hostsim.SEGMENTS_UP, "ok")}
    sim.lib.sim_foreign_capture(0)


@pytest.mark.parametrize("kernel", [L.KERNEL_CELLS, L.KERNEL_PAIRS])
def test_sub_rays_get_lanes_whatever_the_number_of_views(sim, kernel):
    """A view's sub-rays are summed across lanes, or one after the other, which rounds
    differently: the choice goes by the detector alone, so that a view is the same in a
    call of any length, in a chunk of a host result and in a no-allocation call.  Every
    launch keeps its blocks within a grid's limit."""
    v, _ = sim.volume()
    s = sim.settings(rays_per_pixel=(4, 4), kernel=kernel)
    sim.lib.sim_capacity(1 << 45)
    C, R = 1024, 1024
    tiles = (4 * C // 16) * (4 * R // 8)
    for views, kw in ((1, {}), (600, {}), (40000, {}), (600, dict(host=True)), (600, dict(call="ctlcu_project_noalloc"))):
        sim.clear()
        assert sim.project(v, s, views=views, channels=C, rows=R, **kw) == L.OK
        launches = sim.projections()
        assert {p[5] for p in launches} == {(2, 2)} and sum(p[1] for p in launches) == views
        assert all((p[1] + 1) // 2 * tiles <= 0x7fffffff for p in launches)


@pytest.mark.parametrize("form", [L.PLAN_PERSISTENT, L.PLAN_GRIDS])
@pytest.mark.parametrize("requests,lanes", [(40, (2, 2)), (500, (0, 0))])
def test_a_batch_too_large_with_a_lane_per_sub_ray_goes_without(sim, form, requests, lanes):
    """500 views of 1024^2 with 4 x 4 rays a pixel: with a lane for every ray their warps do
    not fit the 32 bits of the persistent launch's counter, one after the other they do."""
    import ctypes as C
    v, _ = sim.volume()
    s = sim.settings(rays_per_pixel=(4, 4))
    q = (L.Request * requests)()
    pm, out = sim.device(96 * 24), sim.device(4 * 24 << 20)
    for r in q:
        r.volume, r.pmats, r.out, r.n_views, r.n_modules, r.channels, r.rows = v, pm, out, 24, 1, 1024, 1024
    plan = C.c_void_p()
    assert sim.lib.ctlcu_plan_create_form(sim.h, q, requests, C.byref(s), form, C.byref(plan)) == L.OK, sim.error()
    if form == L.PLAN_GRIDS:
        assert {p[5] for p in sim.projections()} == {lanes}
    sim.lib.ctlcu_plan_destroy(plan)
    sim.clear()
    assert sim.lib.ctlcu_project_batch(sim.h, q, requests, C.byref(s), None) == L.OK
    assert {p[5] for p in sim.projections()} == {(2, 2)}  # one grid per request: these fit


@pytest.mark.parametrize("devices,free,loop", [
    ((0, 1), (1 << 40, 1 << 40), hostsim.SEGMENTS_UP), ((0, 1), (1 << 40, 1000), hostsim.GATHER),
    ((0, 1), (1000, 1 << 40), hostsim.GATHER), ((0, 1), (1000, 1000), hostsim.GATHER),
    ((0, 0), (1 << 40, 0), hostsim.SEGMENTS_UP), ((0, 0), (1600000, 0), hostsim.GATHER)])
@pytest.mark.parametrize("views", [2, 33])
def test_a_group_projects_all_its_views_with_one_loop(sim, devices, free, loop, views):
    """Whether an up-sampled volume's cells are built goes by the free memory, which
    differs from device to device: the group decides once for all its devices, as the
    result has to be a one-device call's bit for bit.  (A 16^3 volume's cells take 231
    KB, a quarter of 1.6 MB holds one context's and not two.)"""
    import ctypes as C
    import numpy as np
    for d, f in enumerate(free):
        sim.lib.sim_free_of_device(d, f)
    g = C.c_void_p()
    assert sim.lib.ctlcu_group_create((C.c_int * 2)(*devices), 2, C.byref(g)) == L.OK
    vol, P, out = np.zeros(16 ** 3, np.float32), np.zeros(12 * views), np.zeros(64 * views, np.float32)
    for up in (2, 1, 2):
        sim.clear()
        s = sim.settings(volume_upsampling=up)
        assert sim.lib.ctlcu_group_project_volume(g, C.byref(sim.desc((16, 16, 16))), vol.ctypes.data, C.byref(s),
                                                  P.ctypes.data, views, 1, 8, 8, out.ctypes.data) == L.OK
        launches = sim.projections()
        assert sum(p[1] for p in launches) == views
        assert {p[0] for p in launches} == ({loop} if up == 2 else {hostsim.SEGMENTS})
        assert {p[4] for p in launches} <= {"ok", "-"}
    assert sim.lib.ctlcu_group_destroy(g) == L.OK


@pytest.mark.parametrize("what", ["volume", "result", "cells", "pairs"])
@pytest.mark.parametrize("held", [False, True])
def test_memory_that_only_speeds_up_is_given_back_when_it_is_needed(sim, what, held):
    """Cells that up-sampled calls built (they run without) do not stand in the way of what
    a call needs: a new volume, a result, another loop's array.  Cells that replayed work
    may read stay, and so do those that a loop cannot do without."""
    a, _ = sim.volume((40, 40, 40))
    needed, _ = sim.volume((16, 16, 16))
    assert sim.project(needed, sim.settings()) == L.OK
    assert sim.project(a, sim.settings(volume_upsampling=2)) == L.OK
    cells = sim.projections()[-1][3]
    b, _ = sim.volume((30, 30, 30))
    if held:
        assert sim.project(a, sim.settings(volume_upsampling=2), call="ctlcu_project_noalloc") == L.OK
    sim.lib.sim_capacity(sim.lib.sim_used() + 20000)
    used = sim.memory_used()
    sim.clear()
    if what == "volume":
        rc = sim.volume((30, 30, 30))[1]
    elif what == "result":
        rc = sim.project(needed, sim.settings(), views=100, channels=100, rows=30, host=True)
    else:
        rc = sim.project(b, sim.settings(kernel=L.KERNEL_PAIRS if what == "pairs" else L.KERNEL_CELLS))
    assert rc == (L.ERR_OUT_OF_MEMORY if held else L.OK), sim.error()
    freed = [line.split()[1] for line in sim.record() if line.startswith("freed_array")]
    assert freed == ([] if held else [cells]) and sim.count("freed_while_read") == 0
    assert sim.memory_used() == used if held else sim.memory_used() != used
    sim.clear()
    assert sim.project(a, sim.settings(volume_upsampling=2)) == L.OK
    # (a result in host memory has left the device again)
    assert sim.projections()[-1][4] == ("ok" if held or what == "result" else "-")


_NO_MEMORY = """
import sys
import ctypes as C
import numpy as np
import hostsim
from ctl_b200 import _lib as L
nth, towards = int(sys.argv[2]), sys.argv[3]
sim = hostsim.Sim(sys.argv[1])
data = np.arange(128 ** 3 * 4 // 3, dtype=np.float32)[:128 ** 3].reshape(128, 128, 128)
v, _ = sim.volume()
if towards == "device":
    sim.lib.sim_fail_new_after_pin(nth)
    h = C.c_uint64()
    make = lambda: sim.lib.ctlcu_volume_create(sim.h, C.byref(sim.desc((128, 128, 128))), data.ctypes.data, 0, C.byref(h))
    rc = make()
    sim.lib.sim_stop_failing_new()
    assert make() == L.OK
else:
    sim.lib.sim_fail_new_after_pin(nth)
    rc = sim.project(v, sim.settings(), views=9, channels=512, rows=512, host=True)
    sim.lib.sim_stop_failing_new()
    assert sim.project(v, sim.settings(), views=9, channels=512, rows=512, host=True) == L.OK
assert rc in (L.OK, L.ERR_OUT_OF_MEMORY), rc
print("status", rc)
"""


@pytest.mark.parametrize("towards", ["device", "host"])
def test_copies_by_threads_do_not_end_the_process_without_host_memory(library, towards):
    """One allocation of the copying code after another fails (its lists, a thread's start
    among running threads): the call gives a status, the next one works."""
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([hostsim.ROOT, os.path.dirname(hostsim.HERE)]))
    statuses = []
    for nth in range(1, 9):
        r = subprocess.run([sys.executable, "-c", _NO_MEMORY, library, str(nth), towards], env=env, capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, (nth, r.stderr[-400:])
        statuses.append(int(r.stdout.split()[-1]))
    assert L.ERR_OUT_OF_MEMORY in statuses


def test_new_volumes_do_not_ask_for_the_free_memory(library):
    """cudaMemGetInfo can take longer than a small projection: a context asks when it is
    made, and again only when up-sampled calls have built more cells than that allows.
    What is freed is allowed again."""
    s = hostsim.Sim(library, free_at_creation=6 * 1000000)  # an eighth: three 16^3 volumes' cells of 231 KB
    try:
        before = s.lib.sim_info_calls()
        for _ in range(20):
            v, _ = s.volume()
            s.clear()
            assert s.project(v, s.settings(volume_upsampling=2)) == L.OK
            assert {p[0] for p in s.projections()} == {hostsim.SEGMENTS_UP}
            assert s.lib.ctlcu_volume_release(s.h, v) == L.OK
        assert s.lib.sim_info_calls() == before
        loops = []
        s.free_answers([1000, 1200000])  # the fourth volume's look, and the fifth's
        for _ in range(5):
            v, _ = s.volume()
            s.clear()
            assert s.project(v, s.settings(volume_upsampling=2)) == L.OK
            loops += [p[0] for p in s.projections()]
        assert loops == [hostsim.SEGMENTS_UP] * 3 + [hostsim.GATHER, hostsim.SEGMENTS_UP]
        assert s.lib.sim_info_calls() == before + 2
    finally:
        s.close()
