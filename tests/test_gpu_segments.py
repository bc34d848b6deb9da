"""The cell loop that sums a ray's samples cell by cell, at the sizes where it can
go wrong: volumes of one voxel to several hundred along the rays (no sample in the
box, one window of samples, several), rays along an axis or nearly so, partial
warps, and sampling steps on both sides of the line between this loop and the
sample-by-sample one.  Bar: the parity bar of the projector (1e-4 of the value or
of a thousandth of the maximum, tests/_common.py)."""
import numpy as np
import pytest

import oracle
from _common import rel_err
from ctl_b200 import _lib as L
from ctl_b200 import geometry as G
from ctl_b200.projector import Context, Settings, VoxelVolume

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


def _volume(shape_xyz, seed):
    rng = np.random.default_rng(seed)
    return (rng.uniform(0.01, 0.05, shape_xyz[::-1]) * (rng.random(shape_xyz[::-1]) < 0.8)).astype(np.float32)


def _axis_views(channels, rows, pitch, tilt):
    """Views from +x, +y and (nearly) +z, `tilt` rad off each axis."""
    out = []
    for axis in range(3):
        d = np.full(3, tilt)
        d[axis] = 1.0
        up = np.array([0.0, 0.0, 1.0]) if axis < 2 else np.array([1.0, 0.0, 0.0])
        R = G.camera_rotation(-d, up)
        K = G.intrinsic(1200.0, pitch, pitch, (channels - 1) / 2, (rows - 1) / 2)
        out.append(G.normalized(G.compose(K, R, 900.0 * d / np.linalg.norm(d))))
    return np.stack(out)[:, None]


@pytest.mark.parametrize("sampling", [0.05, 0.3, 0.6, 0.61, 1.0, 2.5])
@pytest.mark.parametrize("shape,voxel", [((1, 1, 1), (30.0, 30.0, 30.0)), ((2, 3, 127), (20.0, 15.0, 1.0)),
                                         ((43, 42, 5), (1.0, 1.0, 7.0)), ((300, 6, 5), (0.5, 6.0, 7.0))])
@pytest.mark.parametrize("tilt", [0.0, 1e-7, 0.31])
def test_cell_sums_match_the_oracle(ctx, shape, voxel, sampling, tilt):
    vol = _volume(shape, 3)
    C, R = 37, 21
    P = _axis_views(C, R, 1.9, tilt)
    want, _ = oracle.project_fp64(vol, voxel, P, C, R, ray_sampling=sampling)
    v = ctx.volume(VoxelVolume(vol, voxel))
    try:
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64):
            got = ctx.project(v, P, C, R, Settings(ray_sampling=sampling, accum=accum, kernel=L.KERNEL_CELLS))
            assert want.max() > 0
            assert rel_err(got, want).max() <= 1e-4
    finally:
        v.release()


def test_unusable_matrix_and_partial_warps_leave_the_other_pixels_alone(ctx):
    """A singular view between good ones in one block: its pixels are 0, the others as without it."""
    vol = _volume((20, 18, 16), 5)
    P = _axis_views(11, 7, 4.0, 0.2)
    bad = P.copy()
    bad[1] = 0.0
    v = ctx.volume(VoxelVolume(vol, (2.0, 2.0, 2.0)))
    try:
        good = ctx.project(v, P, 11, 7, Settings())
        out = np.empty_like(good)
        with pytest.raises(L.CtlcuError) as e:
            ctx.project(v, bad, 11, 7, Settings(), out=out)
        assert e.value.status == L.ERR_SINGULAR_GEOMETRY
        np.testing.assert_array_equal(out[1], 0.0)
        np.testing.assert_array_equal(out[[0, 2]], good[[0, 2]])
    finally:
        v.release()


@pytest.mark.parametrize("shape,voxel", [((1, 1, 1), (24.0, 24.0, 24.0)), ((17, 12, 9), (2.0, 2.5, 3.0)),
                                         ((33, 5, 40), (1.0, 4.0, 1.0))])
@pytest.mark.parametrize("factor", [2, 3, 7])
@pytest.mark.parametrize("storage", [L.F32, L.F16])
def test_upsampled_volume_read_from_the_cells(ctx, shape, voxel, factor, storage):
    """Virtual replication through the cell array: against the oracle, and against
    the gather loop that reads the replicated grid voxel by voxel."""
    vol = _volume(shape, 7).astype(np.float16).astype(np.float32)  # the same in both storages
    C, R = 29, 18
    P = _axis_views(C, R, 1.7, 0.13)
    for sampling in (0.3, 1.0):
        st = dict(ray_sampling=sampling, volume_upsampling=factor)
        want, _ = oracle.project_fp64(vol, voxel, P, C, R, ray_sampling=sampling, upsampling=factor)
        v = ctx.volume(VoxelVolume(vol, voxel), storage)
        try:
            before = v.nbytes
            gather = ctx.project(v, P, C, R, Settings(kernel=L.KERNEL_GATHER, **st))
            assert v.nbytes == before
            got = ctx.project(v, P, C, R, Settings(**st))
            assert v.nbytes > before  # the cells were built and read
            assert rel_err(got, want).max() <= 1e-4
            assert rel_err(gather, want).max() <= 1e-4
        finally:
            v.release()


def test_upsampled_calls_take_no_array_from_a_memory_budget():
    """With a budget set the up-sampled call runs as it does without any derived array."""
    vol = _volume((20, 20, 20), 9)
    P = _axis_views(16, 16, 4.0, 0.1)
    with Context(0) as c:
        v = c.volume(VoxelVolume(vol, (1.0, 1.0, 1.0)))
        want = c.project(v, P, 16, 16, Settings(volume_upsampling=2, kernel=L.KERNEL_GATHER))
        used = c.memory_used()
        c.set_memory_budget(used + 1000)
        got = c.project(v, P, 16, 16, Settings(volume_upsampling=2))
        assert c.memory_used() == used
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("shape,voxel", [((1, 1, 1), (30.0, 30.0, 30.0)), ((2, 3, 127), (20.0, 15.0, 1.0)),
                                         ((300, 6, 5), (0.5, 6.0, 7.0)), ((64, 60, 58), (1.0, 1.1, 1.2))])
@pytest.mark.parametrize("sampling", [0.01, 0.3, 1.0, 40.0])
@pytest.mark.parametrize("tilt", [0.0137, 0.31])
def test_nearest_voxel_sums_match_the_oracle(ctx, shape, voxel, sampling, tilt):
    """Every sample in the voxel that FP64 positions put it in: one sample in a
    neighbouring voxel would miss the bar on these random volumes.  The central ray
    passes through the centre of the grid, where at some steps a sample lies exactly
    on a face and either voxel is right: such pixels are those whose oracle value
    jumps when the detector moves by 1e-9 pixel."""
    vol = _volume(shape, 11)
    C, R = 33, 19
    P = _axis_views(C, R, 1.9, tilt)
    want, _ = oracle.project_fp64(vol, voxel, P, C, R, ray_sampling=sampling, interpolate=False)
    ties = np.zeros(want.shape, bool)
    for shift in ((1e-9, 1e-9), (-1e-9, -1e-9), (1e-9, -1e-9), (-1e-9, 1e-9)):
        moved = np.eye(3)
        moved[:2, 2] = shift
        near, _ = oracle.project_fp64(vol, voxel, moved @ P, C, R, ray_sampling=sampling, interpolate=False)
        ties |= rel_err(near, want) > 1e-6
    assert ties[:, :, np.arange(R) != R // 2].sum() == 0 and ties.sum() <= 3
    v = ctx.volume(VoxelVolume(vol, voxel))
    try:
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64):
            got = ctx.project(v, P, C, R, Settings(ray_sampling=sampling, accum=accum, interpolate=False))
            assert rel_err(got, want)[~ties].max() <= 1e-4
    finally:
        v.release()


@pytest.mark.parametrize("where", ["one voxel", "corner block", "diagonal", "empty", "nan"])
@pytest.mark.parametrize("upsampling", [1, 3])
@pytest.mark.parametrize("sampling", [0.3, 1.0])
def test_zero_voxels_outside_the_object_change_nothing(ctx, where, upsampling, sampling):
    """The loops start and end at the bounds of the voxels that are not zero: single
    voxels, blocks at a corner, along a diagonal, nothing at all, and a NaN."""
    n = (27, 22, 31)
    vol = np.zeros(n[::-1], np.float32)
    if where == "one voxel":
        vol[13, 0, 26] = 0.04
    elif where == "corner block":
        vol[25:, 17:, :6] = _volume((6, 5, 6), 3)
    elif where == "diagonal":
        for i in range(22):
            vol[i, i, 21 - i] = 0.03
    elif where == "nan":
        vol[4, 5, 6] = np.nan
    C, R = 45, 37
    P = np.concatenate([_axis_views(C, R, 1.5, t) for t in (0.0, 0.21, 1.0)])
    got = ctx.project_volume(VoxelVolume(vol, (1.0, 1.2, 0.9)), P, C, R,
                             Settings(ray_sampling=sampling, volume_upsampling=upsampling))
    if where == "empty":
        np.testing.assert_array_equal(got, 0.0)
        return
    if where == "nan":  # seen by the rays that pass it, and by no others
        seen, _ = oracle.project_fp64(np.nan_to_num(vol, nan=1.0), (1.0, 1.2, 0.9), P, C, R, ray_sampling=sampling,
                                      upsampling=upsampling)
        assert np.isnan(got[seen > 1e-3]).all() and not np.isnan(got[seen == 0]).any() and (seen > 1e-3).any()
        return
    want, _ = oracle.project_fp64(vol, (1.0, 1.2, 0.9), P, C, R, ray_sampling=sampling, upsampling=upsampling)
    assert want.max() > 0 and rel_err(got, want).max() <= 1e-4


@pytest.mark.parametrize("rays", [(2, 1), (1, 4), (4, 4), (2, 4), (3, 2), (4, 8)])
@pytest.mark.parametrize("kernel,upsampling", [(L.KERNEL_CELLS, 1), (L.KERNEL_PAIRS, 1), (L.KERNEL_AUTO, 2)])
def test_sub_rays_on_lanes_of_their_own(ctx, rays, kernel, upsampling):
    """1, 2 or 4 rays a side get a lane each, other counts run one after the other:
    detectors that leave partial patches and tiles, and every launch shape the same bits."""
    vol = _volume((18, 17, 23), 13)
    C, R = 19, 11
    P = _axis_views(C, R, 2.9, 0.17)
    want, _ = oracle.project_fp64(vol, (1.0, 1.1, 1.2), P, C, R, rays=rays, upsampling=upsampling)
    st = dict(rays_per_pixel=list(rays), kernel=kernel, volume_upsampling=upsampling)
    v = ctx.volume(VoxelVolume(vol, (1.0, 1.1, 1.2)))
    try:
        got = ctx.project(v, P, C, R, Settings(**st))
        assert rel_err(got, want).max() <= 1e-4
        for block, views, lanes in ((128, 1, 4), (512, 4, 8), (128, 2, 8)):
            other = ctx.project(v, P, C, R, Settings(block_rays=block, views_per_block=views, lanes_x=lanes, **st))
            np.testing.assert_array_equal(other, got)
    finally:
        v.release()


@pytest.mark.parametrize("upsampling,step,bits", [(1, 3 / 128, 15), (2, 3 / 128, 15), (4, 3 / 128, 15),
                                                  (2, 3 / 16, 21), (4, 3 / 16, 21)])
def test_fp64_accumulator_adds_no_rounding(ctx, upsampling, step, bits):
    """Rays along the middle rows of 3 x 3 equal rows of voxels, at steps of 3/128 or 3/16
    voxel, through whole numbers of `bits` bits: sample positions, coefficients and
    interpolants all fit FP32's 24 bits, so the value of every sample, and of every cell
    at the midpoint of its samples, is exact (at a multiple of 1/256 of a voxel and of
    1/8).  Only sums can round: four cells of 42 samples, or eight samples, need more than
    24 bits, an FP64 accumulator holds them all, and the result equals the oracle's,
    rounded to FP32 once."""
    n = (18, 36, 36)
    vol = np.random.default_rng(23).integers(0, 1 << bits, (12, 12, 18)).astype(np.float32)
    vol = vol.repeat(3, 0).repeat(3, 1)
    K = G.intrinsic(1024.0, 1.0, 1.0, 0.0, 0.0)
    P = []
    for z in range(1, n[2], 3):
        for y in range(1, n[1], 3):
            src = np.array([512.0, y + 0.5 - n[1] / 2, z + 0.5 - n[2] / 2])
            P.append(G.compose(K, G.camera_rotation(np.array([-1.0, 0.0, 0.0]), np.array([0.0, 0.0, 1.0])), src))
    P = np.stack(P)[:, None]
    st = dict(ray_sampling=step * upsampling)
    want, samples = oracle.project_fp64(vol, (1.0, 1.0, 1.0), P, 1, 1, upsampling=upsampling, **st)
    assert samples > len(P) * n[0] / step and (want > 0).all()
    v = ctx.volume(VoxelVolume(vol, (1.0, 1.0, 1.0)))
    try:
        got = ctx.project(v, P, 1, 1, Settings(volume_upsampling=upsampling, accum=L.ACCUM_FP64, unroll=8, **st))
        np.testing.assert_array_equal(got, want)
    finally:
        v.release()


@pytest.mark.parametrize("upsampling,sampling", [(2, 0.75), (3, 1.0)])
def test_upsampled_samples_are_placed_as_well_as_by_the_gather_loop(ctx, upsampling, sampling):
    """Sample by sample through the cells, over several windows of samples: the 2-norm
    error against the oracle stays below the gather loop's, which serves the same calls
    where there are no cells."""
    rng = np.random.default_rng(5)
    vol = rng.uniform(0.01, 0.05, (150, 160, 170)).astype(np.float32)
    C, R = 61, 43
    P = G.circular_flat(3, 300.0, 600.0, G.FlatDetector(C, R, 2.6, 2.6), rng=np.random.default_rng(1),
                        jitter_mm=0.5, tilt_deg=0.2)
    st = dict(ray_sampling=sampling, volume_upsampling=upsampling)
    want, _ = oracle.project_fp64(vol, (0.5, 0.5, 0.5), P, C, R, ray_sampling=sampling, upsampling=upsampling)
    seen = want > 0.01 * want.max()
    assert seen.mean() > 0.3
    v = ctx.volume(VoxelVolume(vol, (0.5, 0.5, 0.5)))
    try:
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64):
            err = {}
            for kernel in (L.KERNEL_GATHER, L.KERNEL_AUTO):
                got = ctx.project(v, P, C, R, Settings(kernel=kernel, accum=accum, **st))
                err[kernel] = np.sqrt(np.mean(((got - want)[seen] / want[seen].astype(float)) ** 2))
            assert err[L.KERNEL_AUTO] <= err[L.KERNEL_GATHER]
    finally:
        v.release()


@pytest.mark.parametrize("mask", [-3.4e38, 3.4e38, 1e34, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("sampling", [0.05, 1.0])
def test_upsampled_volumes_with_masks_give_what_the_gather_loop_gives(ctx, mask, sampling):
    """Voxels masked with the largest numbers, infinities or NaN, next to each other along
    an edge, a face and a diagonal: an up-sampled call gives the bits of the gather loop,
    which interpolates between voxels and holds no sums over eight of them.  Finite
    masks leave every sample, and an FP64 sum of them, finite."""
    vol = _volume((23, 19, 21), 29)
    for z, y, x in ((5, 5, 5), (5, 6, 6), (9, 9, 9), (9, 9, 10), (14, 12, 4), (15, 13, 5), (0, 0, 22)):
        vol[z, y, x] = mask
    C, R = 43, 31
    P = _axis_views(C, R, 0.9, 0.29)
    v = ctx.volume(VoxelVolume(vol, (0.3, 0.3, 0.3)))
    try:
        for accum in (L.ACCUM_FP64, L.ACCUM_KAHAN):
            st = dict(ray_sampling=sampling, volume_upsampling=2, accum=accum)
            want = ctx.project(v, P, C, R, Settings(kernel=L.KERNEL_GATHER, **st))
            got = ctx.project(v, P, C, R, Settings(**st))
            if np.isfinite(mask) and accum == L.ACCUM_FP64:
                assert np.isfinite(want).all() and (np.abs(want) > 1e33).any()
            np.testing.assert_array_equal(got, want)
    finally:
        v.release()
