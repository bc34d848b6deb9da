"""The nearest-voxel loop on rays that its fast road must not take on trust: warps
in which some or all rays miss the volume, sources so far away that FP64 no longer
places a sample, and sums that FP32 cannot hold."""
import numpy as np
import pytest

import oracle
from _common import dequant_bf16, rel_err
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
    return rng.uniform(0.01, 0.05, shape_xyz[::-1]).astype(np.float16).astype(np.float32)


def _view(source, towards, channels, rows, pitch, sdd=1200.0):
    source, towards = np.asarray(source, float), np.asarray(towards, float)
    up = np.array([0.0, 0.0, 1.0]) if abs(towards[2] - source[2]) < 100 else np.array([1.0, 0.0, 0.0])
    R = G.camera_rotation(towards - source, up)
    K = G.intrinsic(sdd, pitch, pitch, (channels - 1) / 2, (rows - 1) / 2)
    return G.normalized(G.compose(K, R, source))


@pytest.mark.parametrize("storage", [L.F32, L.BF16, L.F16])
@pytest.mark.parametrize("sampling", [0.05, 0.3, 0.8, 0.81])
def test_rays_that_miss_add_nothing(ctx, storage, sampling):
    """Views of a small volume in which a few, most and all rays pass beside it, and
    one whose source has the volume behind it.  Bar: zero where the oracle has no
    sample in the volume, else 1e-4 (the volume is exact in F16; BF16 rounds it first)."""
    vol = _volume((13, 11, 12), 3)
    if storage == L.BF16:
        vol = dequant_bf16(vol)
    voxel, C, R = (1.0, 1.1, 1.2), 67, 43
    P = np.stack([_view((900, 31, 7), (0, 0, 0), C, R, 0.4), _view((900, 31, 7), (0, 9, 4), C, R, 1.3),
                  _view((900, 31, 7), (0, 300, 0), C, R, 1.3), _view((31, 900, 7), (0, 0, 90), C, R, 1.3),
                  _view((60, 3, 2), (900, 31, 7), C, R, 1.3), _view((7, 31, 900), (5, 0, 0), C, R, 0.4)])[:, None]
    want, _ = oracle.project_fp64(vol, voxel, P, C, R, ray_sampling=sampling, interpolate=False)
    some = (want > 0).mean(axis=(1, 2, 3))
    assert 0.05 < some[1] < 0.3 and some[0] > 0.3 and some[2] == some[3] == some[4] == 0
    v = ctx.volume(VoxelVolume(vol, voxel), storage)
    try:
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64, L.ACCUM_FP32):
            got = ctx.project(v, P, C, R, Settings(ray_sampling=sampling, accum=accum, interpolate=False))
            np.testing.assert_array_equal(got[want == 0], 0.0)
            assert rel_err(got, want).max() <= 1e-4
    finally:
        v.release()


def _inner_positions(P, channels, rows, n, voxel, sampling):
    """Voxel positions of the second and the last but one sample of each ray that the
    face tests let in, in FP64 as the ray setup forms them (one voxel size)."""
    inc = sampling * voxel
    qr, src = (x.ravel() for x in oracle.view_setup(P[None, None]))
    up = np.array([[qr[9], qr[10], qr[11]], [0.0, qr[12], qr[13]], [0.0, 0.0, qr[14]]])
    A, out = np.linalg.solve(up, qr[:9].reshape(3, 3).T), []
    s, k, n = src / voxel, -0.5 * np.asarray(n, float), np.asarray(n, float)
    for y in range(rows):
        for x in range(channels):
            d = A @ np.array([x, y, 1.0])
            d *= inc / voxel / np.sqrt(d @ d)
            with np.errstate(all="ignore"):
                hits = [l for l, face in [((c[a] - s[a]) / d[a], a) for c in (k, k + n) for a in range(3)]
                        if all(k[i] - 0.01 <= s[i] + l * d[i] <= k[i] + n[i] + 0.01 for i in range(3) if i != face)]
            i0, i1 = (np.floor(max(min(hits), 0.0)), np.floor(max(hits)) + 1) if hits else (0, 0)
            if i1 - i0 < 2:
                continue  # two samples, both taken on their own
            base = (s - k) + i0 * d
            out += [base + d, base + (i1 - i0 - 1) * d]
    return np.array(out)


@pytest.mark.parametrize("far", [1e8, 1e16, 1e17, 1e18, 1e25])
@pytest.mark.parametrize("storage", [L.F32, L.F16])
def test_sources_beyond_what_fp64_places(ctx, far, storage):
    """Any finite matrix is served.  From 1e16 voxels on the positions are off by more
    than the array's border, samples may land anywhere, and those outside the volume read
    zeros.  The volume is 1 everywhere: a pixel's value is its samples in the volume
    times the step, so no sum exceeds the sample count, and nothing is not a number."""
    n, voxel, C, R = (20, 18, 19), 1.0, 24, 17
    vol = np.ones(n[::-1], np.float32)
    u = np.array([0.83, 0.41, 0.37]) / np.linalg.norm([0.83, 0.41, 0.37])
    P = _view(far * u, (0, 0, 0), C, R, 1.0, sdd=far)[None, None]
    inner = _inner_positions(P[0, 0], C, R, n, voxel, 0.3)
    beyond = max((-inner).max(), (inner - np.array(n)).max()) if len(inner) else 0.0
    assert beyond < 0.02 if far < 1e10 else far != 1e17 or beyond > 4  # 1e17 reaches past the border
    v = ctx.volume(VoxelVolume(vol, (voxel,) * 3), storage)
    try:
        st = dict(ray_sampling=0.3, interpolate=False)
        samples = ctx.count_samples(v, P, C, R, Settings(**st))
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64):
            got = ctx.project(v, P, C, R, Settings(accum=accum, **st))
            assert np.isfinite(got).all() and got.min() >= 0.0
            assert got.sum() <= 0.3 * samples * (1 + 1e-5)
            if far < 1e10:
                want, _ = oracle.project_fp64(vol, (voxel,) * 3, P, C, R, **st)
                assert rel_err(got, want).max() <= 0.02  # a sample on a face may count to either side
    finally:
        v.release()


@pytest.mark.parametrize("storage", [L.F32, L.F16])
@pytest.mark.parametrize("sampling", [0.02, 0.3, 0.8, 0.81])
def test_fp64_accumulator_sums_the_samples_without_fp32_rounding(ctx, storage, sampling):
    """Voxels of both signs, full mantissas, whose sums along a ray nearly cancel.  The
    oracle and an FP64 accumulator differ by the order of at most a few hundred FP64
    additions, below 1e-12 of the sum of magnitudes, and each rounds its result to FP32
    once: one unit in the last place of FP32 (1.2e-7).  A product or a sum of two voxels
    rounded to FP32 shows as 1e-8 of the sum of magnitudes, which exceeds the result by
    a factor of several here.  A sample in a neighbouring voxel shows as a hundredth
    of it.  Pixels with a sample on a face, either of whose voxels is right, are those
    whose oracle value jumps under a shift of 1e-9 pixel."""
    rng = np.random.default_rng(17)
    vol = rng.uniform(0.5, 1.0, (24, 26, 28)) * np.where(np.indices((24, 26, 28)).sum(0) % 2, 1.0, -1.0)
    vol = vol.astype(np.float16 if storage == L.F16 else np.float32).astype(np.float32)
    voxel, C, R = (1.0, 1.1, 1.2), 45, 31
    P = np.stack([_view((900, 31, 7), (0, 0, 0), C, R, 0.9), _view((7, 31, 900), (0, 0, 0), C, R, 0.9),
                  _view((500, 600, 400), (0, 0, 0), C, R, 0.9)])[:, None]
    st = dict(ray_sampling=sampling, interpolate=False)
    want, _ = oracle.project_fp64(vol, voxel, P, C, R, **st)
    total, _ = oracle.project_fp64(np.abs(vol), voxel, P, C, R, **st)
    assert np.median(np.abs(want[total > 0]) / total[total > 0]) < 0.2
    ties = np.zeros(want.shape, bool)
    for shift in ((1e-9, 1e-9), (-1e-9, -1e-9), (1e-9, -1e-9), (-1e-9, 1e-9)):
        moved = np.eye(3)
        moved[:2, 2] = shift
        near, _ = oracle.project_fp64(vol, voxel, moved @ P, C, R, **st)
        ties |= np.abs(near - want) > 1e-6 * total
    assert ties.mean() < 0.01
    v = ctx.volume(VoxelVolume(vol, voxel), storage)
    try:
        got = ctx.project(v, P, C, R, Settings(accum=L.ACCUM_FP64, **st))
        err = np.abs(got.astype(float) - want)
        assert (err <= 1.2e-7 * np.abs(want) + 1e-12 * total)[~ties].all()
    finally:
        v.release()


@pytest.mark.parametrize("storage", [L.F32, L.F16])
@pytest.mark.parametrize("sampling", [0.3, 0.4, 0.5, 0.7, 0.75, 0.76])
def test_a_view_is_the_same_in_calls_of_any_size(ctx, storage, sampling):
    """The loop goes by the number of rays: a view alone (segments up to 0.4), in a call
    of 48 thousand rays (up to 0.55) and of 338 thousand (up to 0.75), on the device and in
    chunks into host memory, has the same bits, with any accumulator."""
    import torch
    vol = np.random.default_rng(31).uniform(0.01, 0.05, (33, 37, 41)).astype(np.float32)
    if storage == L.F16:
        vol = vol.astype(np.float16).astype(np.float32)
    C, R, V = 72, 67, 70
    P = G.circular_flat(V, 300.0, 600.0, G.FlatDetector(C, R, 1.1, 1.1), rng=np.random.default_rng(1), jitter_mm=0.5,
                        tilt_deg=0.2)
    assert C * R < 148 * 256 <= 10 * C * R < 148 * 2048 <= V * C * R
    v = ctx.volume(VoxelVolume(vol, (1.0, 1.1, 1.2)), storage)
    try:
        for accum in (L.ACCUM_KAHAN, L.ACCUM_FP64, L.ACCUM_FP32):
            st = Settings(ray_sampling=sampling, interpolate=False, accum=accum)
            whole = ctx.project(v, P, C, R, st)
            for n in (1, 10):
                np.testing.assert_array_equal(ctx.project(v, P[20:20 + n].copy(), C, R, st), whole[20:20 + n])
            out = torch.empty(whole.shape, device="cuda")
            ctx.project(v, torch.from_numpy(P).cuda(), C, R, st, out=out)
            ctx.sync()
            np.testing.assert_array_equal(out.cpu().numpy(), whole)
        want, _ = oracle.project_fp64(vol, (1.0, 1.1, 1.2), P[:3], C, R, ray_sampling=sampling, interpolate=False)
        assert rel_err(whole[:3], want).max() <= 1e-4
    finally:
        v.release()
