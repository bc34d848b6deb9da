"""The nearest-voxel loop on rays that its fast road must not take on trust: warps
in which some or all rays miss the volume."""
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
