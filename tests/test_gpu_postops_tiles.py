"""The tiled post-projection kernels at the edges of their tiles: Poisson noise (1024
pixels of a view per warp, a stack of the pixels whose first draw needs the full test)
and the spectral combine (1024 pixels of a view per block, a table of 6144 / (materials
+ 2) bins at a time, up to four materials in registers)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from ctl_b200.projector import Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("views,modules,ppm", [(1, 1, 1), (3, 1, 31), (2, 1, 1023), (2, 1, 1024), (3, 1, 1025),
                                               (2, 5, 613), (70, 3, 40)])
@pytest.mark.parametrize("photons", [40.0, 3.0e3, 2.0e4])
def test_noise_is_the_oracles_draw_for_draw(ctx, views, modules, ppm, photons):
    """Every count is the oracle's: the two differ in the last bits of FP64 functions,
    which moves a count with a probability below 1e-9 per pixel.  Counts above 1e4 are
    normal variates rounded to FP32, where such a bit may move the last place: the
    extinction log(i0 / n) then differs by 2^-23 at most, plus the same for logf."""
    rng = np.random.default_rng(ppm)
    x = rng.uniform(0.0, 4.0, (views, modules, 1, ppm)).astype(np.float32)
    i0 = (photons * (1.0 + 0.2 * np.arange(modules))).astype(np.float32)
    want, counts = oracle.poisson_noise(x, i0, 77)
    got = ctx.poisson_noise(x.copy(), i0, 77)
    inf = counts == 0
    np.testing.assert_array_equal(np.isinf(got), inf)
    assert np.abs(got[~inf] - want[~inf]).max(initial=0.0) <= 2.0 ** -22 * max(1.0, np.abs(want[~inf]).max(initial=0.0))


@pytest.mark.parametrize("materials", [1, 2, 4, 5])
@pytest.mark.parametrize("bins,views,per_view", [(1, 1, 1), (7, 3, 1023), (33, 2, 1025), (2500, 2, 130)])
def test_spectral_combine_matches_64_bits(ctx, materials, bins, views, per_view):
    """FP32 sums of `bins` positive terms: relative error at most (bins + 16) 2^-24 in the
    sum (each product and the exponential within 2 ulp, e = 0 .. 3 within 4 ulp of it),
    and the same absolutely in its logarithm."""
    import torch
    rng = np.random.default_rng(bins + materials)
    proj = rng.uniform(0.0, 1.0, (materials, views, per_view)).astype(np.float32)
    mu = rng.uniform(0.1, 3.0 / materials, (bins, materials)).astype(np.float32)
    inten = rng.uniform(10.0, 1000.0, (bins, views))
    inten[1::3] = 0.0  # skipped
    resp = rng.uniform(0.5, 1.0, bins).astype(np.float32)
    total = inten.sum(0)
    d = torch.from_numpy(proj).cuda()
    out = torch.empty((views, per_view), device="cuda")
    torch.cuda.synchronize()
    ctx._check(ctx.lib.ctlcu_spectral_combine(
        ctx.h, C.c_void_p(d.data_ptr()), materials, views, per_view, C.c_void_p(mu.ctypes.data),
        C.c_void_p(inten.ctypes.data), C.c_void_p(resp.ctypes.data), bins, C.c_void_p(total.ctypes.data),
        C.c_void_p(out.data_ptr()), None))
    e = np.einsum("bm,mvp->bvp", mu.astype(np.float64), proj.astype(np.float64))
    acc = (np.float32(inten).astype(np.float64)[:, :, None] * np.exp(-e) * resp.astype(np.float64)[:, None, None]).sum(0)
    want = np.log(np.float32(total).astype(np.float64)[:, None] / acc)
    bound = (bins + 16) * 2.0 ** -24 + 4.0 * 2.0 ** -24 * np.maximum(1.0, np.abs(want))
    assert (np.abs(out.cpu().numpy() - want) <= bound).all()
