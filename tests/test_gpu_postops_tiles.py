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


@pytest.mark.parametrize("views,modules,ppm", [(1, 1, 303104), (1, 1, 303105), (9800, 1, 31), (300, 1, 1023), (299, 1, 1025),
                                               (70, 5, 911), (2, 64, 8000), (1, 1, 3637249)])
@pytest.mark.parametrize("photons", [6.0, 3.0e3])
def test_noise_of_larger_jobs_is_the_oracles_draw_for_draw(ctx, views, modules, ppm, photons):
    """The largest job of one pixel per thread and the smallest of tiles, views that end
    within a tile, tiles of 128, 256 and 512 pixels: the bar of the test above."""
    test_noise_is_the_oracles_draw_for_draw(ctx, views, modules, ppm, photons)


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


@pytest.mark.parametrize("materials", [2, 8, 9])
@pytest.mark.parametrize("bins,views,per_view", [(5, 300, 33), (5, 300, 1024), (5, 300, 1100), (9, 700, 64), (3, 2, 20000),
                                                 (1200, 1, 257)])
def test_spectral_combine_over_small_views_and_many_materials(ctx, materials, bins, views, per_view):
    """Both numbers of pixels per thread, blocks of every size, materials in registers and
    not, more bins than a table holds, every third bin skipped: the bound of the test above."""
    test_spectral_combine_matches_64_bits(ctx, materials, bins, views, per_view)


def test_spectral_combine_without_a_live_bin(ctx):
    """No intensity in any bin: log(total / 0)."""
    import torch
    proj = torch.zeros((1, 2, 40), device="cuda")
    out = torch.empty((2, 40), device="cuda")
    mu, inten, total = np.ones((3, 1), np.float32), np.zeros((3, 2)), np.ones(2)
    torch.cuda.synchronize()
    ctx._check(ctx.lib.ctlcu_spectral_combine(
        ctx.h, C.c_void_p(proj.data_ptr()), 1, 2, 40, C.c_void_p(mu.ctypes.data), C.c_void_p(inten.ctypes.data), None, 3,
        C.c_void_p(total.ctypes.data), C.c_void_p(out.data_ptr()), None))
    assert np.isposinf(out.cpu().numpy()).all()


def test_spectral_combine_takes_more_materials_than_a_table_holds(ctx):
    """6143 materials: the exponent is a chain of as many FP32 additions of positive terms,
    within 6143 2^-24 of itself (0.5), which the logarithm passes on absolutely."""
    import torch
    M, bins, views, px = 6143, 2, 2, 40
    rng = np.random.default_rng(3)
    proj = rng.uniform(0.0, 1.0, (M, views, px)).astype(np.float32)
    mu = rng.uniform(0.0, 2.0 / M, (bins, M)).astype(np.float32)
    inten = rng.uniform(10.0, 1000.0, (bins, views))
    total = inten.sum(0)
    d = torch.from_numpy(proj).cuda()
    out = torch.empty((views, px), device="cuda")
    torch.cuda.synchronize()
    ctx._check(ctx.lib.ctlcu_spectral_combine(
        ctx.h, C.c_void_p(d.data_ptr()), M, views, px, C.c_void_p(mu.ctypes.data), C.c_void_p(inten.ctypes.data), None,
        bins, C.c_void_p(total.ctypes.data), C.c_void_p(out.data_ptr()), None))
    e = np.einsum("bm,mvp->bvp", mu.astype(np.float64), proj.astype(np.float64))
    want = np.log(total[:, None] / (inten[:, :, None] * np.exp(-e)).sum(0))
    assert np.abs(out.cpu().numpy() - want).max() <= 6143 * 2.0 ** -24 * e.max() + 1e-6
