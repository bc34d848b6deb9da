"""The tiled post-projection kernels at the edges of their tiles: Poisson noise (1024
pixels of a view per warp, a stack of the pixels whose first draw needs the full test)."""
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
