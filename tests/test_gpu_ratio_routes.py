"""The ratio's branch-free route takes no value that the general one treats
otherwise, and both give the same on the values they share."""
import numpy as np
import pytest

import deconwolf_b200 as dw
from tests.helpers import gauss_psf, poisson_image

pytestmark = pytest.mark.gpu


def _inputs():
    psf = gauss_psf((7, 9, 11), (1.3, 1.6, 1.9), seed=71, jitter=0.2)
    im = poisson_image((9, 33, 41), psf, seed=71, bg=30.0, npts=20)
    im[:, ::7, ::5] = 0.0
    return im, psf


@pytest.mark.parametrize("method", ["shb", "rl"])
def test_nan_adds_nothing_to_the_divergence(method):
    """A NaN projection is not positive: the I-divergence skips it (dw.c:1514),
    in an iteration that forms a ratio and in one that forms the error alone."""
    im, psf = _inputs()
    j = dw.Job(im.shape, psf.shape, method=method, n_iter=3, iter_type=dw.ITER_FIXED)
    j.setup(im, psf)
    j.step(1)
    s = j.snapshot()
    for k in ("x", "x_prev"):
        if s[k] is not None:
            s[k] = np.full_like(s[k], np.nan)
    j.restore(s)
    j.step(1 << 30)
    trace = j.result().trace
    j.close()
    assert trace[0] > 0
    np.testing.assert_array_equal(trace[1:], 0.0)


@pytest.mark.parametrize("method", ["shb", "rl"])
@pytest.mark.parametrize("metric", [dw.METRIC_IDIV, dw.METRIC_MSE])
def test_routes_agree_for_every_op(method, metric):
    """Values scaled by 2^54 leave the branch-free route's range (2^60), and a
    power of two scales every step exactly, so the estimates agree bit for bit.
    The squared error's terms do too; the divergence's have logarithms of other
    code, a unit in the last place each."""
    im, psf = _inputs()
    s = np.float32(2.0 ** 54)
    assert im.max() * s > 2.0 ** 60
    kw = dict(method=method, metric=metric, n_iter=6, iter_type=dw.ITER_FIXED)
    a = dw.run_method(im, psf, bg=1.0, **kw)
    b = dw.run_method(im * s, psf, bg=float(s), **kw)
    np.testing.assert_array_equal(b.out, a.out * s)
    if metric == dw.METRIC_MSE:
        np.testing.assert_array_equal(b.trace, a.trace * s * s)
    else:
        np.testing.assert_allclose(b.trace / s, a.trace, rtol=1e-5)
