"""Restoring into flat-start jobs, whose first convolution is a shortcut as
long as the estimate is the constant; the flat start with a PSF larger than
its job, which has no shortcut."""
import numpy as np
import pytest

import deconwolf_b200 as dw
from tests.helpers import gauss_psf, poisson_image, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture
def heuristic_plans():
    dw.tune_set_mode(dw.TUNE_OFF)
    dw.tune_clear()
    yield
    dw.tune_set_mode(dw.TUNE_MEASURE)
    dw.tune_clear()


@pytest.mark.parametrize("method", ["shb", "rl"])
def test_a_flat_job_takes_other_estimates_and_its_own_back(method, heuristic_plans):
    """(On this image the shortcut and the transformed constant differ in the
    last bits, so which of them a job takes shows.)"""
    psf = gauss_psf((7, 9, 11), (1.3, 1.6, 1.9), seed=4, jitter=0.2)
    im = poisson_image((12, 40, 44), psf, seed=4, bg=60.0, npts=20)

    def job(start):
        j = dw.Job(im.shape, psf.shape, method=method, n_iter=8, iter_type=dw.ITER_FIXED, start=start)
        j.setup(im, psf)
        return j

    def finish(j):
        j.step(1 << 30)
        return j.result()

    flat, ident, j = job(dw.START_FLAT), job(dw.START_IDENTITY), job(dw.START_FLAT)
    of_flat, of_ident = flat.snapshot(), ident.snapshot()
    ref_flat, ref_ident = finish(flat), finish(ident)
    assert not np.array_equal(ref_flat.out, ref_ident.out)
    j.restore(of_ident)
    r = finish(j)
    np.testing.assert_array_equal(r.out, ref_ident.out)
    np.testing.assert_array_equal(r.trace, ref_ident.trace)
    j.restore(of_flat)
    r = finish(j)
    np.testing.assert_array_equal(r.out, ref_flat.out)
    np.testing.assert_array_equal(r.trace, ref_flat.trace)
    for k in (flat, ident, j):
        k.close()


# border_quality 1: the job is M + (pM + 1) / 2, less than a PSF of 2 M and more
@pytest.mark.parametrize("method", ["shb", "rl"])
@pytest.mark.parametrize("shape,psf_shape,fits", [((3, 30, 12), (3, 9, 31), False), ((3, 12, 31), (3, 31, 9), False),
                                                  ((2, 25, 19), (9, 9, 9), False), ((4, 30, 19), (7, 9, 9), True)])
def test_the_first_step_from_a_constant(method, shape, psf_shape, fits, heuristic_plans):
    """The flat start's first convolution against the transformed one, which
    the same constant takes in a job of another start.  A PSF larger than its
    job is not all in its transfer function, so its sum does not give the
    first convolution: both jobs transform."""
    psf = gauss_psf(psf_shape, tuple(0.3 * s for s in psf_shape), seed=5, jitter=0.2)
    for ax, w in enumerate(dw.plan_size(shape, psf_shape, 1)[0][::-1]):
        # voxels that wrap onto the same place hold the same value
        v = np.moveaxis(psf, ax, 0)
        if len(v) > w:
            v[w:] = v[: len(v) - w]
    im = poisson_image(shape, gauss_psf((1, 5, 5), (1, 1.5, 1.5)), seed=5, bg=60.0, npts=8)

    def job(start):
        j = dw.Job(im.shape, psf.shape, method=method, n_iter=4, border_quality=1, iter_type=dw.ITER_FIXED, start=start)
        j.setup(im, psf)
        return j

    flat, other = job(dw.START_FLAT), job(dw.START_IDENTITY)
    other.restore(flat.snapshot())
    flat.step(1 << 30)
    other.step(1 << 30)
    a, b = flat.result(), other.result()
    assert fits == all(p <= w for p, w in zip(psf_shape, a.work[::-1]))
    if fits:  # the constant's rounding, about 2^-24, and the transforms'
        assert rel_l2(a.out, b.out) < 1e-5
        np.testing.assert_allclose(a.trace, b.trace, rtol=1e-5)
    else:
        np.testing.assert_array_equal(a.out, b.out)
        np.testing.assert_array_equal(a.trace, b.trace)
    flat.close()
    other.close()
