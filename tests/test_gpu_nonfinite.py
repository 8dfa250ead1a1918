"""A PSF without any finite value (a zero PSF divided by its sum) has no
maximum to move to the origin: refused, with nothing read outside it."""
import numpy as np
import pytest

import deconwolf_b200 as dw
from tests.helpers import gauss_psf, poisson_image

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("psf_shape", [(1, 1, 1), (3, 3, 3), (7, 9, 11), (9, 9, 9)])
@pytest.mark.parametrize("bq", [2, 1, 0])
@pytest.mark.parametrize("value", [np.nan, -np.inf])
def test_psf_without_finite_values(psf_shape, bq, value):
    good = gauss_psf((7, 9, 11), (1.3, 1.6, 1.9), seed=7, jitter=0.2)
    im = poisson_image((12, 40, 44), good, seed=7, bg=60.0, npts=20)
    before = dw.run_method(im, good, n_iter=4, border_quality=bq)
    bad = np.full(psf_shape, value, dtype=np.float32)
    with pytest.raises(dw.DwcuError):
        dw.run_method(im, bad, n_iter=4, border_quality=bq)
    if bq == 2:
        with pytest.raises(dw.DwcuError):
            dw.run_slabs(im, bad, parts=2, n_iter=4)
    after = dw.run_method(im, good, n_iter=4, border_quality=bq)
    np.testing.assert_array_equal(after.out, before.out)
