"""The x pass on the GPU: its transforms at the edges of its thread layouts
(4 to 256 threads per row, odd and even butterfly counts, one to three
stages, partial row tiles) against float64, and the ratio's two routes (the
usual range and the general one) against each other."""
import numpy as np
import pytest

import deconwolf_b200 as dw
from tests.helpers import gauss_psf, poisson_image

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


# half lengths: one stage (2..16), two, three; M = L / first radix odd and even
@pytest.mark.parametrize("L", [2, 3, 5, 7, 9, 16, 21, 25, 27, 45, 49, 75, 125, 135, 189, 343, 375, 512, 625, 729,
                               1000, 1029, 1323, 1715, 2048])
def test_transforms_match_float64(L):
    import torch
    n = 2 * L
    if dw.tune_plans(dw.PLAN_X, L) == []:
        pytest.skip("no transform of this length")
    for N, P in ((1, 1), (37, 2)):  # 37 rows: a partial tile for every tile height
        shape = (P, N if N == 1 else 35, n)
        g = torch.Generator(device="cuda").manual_seed(L)
        x = torch.randn(shape, generator=g, device="cuda")
        out = torch.empty(shape[:2] + (L + 1, 2), device="cuda")
        dw.fft_r2c_device(x.data_ptr(), shape, out.data_ptr())
        ref = torch.fft.rfftn(x.double())
        # every stage rounds: a few eps per factor of two of the length
        tol = 4 * EPS * max(2.0, np.log2(x.numel()))
        got = torch.view_as_complex(out.double())
        assert float((got - ref).norm() / ref.norm()) < tol
        spec = torch.view_as_real(ref.to(torch.complex64)).contiguous()
        y = torch.empty(shape, device="cuda")
        dw.fft_c2r_device(spec.data_ptr(), shape, y.data_ptr())
        assert float((y.double() / x.numel() - x.double()).norm() / x.double().norm()) < tol


def test_ratio_routes_agree():
    """Values scaled by 2^64 leave the ratio pass's usual range; every step of
    SHB with a fixed background scales exactly, and both routes round the
    quotient correctly, so the results agree bit for bit.  The traces' terms
    have logarithms of other code: a unit in the last place each."""
    psf = gauss_psf((7, 9, 11), (1.3, 1.6, 1.9), seed=71, jitter=0.2)
    im = poisson_image((9, 33, 41), psf, seed=71, bg=30.0, npts=20)
    im[:, ::7, ::5] = 0.0
    s = np.float32(2.0 ** 64)
    a = dw.run_method(im, psf, n_iter=6, bg=1.0)
    b = dw.run_method(im * s, psf, n_iter=6, bg=float(s))
    np.testing.assert_array_equal(b.out, a.out * s)
    np.testing.assert_allclose(b.trace / s, a.trace, rtol=1e-5)
