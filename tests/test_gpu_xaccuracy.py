"""The x transforms' rounding error, each direction by itself, against
float64.

A transform of X points has log2(X) factors of two.  Each contributes a sum
and a product by a root of unity that is itself rounded to float, which
together stay below one unit of rounding (2^-24) in the root mean square as
long as the root is no worse than a table value or two; the factors' errors
are independent and add in squares.  So the relative error is at most
2^-24 sqrt(log2 X).  Roots made as long chains of products of one table value
break this: their errors add up along the chain (1.3 to 1.6 at the lengths
below that have radices of 9 to 16 behind the first stage).
"""
import numpy as np
import pytest

import deconwolf_b200 as dw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [2, 9, 14, 21, 25, 27, 50, 96, 125, 147, 210, 300, 375, 392, 420, 448, 486, 560, 630,
                               810, 896, 1080, 1120, 1350, 1764, 1890, 2048])
def test_rounding_error_of_each_direction(L):
    import torch
    X, n = 2 * L, max(32, 8192 // L)
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn((n, X), generator=g, device="cuda")
    spec = torch.view_as_real(torch.fft.rfft(x.double()).to(torch.complex64)).contiguous()
    spec[:, 0, 1] = spec[:, L, 1] = 0.0
    out, y = torch.empty_like(spec), torch.empty_like(x)
    torch.cuda.synchronize()
    for i in range(n):  # a row a call: no other axis adds its error
        dw.fft_r2c_device(x[i].data_ptr(), (1, 1, X), out[i].data_ptr())
        dw.fft_c2r_device(spec[i].data_ptr(), (1, 1, X), y[i].data_ptr())
    tol = 2.0 ** -24 * np.sqrt(np.log2(X))
    fwd = torch.fft.rfft(x.double())
    inv = torch.fft.irfft(torch.view_as_complex(spec.double()), n=X, norm="forward")
    assert float((torch.view_as_complex(out.double()) - fwd).norm() / fwd.norm()) < tol
    assert float((y.double() - inv).norm() / inv.norm()) < tol
