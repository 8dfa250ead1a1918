"""Single-plane jobs (their convolution is one kernel along y) and the
standalone transforms on volumes at odd addresses and ragged row lengths."""
import numpy as np
import pytest

import deconwolf_b200 as dw
from oracle import pyoracle as po
from tests.helpers import gauss_psf, poisson_image, rel_l2

pytestmark = pytest.mark.gpu


# y lengths of one, two and three stages; the shortest and a long one
@pytest.mark.parametrize("N", [1, 3, 6, 27, 90, 500, 1500])
@pytest.mark.parametrize("method,bq", [("shb", 2), ("rl", 2), ("shb", 1), ("rl", 0)])
def test_plane_jobs_match_the_oracle(N, method, bq):
    psf = gauss_psf((1, min(7, 2 * ((N + 1) // 2) - 1), 9), (1.0, 1.5, 1.9), seed=N, jitter=0.2)
    im = poisson_image((1, N, 38), psf, seed=N, bg=60.0, npts=10)
    g = dw.run_method(im, psf, method=method, n_iter=8, border_quality=bq)
    kw = dict(work=g.work) if bq == 2 else {}
    r = po.deconvolve(im, psf, method=method, n_iter=8, border_quality=bq, **kw)
    assert rel_l2(g.out, r.out) < 1e-4
    assert np.max(np.abs(g.trace - r.trace) / np.abs(r.trace)) < 1e-5


def test_one_part_of_a_plane_equals_the_whole_job():
    psf = gauss_psf((1, 7, 9), (1.0, 1.5, 1.9), seed=5, jitter=0.2)
    im = poisson_image((1, 90, 70), psf, seed=5, bg=60.0, npts=10)
    a = dw.run_method(im, psf, n_iter=8)
    b = dw.run_slabs(im, psf, parts=1, n_iter=8)
    np.testing.assert_array_equal(b.out, a.out)


@pytest.mark.parametrize("shape", [(1, 1, 4), (3, 5, 10), (7, 12, 54), (1, 30, 64), (16, 1, 30), (2, 3840, 20)])
def test_transforms_at_odd_addresses(shape):
    """Real volumes that start at an odd float (through a staging copy) give
    the bits of aligned ones; rows of any even length are taken as they lie."""
    import torch
    P, N, M = shape
    n = P * N * M
    g = torch.Generator(device="cuda").manual_seed(M)
    pad = torch.randn(n + 4, generator=g, device="cuda")
    outs, backs = [], []
    for o in (0, 1, 2):
        buf = torch.empty(n + 4, device="cuda")
        x = buf[o: o + n]
        x.copy_(pad[:n])
        X = torch.full((P, N, M // 2 + 1, 2), float("nan"), device="cuda")
        dw.fft_r2c_device(x.data_ptr(), shape, X.data_ptr())
        outs.append(X.cpu().numpy())
        ybuf = torch.full((n + 4,), 7.0, device="cuda")
        dw.fft_c2r_device(X.data_ptr(), shape, ybuf.data_ptr() + 4 * o)
        yb = ybuf.cpu().numpy()
        backs.append(yb[o: o + n])
        assert np.all(yb[:o] == 7.0) and np.all(yb[o + n:] == 7.0)
    ref = np.fft.rfftn(pad[:n].cpu().numpy().astype(np.float64).reshape(shape))
    got = outs[0][..., 0] + 1j * outs[0][..., 1]
    tol = 4 * 2.0 ** -24 * max(2.0, np.log2(n))
    assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref)
    for a, b in zip(outs[1:], backs[1:]):
        np.testing.assert_array_equal(a, outs[0])
        np.testing.assert_array_equal(b, backs[0])
