"""Host arrays through the staged copies (pitched rows and whole pieces),
page-locked ones through the driver's, and two callers at once: the bits of
the same call on device buffers."""
import threading

import numpy as np
import pytest

import deconwolf_b200 as dw
from tests.helpers import gauss_psf

pytestmark = pytest.mark.gpu

SHAPES = [(31, 260, 301), (3, 601, 701), (20, 256, 256)]  # 4 to 10 MB; rows of the first two are pitched


def _inputs(shape):
    rng = np.random.default_rng(shape[2])
    return rng.poisson(60.0, shape).astype(np.float32), gauss_psf((3, 9, 9), (1.0, 1.6, 1.9), seed=3, jitter=0.2)


def _on_device(im, psf):
    import torch
    d, k, out = torch.from_numpy(im).cuda(), torch.from_numpy(psf).cuda(), torch.empty(im.shape, device="cuda")
    torch.cuda.synchronize()
    r = dw.run_method_device(d.data_ptr(), k.data_ptr(), out.data_ptr(), im.shape, psf.shape, n_iter=4)
    return out.cpu().numpy(), r.trace


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("locked", [False, True])
def test_host_arrays_equal_device_buffers(shape, locked):
    import torch
    im, psf = _inputs(shape)
    ref, trace = _on_device(im, psf)
    out = np.full(shape, -1.0, dtype=np.float32)
    if locked:
        im, out = torch.from_numpy(im).pin_memory().numpy(), torch.from_numpy(out).pin_memory().numpy()
    r = dw.run_method(im, psf, n_iter=4, out=out)
    np.testing.assert_array_equal(r.out, ref)
    np.testing.assert_array_equal(r.trace, trace)


def test_two_callers_at_once():
    import torch
    cases = [_inputs(s) for s in SHAPES[:2]]
    refs = [_on_device(*c)[0] for c in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    jobs = [dw.Job(im.shape, psf.shape, n_iter=4) for im, psf in cases]
    got = [[], []]

    def work(i):
        jobs[i].set_stream(streams[i].cuda_stream)
        for _ in range(5):
            jobs[i].setup(*cases[i])
            jobs[i].step(4)
            got[i].append(jobs[i].result().out)

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in th]
    [t.join(120) for t in th]
    assert not any(t.is_alive() for t in th)
    for j in jobs:
        j.close()
    for i in range(2):
        assert len(got[i]) == 5
        for g in got[i]:
            np.testing.assert_array_equal(g, refs[i])
