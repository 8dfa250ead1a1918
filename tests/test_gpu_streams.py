"""A job that changes its stream: its pooled memory is given back only when
both streams are done with it."""
import numpy as np
import pytest

import deconwolf_b200 as dw

pytestmark = pytest.mark.gpu


def test_a_stopped_job_leaves_no_read_back_behind():
    """A REL job has one iteration queued ahead when its rule stops it, with
    the error's copy into a page-locked slot behind it.  The slot goes to the
    next job, so the copy has to have landed, on whichever stream."""
    import torch
    im = torch.full((60, 768, 768), 50.0, device="cuda")
    im[30, 300:400, 300:400] += 500.0
    psf = torch.zeros((9, 9, 9), device="cuda")
    psf[4, 4, 4] = 0.5
    psf += 0.5 / psf.numel()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        j = dw.Job(tuple(im.shape), tuple(psf.shape), iter_type=dw.ITER_REL, err_rel=0.2, maxiter=50)
        j.set_stream(a.cuda_stream)
        j.setup(im.data_ptr(), psf.data_ptr(), on_device=True)
        j.step(1 << 30)
        j.set_stream(b.cuda_stream)
        j.close()
        drained = a.query()
        torch.cuda.synchronize()
        assert drained
