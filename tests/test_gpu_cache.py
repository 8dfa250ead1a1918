"""What the library keeps between calls, and gives back."""
import pytest

import deconwolf_b200 as dw

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def test_transforms_of_many_sizes_keep_a_bounded_share():
    """Work space of sizes too far apart to share a block: kept up to a
    thirty-second of the device together, given back by release_cache."""
    import torch
    dw.release_cache()
    planes = [180, 256, 360, 500, 700, 1000]  # of 1024 x 1024: 0.8 to 4.2 GB of work space each
    x = torch.zeros(max(planes) * 1024 * 1024, device="cuda")
    out = torch.empty(max(planes) * 1024 * 513 * 2, device="cuda")
    dw.fft_r2c_device(x.data_ptr(), (4, 1024, 1024), out.data_ptr())  # kernels and tables of the rows
    torch.cuda.synchronize()
    dw.release_cache()
    free, total = torch.cuda.mem_get_info()
    for p in planes:
        dw.fft_r2c_device(x.data_ptr(), (p, 1024, 1024), out.data_ptr())
        kept = free - torch.cuda.mem_get_info()[0]
        assert kept <= total / 32 + 256 * MIB  # (and the kernels and tables of the lengths)
    # a block within the share is kept: the same transform again allocates nothing
    before = torch.cuda.mem_get_info()[0]
    dw.fft_r2c_device(x.data_ptr(), (planes[-1], 1024, 1024), out.data_ptr())
    assert torch.cuda.mem_get_info()[0] == before
    dw.release_cache()
    assert free - torch.cuda.mem_get_info()[0] <= 256 * MIB


def _ring_mapped():
    """Whether the staging buffers (32 MiB, page-locked) are mapped in this process."""
    with open("/proc/self/maps") as f:
        for line in f:
            a, b = (int(v, 16) for v in line.split(None, 1)[0].split("-"))
            if b - a == 32 * MIB and "rw-s" in line and line.rstrip().endswith("/dev/zero (deleted)"):
                return True
    return False


@pytest.mark.parametrize("device", [-1, 0])
def test_release_cache_gives_the_host_buffers_back(device):
    """With no device block cached too: here the only one is in use."""
    import numpy as np
    dw.release_cache()
    if _ring_mapped():
        pytest.skip("another mapping looks like the staging buffers")
    im = np.full((32, 300, 300), 5.0, dtype=np.float32)
    psf = np.ones((3, 3, 3), dtype=np.float32)
    j = dw.Job(im.shape, psf.shape, n_iter=2)
    j.setup(im, psf)
    if not _ring_mapped():
        pytest.skip("page-locked memory is not mapped as expected here")
    dw.release_cache(device)
    assert not _ring_mapped()
    j.step(2)
    r = j.result()  # staged again
    assert _ring_mapped() and np.isfinite(r.out).all()
    j.close()
    dw.release_cache()
    assert not _ring_mapped()
