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
