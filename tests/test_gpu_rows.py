"""tace_rows_segment_add against the same sums on the CPU, bit for bit: targets with none, one and many rows, row lengths around
a block, both element sizes."""
import pytest
import torch

from tace_b200 import lib as _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("row_len", [1, 3, 64, 257])
def test_segment_add(dtype, row_len):
    lib, gen = _lib.load(), torch.Generator().manual_seed(row_len)
    counts = [0, 1, 2, 26, 1, 0, 7]
    n = sum(counts)
    src, dst = torch.randn(n, row_len, generator=gen, dtype=dtype), torch.randn(11, row_len, generator=gen, dtype=dtype)
    order, targets = torch.randperm(n, generator=gen), torch.randperm(11, generator=gen)[: len(counts)]
    ptr = torch.tensor([0] + counts).cumsum(0)
    ref = dst.clone()
    for t, i in enumerate(targets.tolist()):
        for j in range(int(ptr[t]), int(ptr[t + 1])):
            ref[i] += src[order[j]]
    dev = [x.cuda() for x in (src, order, targets, ptr, dst)]
    _lib.check(lib.tace_rows_segment_add(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), dev[3].data_ptr(), len(counts), row_len,
                                         src.element_size(), dev[4].data_ptr(), torch.cuda.current_stream().cuda_stream), "tace_rows_segment_add")
    assert torch.equal(dev[4].cpu(), ref)
