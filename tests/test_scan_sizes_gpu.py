"""The row-pointer scan of the format conversions on both sides of the size from which one CTA scans
the block sums first (8,192 blocks of 2,048 rows)."""
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import dev

pytestmark = pytest.mark.gpu
LINE = 8192 * 2048


@pytest.mark.parametrize("n_rows", [LINE - 2, LINE - 1, LINE, LINE + 1, LINE + 2049, 3 * LINE + 5])
def test_conversion_row_pointers(n_rows):
    gen = torch.Generator(device=dev()).manual_seed(n_rows)
    filled = torch.rand(n_rows, generator=gen, device=dev()) < 0.03
    filled[-1] = True
    rp = torch.zeros(n_rows + 1, dtype=torch.int32, device=dev())
    rp[1:] = torch.cumsum(filled, 0)
    nnz = int(rp[-1])
    ci = torch.randint(0, 1000, (nnz,), generator=gen, device=dev(), dtype=torch.int32)
    v = torch.rand(nnz, generator=gen, device=dev())
    vrp, vci, vval = A.csr_to_vcsr4(rp, ci, v)  # one entry: one block of four slots
    assert torch.equal(vrp, 4 * rp) and vci.numel() == 4 * nnz
    rp2, ci2, v2, _ = A.csr_to_rowpair(rp, ci, v)
    assert torch.equal(rp2[::2], rp[::2]) and int(rp2[-1]) == nnz  # a pair holds its two rows' entries
    A.sync_status()
