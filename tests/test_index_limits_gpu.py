"""Calls with as many entries as an int counts (2^31 - 1): the kernels read ahead of the entry they
work on, and the last entries' look-ahead has to end at the last entry."""
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import dev

pytestmark = pytest.mark.gpu
NNZ = 2 ** 31 - 1


def _rowptr(*ends):
    return torch.tensor([0, *ends], dtype=torch.int32, device=dev())


def _columns():
    """Column 1 for the last three entries, else 0."""
    ci = torch.zeros(NNZ, dtype=torch.int32, device=dev())
    ci[-3:] = 1
    return ci


def test_sddmm_reads_no_column_past_the_last():
    X = torch.tensor([[1.0, 2, 3, 4], [0, 0, 0, 0], [2, 0, 1, 0]], device=dev())
    Y = torch.tensor([[1.0, 1, 1, 1], [5, 0, 7, 0]], device=dev())
    out = A.sddmm(_rowptr(5, 5, NNZ), _columns(), X, Y)
    A.sync_status()
    want = X @ Y.T
    assert out[:5].tolist() == [want[0, 0].item()] * 5
    assert out[-3:].tolist() == [want[2, 1].item()] * 3
    for lo in range(5, NNZ - 3, 1 << 28):
        assert bool((out[lo:min(lo + (1 << 28), NNZ - 3)] == want[2, 0]).all())


@pytest.mark.parametrize("name", ["nnzsplit_v4_g32_c1_ch1024", "nnzsplit_v16_g8_c1_ch128",
                                  "nnzme_v16_g8_ch1024"])
def test_entry_balanced_reads_no_entry_past_the_last(name):
    variant = A.spmm_variants(torch.bfloat16).index(name) + 1
    rp, ci = _rowptr(5, NNZ - 3, NNZ), _columns()  # the last row: three entries of column 1
    v = torch.ones(NNZ, dtype=torch.bfloat16, device=dev())
    B = torch.zeros(2, 8, dtype=torch.bfloat16, device=dev())
    B[1] = torch.arange(8)
    C = A.spmm(rp, ci, v, B, variant=variant)
    A.sync_status()
    assert C.tolist() == [[0.0] * 8, [0.0] * 8, [3.0 * i for i in range(8)]]
    F = torch.ones(3, 8, dtype=torch.bfloat16, device=dev())
    C, dA = A.spmm_sddmm(rp, ci, v, B, F, variant=variant)
    A.sync_status()
    assert C[2].tolist() == [3.0 * i for i in range(8)]
    assert dA[:5].tolist() == [0.0] * 5 and dA[-4:].tolist() == [0.0, 28.0, 28.0, 28.0]


@pytest.mark.parametrize("length", [70, 2, 33])  # of B's last row, one past whole steps of 32
def test_spgemm_reads_no_entry_past_the_last(length):
    b_rp = _rowptr(NNZ - length, NNZ)
    b_ci = torch.zeros(NNZ, dtype=torch.int32, device=dev())
    b_ci[-length:] = torch.arange(length, dtype=torch.int32, device=dev())
    b_v = torch.ones(NNZ, device=dev())
    a_rp = _rowptr(1, 2)
    a_ci = torch.tensor([1, 1], dtype=torch.int32, device=dev())
    a_v = torch.tensor([2.0, 3.0], device=dev())
    C = A.spgemm_dense(a_rp, a_ci, a_v, b_rp, b_ci, b_v, 80)
    A.sync_status()
    rest = [0.0] * (80 - length)
    assert C.tolist() == [[2.0] * length + rest, [3.0] * length + rest]
