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


def test_row_kernels_read_no_entry_past_the_last():
    """Rows of at most 256 entries, the last of 250 (no whole number of steps)."""
    lens = torch.full((2 ** 23 + 1,), 256, dtype=torch.int64, device=dev())
    lens[0], lens[1], lens[-1] = 6, 255, 250
    rp = torch.zeros(lens.numel() + 1, dtype=torch.int32, device=dev())
    rp[1:] = torch.cumsum(lens, 0)
    assert int(rp[-1]) == NNZ
    ci, v = _columns(), torch.ones(NNZ, device=dev())
    B = torch.zeros(2, 8, device=dev())
    B[1] = torch.arange(8)

    def check(C, last):
        A.sync_status()
        assert C[-1].tolist() == last and not C[:-1].any()

    total = [3.0 * i for i in range(8)]
    check(A.spmm(rp, ci, v, B), total)
    check(A.spmm(rp, ci, v, B, variant=A.spmm_variants().index("rowsplit_v8_g32_c4_u4_pf") + 1), total)
    check(A.spmm_reduce(rp, ci, B, op="sum"), total)
    check(A.spmm_reduce(rp, ci, B, val=v, op="max"), [float(i) for i in range(8)])
    check(A.spmv(rp, ci, v, torch.tensor([0.0, 2.0], device=dev()))[:, None], [6.0])
    flags = torch.zeros(NNZ, dtype=torch.uint8, device=dev())
    check(A.spmm_rowpair(rp, ci, v, flags, B), total)


def test_row_pairs_of_a_matrix_past_half_the_limit():
    """The search for a column in a row's second half, past 2^30 entries."""
    rows = 2 ** 20 + 2 ** 18
    rp = torch.arange(rows + 1, dtype=torch.int32, device=dev()) * 1024
    ci = (torch.arange(1024, dtype=torch.int32, device=dev())).repeat(rows)
    rp2, ci2, _, flag2 = A.csr_to_rowpair(rp, ci, torch.ones(rows * 1024, device=dev()))
    A.sync_status()
    # both rows of a pair hold the same columns: the first takes all of its partner's entries
    assert torch.equal(rp2[::2], rp[::2]) and torch.equal(rp2[1:-1:2], rp[2::2])
    assert ci2[-4:].tolist() == [1022, 1022, 1023, 1023] and flag2[-4:].tolist() == [0, 1, 0, 1]
