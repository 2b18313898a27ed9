"""Which rows the long-row kernel takes: rows at its threshold (256 entries) and past it for each of its
callers, bit for bit, and a matrix of equal rows among empty ones, which belongs to the row kernels
(the long-row kernel takes two to three times as long for it)."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import bits, csr_dev, dev, to_dev

pytestmark = pytest.mark.gpu
LENS = [64, 65, 128, 255, 256, 257, 258, 512, 513]  # among single entries
K = 640


def _matrix():
    rng = np.random.default_rng(5)
    lens = np.ones(16 * len(LENS), np.int64)
    lens[::16] = LENS
    lens[1::16] = 0
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(K, n, replace=False)) for n in lens]).astype(np.int32)
    return S.CSR(rp, ci, rng.uniform(0.5, 1.0, ci.size).astype(np.float32), lens.size, K)


@pytest.mark.parametrize("N_", [1, 8, 33, 64])
def test_rows_around_the_threshold(oracle, N_):
    a = _matrix()
    rp, ci, v = csr_dev(a)
    B = S.dense_uniform((K, N_), 3)
    Bd = to_dev(B)
    ref = oracle.spmm_fma_chain_f32(a.rowptr, a.colind, a.val, B)
    assert np.array_equal(bits(A.spmm(rp, ci, v, Bd)), bits(ref))
    assert np.array_equal(bits(A.spmm_reduce(rp, ci, Bd, val=v, op="sum")), bits(ref))
    # 1x4 blocks: no stored value is zero, so the chains are the CSR's (a row of n entries has up to
    # 4 n slots, so the rows of 64 and 65 lie on both sides of the threshold too)
    assert np.array_equal(bits(A.spmm_vcsr4(*A.csr_to_vcsr4(rp, ci, v), Bd)), bits(ref))
    # row pairs: an even row is its CSR chain (its partner here is empty)
    pairs = A.spmm_rowpair(*A.csr_to_rowpair(rp, ci, v), Bd)
    assert np.array_equal(bits(pairs)[::16], bits(ref)[::16])
    A.sync_status()


def _us(fn):
    fn()
    best = float("inf")
    for _ in range(5):
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda.synchronize()
        torch.cuda._sleep(500_000)
        start.record()
        for _ in range(5):
            fn()
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) * 200)
    return best


@pytest.mark.parametrize("op", ["spmm", "max"])
def test_equal_rows_among_empty_ones(op):
    """20,000 rows of 205 entries, alone and spread over 100,000 rows: the empty rows are 80,000 more
    row pointers and zeroed rows (51 MB), under a quarter of the work (bound: 1.6)."""
    n, width = 20_000, 128
    gen = torch.Generator(device=dev()).manual_seed(1)
    ci = torch.randint(0, 100_000, (n * 205,), generator=gen, device=dev(), dtype=torch.int32)
    v = torch.rand(n * 205, generator=gen, device=dev())
    B = torch.rand(100_000, width, generator=gen, device=dev())
    lens = torch.zeros(100_000, dtype=torch.int64, device=dev())
    lens[::5] = 205
    times = []
    for ln in (lens[::5], lens):
        rp = torch.zeros(ln.numel() + 1, dtype=torch.int32, device=dev())
        rp[1:] = torch.cumsum(ln, 0)
        if op == "spmm":
            times.append(_us(lambda: A.spmm(rp, ci, v, B)))
        else:
            times.append(_us(lambda: A.spmm_reduce(rp, ci, B, val=v, op="max")))
    assert times[1] < 1.6 * times[0], times
