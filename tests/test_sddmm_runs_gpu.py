"""The CUDA-core SDDMM across runs of empty rows: as long as a group walks row by row (64), one more and
fewer, and far longer, for one lane per group and for many; bit for bit the oracle's order."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import bits, csr_dev, to_dev

pytestmark = pytest.mark.gpu


def _matrix(gaps, rng, n_cols):
    lens = np.concatenate([[0] * gap + [n] for gap in gaps for n in (1, 2, 5)])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(n_cols, n, replace=False)) for n in lens]).astype(np.int32)
    return S.CSR(rp, ci, rng.uniform(0.5, 1.5, ci.size).astype(np.float32), lens.size, n_cols)


@pytest.mark.parametrize("K", [1, 3, 4, 16, 20, 128, 130])
def test_runs_around_the_walk(oracle, K):
    a = _matrix((0, 62, 63, 64, 65, 66, 127, 128, 129, 5000), np.random.default_rng(K), 90)
    assert a.n_rows > 4 * a.nnz
    X, Y = S.dense_normal((a.n_rows, K), 1), S.dense_normal((90, K), 2)
    rp, ci, av = csr_dev(a)
    out = A.sddmm(rp, ci, to_dev(X), to_dev(Y), aval=av)
    assert np.array_equal(bits(out), bits(oracle.sddmm_f32_group(a.rowptr, a.colind, X, Y, aval=a.val)))
    A.sync_status()


def _gapped(n_rows, nnz, gap):
    """`nnz` entries spread evenly over `n_rows` rows but for a run of `gap` empty ones before the
    last entry's row; columns below 90."""
    starts = torch.linspace(0, nnz - 1, n_rows - gap, dtype=torch.float64).long()
    rp = torch.cat([starts, torch.full((gap + 1,), nnz - 1)])
    rp[-1] = nnz
    ci = torch.arange(nnz) * 7 % 90
    return rp.to(torch.int32), ci.to(torch.int32)


@pytest.mark.parametrize("K", [4, 16, 20, 128, 512])
@pytest.mark.parametrize("gap", [63, 64, 65, 1023, 1024, 1025, 60_000])
def test_one_run_among_rows_that_are_not_mostly_empty(oracle, K, gap):
    rp, ci = _gapped(gap + 400, max(1000, (gap + 400) // 4 + 1), gap)
    assert rp.numel() - 1 <= 4 * ci.numel()
    X, Y = S.dense_normal((rp.numel() - 1, K), 1), S.dense_normal((90, K), 2)
    out = A.sddmm(to_dev(rp.numpy()), to_dev(ci.numpy()), to_dev(X), to_dev(Y))
    assert np.array_equal(bits(out), bits(oracle.sddmm_f32_group(rp.numpy(), ci.numpy(), X, Y)))
    A.sync_status()


@pytest.mark.parametrize("K", [16, 32, 128])
def test_a_long_run_is_not_walked_row_by_row(K):
    """2M rows and 500,000 entries, the last after 1.9M empty rows: row by row the run alone takes some
    100 ms (a dependent load a row), a search microseconds; 20 ms parts the two."""
    rp, ci = (t.to("cuda") for t in _gapped(2_000_000, 500_000, 1_900_000))
    X, Y = torch.ones(2_000_000, K, device="cuda"), torch.ones(90, K, device="cuda")
    A.sddmm(rp, ci, X, Y)
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    start.record()
    out = A.sddmm(rp, ci, X, Y)
    end.record()
    torch.cuda.synchronize()
    assert bool((out == K).all())
    assert start.elapsed_time(end) < 20.0
