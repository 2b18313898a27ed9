"""The long-row kernel (csrc/spmm_long.cu) at its edges: rows around whole blocks of 64 entries and
around a turn of its producers (384), columns around whole slices (32 fp32, 64 bf16) and every way
it reads B (16-byte, 4-byte and 2-byte pieces), bit for bit the oracle's chain; the same chain
length for the max, whose padding repeats a row's last entry."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import bits, csr_dev, dev, to_dev

pytestmark = pytest.mark.gpu

# four short rows for each long one keep the mean low, so that every row past 64 entries is long
LENS = [65, 127, 128, 129, 320, 383, 384, 385, 449, 768, 833]
K = 900


def _matrix(seed):
    rng = np.random.default_rng(seed)
    lens = np.zeros(64 * len(LENS), np.int64)
    lens[::64] = LENS
    lens[1::64] = 3
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(K, n, replace=False)) for n in lens]).astype(np.int32)
    return S.CSR(rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32), lens.size, K)


@pytest.mark.parametrize("offset", [0, 1])  # of B and C inside wider buffers: unaligned rows
@pytest.mark.parametrize("N_", [1, 2, 31, 32, 33, 64, 65, 136])
def test_long_row_edges_bit_exact(oracle, N_, offset):
    a = _matrix(N_)
    rp, ci, v = csr_dev(a)
    ld = N_ + 3 * offset
    Bw = S.dense_uniform((K, ld), 7 + N_)
    B = np.ascontiguousarray(Bw[:, offset:offset + N_])
    Bd = to_dev(Bw)[:, offset:offset + N_]
    C = A.spmm(rp, ci, v, Bd)
    ref = oracle.spmm_fma_chain_f32(a.rowptr, a.colind, a.val, B)
    assert np.array_equal(bits(C), bits(ref))
    A.spmm(rp, ci, v, Bd, C=C, beta=1.0)  # the chain goes on from C
    ref2 = oracle.spmm_fma_chain_f32(a.rowptr, a.colind, a.val, B, C=ref)
    assert np.array_equal(bits(C), bits(ref2))
    vb, Bb = oracle.bf16_round(a.val), oracle.bf16_round(B)
    refb = oracle.spmm_fma_chain_f32(a.rowptr, a.colind, vb, Bb)
    Cb = A.spmm(rp, ci, v.to(torch.bfloat16), to_dev(Bw).to(torch.bfloat16)[:, offset:offset + N_])
    assert np.array_equal(bits(Cb), bits(refb))
    # max: padded positions leave the result (all products negative in half of the columns)
    Bm = Bd - 2.0 * (torch.arange(N_, device=dev()) % 2)
    got = A.spmm_reduce(rp, ci, Bm.contiguous(), val=v.abs(), op="max")
    rows = np.repeat(np.arange(a.n_rows), np.diff(a.rowptr))
    want = np.full((a.n_rows, N_), -np.inf, np.float32)
    np.maximum.at(want, rows, np.abs(a.val)[:, None] * Bm.cpu().numpy()[a.colind])
    want[np.diff(a.rowptr) == 0] = 0.0
    assert np.array_equal(got.cpu().numpy(), want)
    A.sync_status()


def test_negative_zero_and_nan_survive_padding():
    """A chain that stands at -0.0 stays -0.0 through a block's padded positions; infinities and
    NaN of an entry come through."""
    a = _matrix(3)
    rp, ci, v = csr_dev(a)
    v = torch.where(v == 0, torch.ones_like(v), v.abs())
    B = torch.full((K, 40), -0.0, device=dev())
    B[:, 1], B[:, 2] = float("inf"), float("nan")
    C = torch.full((a.n_rows, 40), -0.0, device=dev())
    A.spmm(rp, ci, v, B, C=C, beta=1.0)
    filled = torch.from_numpy(np.diff(a.rowptr) > 0).to(dev())
    rest = torch.cat([C[:, :1], C[:, 3:]], 1)
    assert bool((rest.view(torch.int32) == -(1 << 31)).all())
    assert bool(torch.isposinf(C[filled, 1]).all()) and bool(torch.isnan(C[filled, 2]).all())
    A.sync_status()
