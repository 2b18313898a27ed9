"""The CUDA-core SDDMM with a row held in registers (csrc/sddmm_simt.cu, sddmm_rows) at its edges: K
around whole blocks per lane (4 .. 512) and past them, runs of empty rows, one-entry rows and a row
over many groups, bad columns between good ones; bit for bit the oracle's lane-group order."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import bits, csr_dev, to_dev

pytestmark = pytest.mark.gpu


def _matrix(rng, n_cols):
    lens = np.concatenate([[0] * 70, [1] * 90, [0], [400], [0] * 45, rng.integers(0, 9, 200), [3, 0]])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(n_cols, n, replace=False)) for n in lens]).astype(np.int32)
    return S.CSR(rp, ci, rng.uniform(0.5, 1.5, ci.size).astype(np.float32), lens.size, n_cols)


@pytest.mark.parametrize("K", [1, 4, 8, 16, 20, 60, 64, 68, 128, 132, 500, 512, 516, 6])
def test_rows_bit_exact(oracle, K):
    a = _matrix(np.random.default_rng(K), 450)
    X, Y = S.dense_normal((a.n_rows, K), 1), S.dense_normal((450, K), 2)
    rp, ci, av = csr_dev(a)
    out = A.sddmm(rp, ci, to_dev(X), to_dev(Y), aval=av)
    ref = oracle.sddmm_f32_group(a.rowptr, a.colind, X, Y, aval=a.val)
    assert np.array_equal(bits(out), bits(ref))
    Xb, Yb = oracle.bf16_round(X), oracle.bf16_round(Y)
    out = A.sddmm(rp, ci, to_dev(Xb).to(torch.bfloat16), to_dev(Yb).to(torch.bfloat16))
    assert np.array_equal(bits(out), bits(oracle.sddmm_f32_group(a.rowptr, a.colind, Xb, Yb)))
    A.sync_status()
    if K == 64:  # bad columns are flagged and give 0; their neighbours stand
        bad = a.colind.copy()
        bad[[0, 5, 100, 101]] = [-1, 450, 1 << 30, -7]
        out = A.sddmm(rp, to_dev(bad), to_dev(X), to_dev(Y), aval=av).cpu().numpy()
        with pytest.raises(A.NativeError):
            A.sync_status()
        want = ref.copy()
        want[[0, 5, 100, 101]] = 0.0
        assert np.array_equal(bits(out), bits(want))


@pytest.mark.parametrize("K", [4, 16, 32, 128])
def test_mostly_empty_rows(oracle, K):
    """Runs of empty rows about as long as a group walks before it searches, and far longer."""
    lens = np.concatenate([([0] * gap + [n]) for gap in (0, 1, 15, 16, 17, 18, 33, 3000)
                           for n in (1, 2, 5)] + [[0] * 40])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    rng = np.random.default_rng(K)
    ci = np.concatenate([np.sort(rng.choice(90, n, replace=False)) for n in lens]).astype(np.int32)
    a = S.CSR(rp, ci, rng.uniform(0.5, 1.5, ci.size).astype(np.float32), lens.size, 90)
    assert a.n_rows > 4 * a.nnz
    X, Y = S.dense_normal((a.n_rows, K), 1), S.dense_normal((90, K), 2)
    rpd, cid, av = csr_dev(a)
    out = A.sddmm(rpd, cid, to_dev(X), to_dev(Y), aval=av)
    assert np.array_equal(bits(out), bits(oracle.sddmm_f32_group(a.rowptr, a.colind, X, Y, aval=a.val)))
    A.sync_status()
