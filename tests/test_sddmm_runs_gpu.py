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
