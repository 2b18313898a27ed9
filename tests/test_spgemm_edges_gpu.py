"""The sparse x sparse -> dense kernel at its edges: rows of B around one and two loads of 32 entries
and past them, output widths around the column tiles (1024 to 4096), few and many rows of A, C
aligned and not, bit for bit the oracle's chains."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import bits, dev, to_dev

pytestmark = pytest.mark.gpu


def _csr(rng, lens, n_cols):
    rp = np.zeros(len(lens) + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(n_cols, n, replace=False)) for n in lens]).astype(np.int32)
    return rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32)


@pytest.mark.parametrize("M,N_", [(3, 300), (40, 1024), (40, 1025), (700, 2049), (2100, 4095),
                                  (2100, 4097), (1, 9000)])
def test_spgemm_edges_bit_exact(oracle, M, N_):
    rng = np.random.default_rng(M + N_)
    K = 90
    lens_b = rng.choice([0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 130, 290], K)
    a = _csr(rng, rng.integers(0, 70, M), K)
    b = _csr(rng, lens_b, N_)
    C0 = rng.uniform(-1, 1, (M, N_ + 3)).astype(np.float32)
    ad, bd = [to_dev(x) for x in a], [to_dev(x) for x in b]
    ref = oracle.spgemm_dense_f32(*a, *b, N_)
    assert np.array_equal(bits(A.spgemm_dense(*ad, *bd, N_)), bits(ref))
    for off in (0, 3):  # C inside a wider buffer
        C = to_dev(C0)[:, off:off + N_]
        A.spgemm_dense(*ad, *bd, N_, C=C, beta=1.0)
        ref = oracle.spgemm_dense_f32(*a, *b, N_, C=np.ascontiguousarray(C0[:, off:off + N_]))
        assert np.array_equal(bits(C.contiguous()), bits(ref))
    A.sync_status()
