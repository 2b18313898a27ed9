"""The tensor-core SDDMM's tile widths (csrc/sddmm_tc.cu, tile_width): shapes that 152 SMs take with
128-, 160-, 192-, 224- and 256-column tiles (the last columns in a ragged tile), against FP64 within
the split-bf16 path's 3e-5 of the terms, the same bits as the fixed 256-column kernel."""
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import csr_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N_", [(130, 300), (500, 5003), (1500, 2001), (1500, 2507), (2000, 2000),
                                  (1500, 3001)])
@pytest.mark.parametrize("K", [40, 200])
def test_tile_widths(oracle, M, N_, K):
    a = S.uniform_csr(M, N_, M * N_ // 40, seed=M + K, values="u0515")
    X, Y = S.dense_normal((M, K), 1), S.dense_normal((N_, K), 2)
    rp, ci, av = csr_dev(a)
    Xd, Yd = to_dev(X), to_dev(Y)
    out = A.sddmm(rp, ci, Xd, Yd, aval=av, tensor_cores=True)
    r64, ab = oracle.sddmm_f64(a.rowptr, a.colind, X, Y, aval=a.val)
    assert oracle.scaled_err(out.cpu().numpy(), r64, ab).max() < 3e-5
    # the MMA sums an output's terms alike in every tile (variant 2: 256 columns, wider stages)
    assert torch.equal(out, A.sddmm(rp, ci, Xd, Yd, aval=av, tensor_cores=True, variant=2))
    A.sync_status()
