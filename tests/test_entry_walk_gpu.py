"""The entry-balanced SpMM's walk over entries (csrc/spmm_nnz.cu) where it can go wrong: runs of empty
rows longer than a window of row ends (8, 16, 32), rows that end at batch and chunk edges, runs of
one-entry rows; plain and fused with the SDDMM, bit for bit the oracle's order, and the fused pass's
library choice over its classes of size and layout."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from armsparse_gb300 import synthetic as S
from gpu_util import bits, csr_dev, to_dev
from test_spmm_nnz_order_gpu import _params

pytestmark = pytest.mark.gpu
K = 700


def _matrix(seed):
    rng = np.random.default_rng(seed)
    lens = np.concatenate([
        [0] * 40, [1] * 70, [0] * 33, [32, 0, 25, 1], [0] * 7, [8, 8, 16], [0] * 200,
        [300], [0] * 32, [1, 0] * 50, rng.integers(0, 6, 300), [129, 127, 256], [0] * 65, [3], [0] * 90])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(K, n, replace=False)) for n in lens]).astype(np.int32)
    return S.CSR(rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32), lens.size, K)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N_", [8, 33, 64])
def test_walk_bit_exact(oracle, dtype, N_):
    a = _matrix(N_)
    B, C0 = S.dense_uniform((K, N_), 1), S.dense_uniform((a.n_rows, N_), 2)
    F = S.dense_uniform((a.n_rows, N_), 3)
    v = a.val
    if dtype == torch.bfloat16:
        v, B, F = (oracle.bf16_round(x) for x in (v, B, F))
    rp, ci, _ = csr_dev(a)
    vd, Bd, Fd = (to_dev(x).to(dtype) for x in (v, B, F))
    rows = np.repeat(np.arange(a.n_rows), np.diff(a.rowptr))
    dots = np.einsum("ij,ij->i", B[a.colind].astype(np.float64), F[rows].astype(np.float64))
    size = np.einsum("ij,ij->i", np.abs(B[a.colind]).astype(np.float64), np.abs(F[rows]))
    ran = 0
    for i, name in enumerate(A.spmm_variants(dtype)):
        if not name.startswith("nnzsplit") or not A.spmm_variant_supported(i + 1, N_, dtype):
            continue
        ch, sub = _params(name)
        for beta in (0.0, 0.5):
            C = to_dev(C0).clone()
            A.spmm(rp, ci, vd, Bd, C=C, beta=beta, variant=i + 1)
            ref = oracle.spmm_nnz_order_f32(a.rowptr, a.colind, v, B, ch, sub, C=C0, beta=beta)
            assert np.array_equal(bits(C), bits(ref)), (name, beta)
        ran += 1
        try:
            Cf, dA = A.spmm_sddmm(rp, ci, vd, Bd, Fd, variant=i + 1)
        except A.NativeError as e:
            assert e.status == 3  # a column tile narrower than N
            continue
        ref = oracle.spmm_nnz_order_f32(a.rowptr, a.colind, v, B, ch, sub)
        assert np.array_equal(bits(Cf), bits(ref)), name
        err = np.abs(dA.cpu().numpy() - dots)
        assert (err <= 2.0 ** -23 * (N_ + 6) * size).all(), name  # N products, then the lanes' tree
    assert ran >= 3
    A.sync_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N_", [2, 30, 32, 48, 64, 66, 128, 136, 256])
def test_fused_choice_serves_every_layout(oracle, dtype, N_):
    """Small classes, aligned and not: the product and the dots within fp32 summation error."""
    a = _matrix(5)
    for off in (0, 2):  # columns 2.. of wider buffers: 8- (fp32) or 4-byte (bf16) aligned rows
        if off and N_ > (64 if dtype == torch.bfloat16 else 32):
            continue  # only 16-byte vectors cover these widths
        B, F = S.dense_uniform((K, N_ + off), 4), S.dense_uniform((a.n_rows, N_ + off), 5)
        v = a.val
        if dtype == torch.bfloat16:
            v, B, F = (oracle.bf16_round(x) for x in (v, B, F))
        rp, ci, _ = csr_dev(a)
        args = (rp, ci, to_dev(v).to(dtype), to_dev(B).to(dtype)[:, off:], to_dev(F).to(dtype)[:, off:])
        if N_ == 66:  # wider than the narrow vectors' tile, no multiple of the wide ones: refused
            with pytest.raises(A.NativeError):
                A.spmm_sddmm(*args)
            continue
        C, dA = A.spmm_sddmm(*args)
        R, Ab = oracle.spmm_f64(a.rowptr, a.colind, v, np.ascontiguousarray(B[:, off:]))
        assert oracle.scaled_err(C.cpu().numpy(), R, Ab).max() < 1e-5
        rows = np.repeat(np.arange(a.n_rows), np.diff(a.rowptr))
        x, y = B[a.colind, off:].astype(np.float64), F[rows, off:].astype(np.float64)
        err = np.abs(dA.cpu().numpy() - (x * y).sum(1))
        assert (err <= 2.0 ** -23 * (N_ + 6) * np.abs(x * y).sum(1)).all()
    A.sync_status()


def test_fused_choice_captured_without_room(monkeypatch):
    """A captured call whose arena holds the 1024-entry kernel's carry slots only runs that kernel."""
    from armsparse_gb300 import _native
    ctx = _native.Context(0)
    monkeypatch.setattr(_native, "context", lambda device=0: ctx)
    a = S.powerlaw_csr(3000, 2.1, 20.0, 3)
    B, F = (to_dev(S.dense_uniform((n, 48), s)) for n, s in ((a.n_cols, 1), (a.n_rows, 2)))
    args = (*csr_dev(a), B, F)
    long_chunks = A.spmm_variants(torch.float32).index("nnzsplit_v16_g32_c1_ch1024") + 1
    want, dwant = A.spmm_sddmm(*args, variant=long_chunks)
    C, dA = torch.empty_like(want), torch.empty_like(dwant)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.spmm_sddmm(*args, C=C, dA=dA)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(bits(C), bits(want)) and np.array_equal(bits(dA), bits(dwant))
    ctx.sync_status()
    g.reset()
    ctx.close()
