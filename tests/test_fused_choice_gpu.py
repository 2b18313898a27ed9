"""The fused SpMM + SDDMM's library choice is by entries, width and type: on both sides of its lines
(300,000 and 5,000,000 entries) variant 0 gives bit for bit what the variant that it stands for gives,
and its dot products and rows are the sums in 64 bits to within fp32 rounding."""
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import dev

pytestmark = pytest.mark.gpu
M = 40_000


def _expected(nnz, width, dtype):
    e = 4 if dtype == torch.float32 else 2  # bytes of an element
    if nnz >= 5_000_000:
        for name, cols in (("nnzme_v8_g8_ch1024", 64 // e), ("nnzme_v8_g16_ch1024", 128 // e),
                           ("nnzsplit_v16_g16_c1_ch256_u8", 256 // e),
                           ("nnzsplit_v16_g32_c1_ch256_u8", 512 // e),
                           ("nnzsplit_v16_g32_c2_ch256_u8", 1024 // e)):
            if width <= cols:
                return name
    if nnz >= 300_000:
        names = (("nnzsplit_v4_g32_c1_ch128", 128 // e), ("nnzsplit_v16_g16_c1_ch128", 256 // e),
                 ("nnzsplit_v16_g32_c1_ch128", 512 // e), ("nnzsplit_v16_g32_c2_ch128", 1024 // e))
    else:
        names = (("nnzsplit_v4_g32_c1_ch32", min(64, 128 // e)), ("nnzsplit_v4_g32_c2_ch32", min(64, 256 // e)),
                 ("nnzsplit_v4_g32_c2_ch128", 256 // e), ("nnzsplit_v16_g32_c1_ch128", 512 // e),
                 ("nnzsplit_v16_g32_c2_ch128", 1024 // e))
    return next(name for name, cols in names if width <= cols)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nnz", [299_999, 300_000, 4_999_999, 5_000_000])
def test_variant_zero_is_the_class_pick(nnz, dtype):
    gen = torch.Generator(device=dev()).manual_seed(nnz)
    u = torch.rand(M, generator=gen, device=dev(), dtype=torch.float64)
    w = (1 - u) ** -0.6  # skewed lengths, some rows over several chunks
    cum = torch.cumsum(w, 0)
    rp = torch.zeros(M + 1, dtype=torch.int32, device=dev())
    rp[1:] = (cum / cum[-1] * nnz).round().int()
    ci = torch.randint(0, M, (nnz,), generator=gen, device=dev(), dtype=torch.int32)
    v = (torch.rand(nnz, generator=gen, device=dev()) - 0.5).to(dtype)
    rows = torch.repeat_interleave(torch.arange(M, device=dev()), rp.diff().long())
    for width in (8, 16, 24, 32, 48, 64, 72, 128, 136, 256):
        B = torch.randn(M, width, generator=gen, device=dev()).to(dtype)
        F = torch.randn(M, width, generator=gen, device=dev()).to(dtype)
        name = _expected(nnz, width, dtype)
        variant = A.spmm_variants(dtype).index(name) + 1
        want, dwant = A.spmm_sddmm(rp, ci, v, B, F, variant=variant)
        C, dA = A.spmm_sddmm(rp, ci, v, B, F)
        assert torch.equal(C.view(torch.int32), want.view(torch.int32)), (name, width)
        assert torch.equal(dA.view(torch.int32), dwant.view(torch.int32)), (name, width)
        if width in (16, 72):
            # a chain of n products in fp32 is within n roundings of their absolute sum
            s = torch.randint(0, nnz, (20_000,), generator=gen, device=dev())
            p = B[ci[s].long()].double() * F[rows[s]].double()
            assert ((dA[s] - p.sum(1)).abs() <= 2.0 ** -23 * (width + 6) * p.abs().sum(1)).all(), name
            terms = B[ci.long()].double() * v.double()[:, None]
            ref = torch.zeros(M, width, dtype=torch.float64, device=dev()).index_add_(0, rows, terms)
            size = torch.zeros_like(ref).index_add_(0, rows, terms.abs())
            n = rp.diff()[:, None].double() + 2
            assert ((C - ref).abs() <= 2.0 ** -23 * n * size).all(), name
    A.sync_status()
