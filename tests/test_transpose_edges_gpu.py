"""The transpose at the edges of its tiles (1,024 and, from 300,000 entries on, 4,096), of its digits
(1 to 3 passes) and of its row marks: empty rows at either end and in long runs, one row over many
tiles, many one-entry rows; with values, with the permutation and pattern only, bit for bit."""
import numpy as np
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import dev, to_dev

pytestmark = pytest.mark.gpu


def _lens(kind, nnz, rng):
    if kind == "hub":  # one row holds nearly all, empty rows around it
        return np.concatenate([[0] * 5, [3], [0] * 3000, [nnz - 10], [0] * 40, [7], [0] * 70])
    if kind == "ones":
        return np.concatenate([[0] * 33, np.ones(nnz, np.int64), [0]])
    lens = rng.integers(0, 12, nnz)  # mixed, cut to nnz
    cut = np.searchsorted(np.cumsum(lens), nnz)
    lens = lens[:cut + 1]
    lens[-1] -= lens.sum() - nnz
    return lens


@pytest.mark.parametrize("nnz,cols", [(1, 1), (1023, 2), (1024, 256), (1025, 257), (4097, 65536),
                                      (5000, 65537), (299_999, 70_000), (300_000, 300),
                                      (303_105, 2_100_000)])
@pytest.mark.parametrize("kind", ["hub", "ones", "mixed"])
def test_transpose_edges(nnz, cols, kind):
    rng = np.random.default_rng(nnz + cols)
    lens = _lens(kind, nnz, rng) if nnz > 10 else np.array([0, nnz, 0])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    assert rp[-1] == nnz
    # any order within a row, repeats included: the transpose is a stable sort by column
    ci = rng.integers(0, cols, nnz).astype(np.int32)
    v = rng.uniform(-1, 1, nnz).astype(np.float32)
    order = np.argsort(ci, kind="stable")
    rows = np.repeat(np.arange(lens.size), lens)[order]
    colptr = np.concatenate([[0], np.cumsum(np.bincount(ci, minlength=cols))])
    rpd, cid, vd = to_dev(rp), to_dev(ci), to_dev(v)
    cp, ri, cv = A.csr2csc(rpd, cid, vd, cols)
    cp1, ri1, none = A.csr2csc(rpd, cid, None, cols)
    cp2, ri2, perm = A.csr2csc_perm(rpd, cid, cols)
    assert none is None
    for c, r in ((cp, ri), (cp1, ri1), (cp2, ri2)):
        assert np.array_equal(c.cpu().numpy(), colptr) and np.array_equal(r.cpu().numpy(), rows)
    assert np.array_equal(cv.cpu().numpy(), v[order])
    assert np.array_equal(perm.cpu().numpy(), order)
    # columns read at an unaligned address
    wide = torch.empty(nnz + 1, dtype=torch.int32, device=dev())
    wide[1:] = cid
    assert np.array_equal(A.csr2csc(rpd, wide[1:], vd, cols)[1].cpu().numpy(), rows)
    A.sync_status()


@pytest.mark.parametrize("nnz,gap", [(3000, 16_384), (3000, 16_390), (301_000, 65_536), (301_000, 70_000)])
def test_transpose_long_runs_of_empty_rows(nnz, gap):
    """Runs of empty rows inside a tile about as long as where its entries look their rows up."""
    rng = np.random.default_rng(gap)
    part = rng.integers(1, 4, 40)
    lens = np.concatenate([[0] * gap, part, [0] * gap, [1], [0] * (gap - 1), part, [nnz - 2 * part.sum() - 2],
                           [0] * gap, [1], [0] * gap])
    rp = np.zeros(lens.size + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    assert rp[-1] == nnz
    ci = rng.integers(0, 900, nnz).astype(np.int32)
    order = np.argsort(ci, kind="stable")
    cp, ri, perm = A.csr2csc_perm(to_dev(rp), to_dev(ci), 900)
    assert np.array_equal(ri.cpu().numpy(), np.repeat(np.arange(lens.size), lens)[order])
    assert np.array_equal(perm.cpu().numpy(), order)
    A.sync_status()
