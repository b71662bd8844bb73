"""FP64 SIPG operator on vectors whose magnitudes differ from cell to cell and from value to value, against an
evaluation in extended precision, value by value: the error over sum |matrices| |u| of the FP64 factorization.

Tolerance, in units of 2^-53, per direction: a contraction of N = k + 1 values is rounded by (N / 4 + 2) 2^-58 of (largest row
sum) x (largest value of its pencil, up to a binade: twice); that value enters every result, with the smallest
entry at least, hence the factor (row sum / smallest entry). FP64's own part is some 2 (N + 2). A unit that a value
outside the pencil has set is off by 1e5 and more on cells that differ by up to 1e14. (For k = 1 the two nodes of a cell
do not couple at all: values that differ within a cell have no such bound there, with FP64's even/odd form neither.)"""
import numpy as np
import pytest

import extended as X

pytestmark = pytest.mark.gpu

# sizes on which the operator goes line by line
SIZES = [(2, 1, (41, 830)), (2, 2, (13, 320)), (2, 3, (24, 25)), (2, 4, (12, 13)), (2, 7, (8, 7)), (3, 3, (11, 11, 10)),
         (3, 4, (3, 10, 9)), (3, 5, (5, 4, 5)), (3, 7, (4, 3, 4))]


def operator(tpss, dim, k, nc):
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=1))
    return tpss.LaplaceOperator(sh)


def apply(op, src, cuda):
    import torch
    s = torch.tensor(src, dtype=torch.float64, device=cuda)
    d = torch.full_like(s, float("nan"))
    op.vmult(d, s)
    return d.cpu().numpy()


def vectors(dim, k, nc, seed):
    cells, nd = int(np.prod(nc)), (k + 1) ** dim
    g = np.random.Generator(np.random.Philox(seed))
    u = g.uniform(-1.0, 1.0, (cells, nd))
    yield "cells", u * 10.0 ** g.uniform(-14.0, 0.0, (cells, 1))
    spread = 10.0 ** g.uniform(-12.0, 0.0, (cells, nd))
    if k > 1:
        yield "values", u * spread
    # one cell's values are zero beside large ones; three regions, two of which the integers do not cover
    yield "zero", u * (g.uniform(0.0, 1.0, (cells, 1)) > 0.5) * 1e9
    yield "regions", u * np.ldexp(1.0, np.array([-900, 0, 850])[np.minimum(np.arange(cells) * 3 // cells, 2)])[:, None]


@pytest.mark.parametrize("dim,k,nc", SIZES)
def test_value_by_value(tpss, cuda, dim, k, nc):
    op = operator(tpss, dim, k, nc)
    N = k + 1
    spread = max(X.spread(B) for B in X.dg_1d(k, 5))
    tol = dim * (2 * (N / 4 + 2) * spread / 32 + 2 * (N + 2))
    for name, u in vectors(dim, k, nc, 70 + k):
        ref, bound = X.sipg(k, nc, u)
        assert X.worst(apply(op, u.reshape(-1), cuda), ref, bound) <= tol, (name, tol)


def test_tiles_and_segments_agree(tpss, cuda):
    """A trace is the same wherever it is computed: in its cell's own tile and segment or as the first value beside
    another's. With a large value in the cell, moved along the level by whole cells, the result moves with it."""
    dim, k, nc = 2, 4, (60, 60)
    op = operator(tpss, dim, k, nc)
    u = np.random.Generator(np.random.Philox(5)).uniform(-1.0, 1.0, (25,))
    big = u[::-1] * 1e9
    got = []
    for y in range(8, 52):
        for x in (8 + y % 9, 30 + y % 11):
            v = np.zeros((60, 60, 25))
            v[y, x], v[y, x + 1], v[y + 1, x] = u, big, big
            got.append(apply(op, v.reshape(-1), cuda).reshape(60, 60, 25)[y - 1:y + 3, x - 1:x + 3])
    for g in got[1:]:
        assert np.array_equal(g, got[0])
