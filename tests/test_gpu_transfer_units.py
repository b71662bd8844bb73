"""FP64 level transfer on vectors whose magnitudes differ from value to value, against an evaluation in extended
precision, value by value: the error over sum |matrices| |x| of the FP64 passes.

Tolerance, in units of 2^-53, per direction: a pass over N = k + 1 (restriction: 2 N) values is rounded by 4 units of
2^-58 of (largest row sum) x (largest value of its pencil, up to a binade: twice); that value enters every result, with the
smallest entry at least, hence the factor (row sum / smallest entry). FP64's own part is some 2 (2 N + 2). With one unit per
cell, or with values that a result does not depend on in it, small results are off by 1e6 and more."""
import numpy as np
import pytest

import extended as X

pytestmark = pytest.mark.gpu

SIZES = [(2, 1, (13, 5)), (2, 2, (7, 6)), (2, 3, (17, 3)), (2, 4, (5, 5)), (2, 7, (9, 2)), (3, 1, (3, 3, 2)), (3, 2, (2, 5, 3)),
         (3, 3, (5, 1, 2)), (3, 4, (3, 2, 3)), (3, 5, (2, 1, 3)), (3, 6, (2, 2, 1)), (3, 7, (1, 3, 2))]


def vectors(cells, nd, seed):
    g = np.random.Generator(np.random.Philox(seed))
    u = g.uniform(-1.0, 1.0, (cells, nd))
    yield "cells", u * 10.0 ** g.uniform(-14.0, 0.0, (cells, 1))
    yield "values", u * 10.0 ** g.uniform(-12.0, 0.0, (cells, nd))
    large = u.copy()
    large[:, g.integers(0, nd, max(1, nd // 8))] *= 1e12
    yield "a few large", large
    yield "regions", u * np.ldexp(1.0, np.array([-900, 0, 850])[np.minimum(np.arange(cells) * 3 // cells, 2)])[:, None]


@pytest.mark.parametrize("dim,k,ncc", SIZES)
def test_value_by_value(tpss, cuda, dim, k, ncc):
    import torch
    N, cells, nd = k + 1, int(np.prod(ncc)), (k + 1) ** dim
    E = X.embedding(k, 1)
    for restrict in (False, True):
        tol = dim * (2 * 4 * max(X.spread(E), X.spread(E.T)) / 32 + 2 * (2 * N + 2))
        for name, v in vectors(cells * 2 ** dim if restrict else cells, nd, 80 + k):
            v = v.reshape(-1)
            ref, bound = X.transfer(k, ncc, v, restrict)
            src = torch.tensor(v, dtype=torch.float64, device=cuda)
            out = torch.zeros(ref.size, dtype=torch.float64, device=cuda)
            if restrict:
                tpss.restrict_add(dim, k, ncc, out, src)
            else:
                tpss.prolongate_add(dim, k, ncc, out, src)
            assert X.worst(out.cpu().numpy(), ref, bound) <= tol, (restrict, name, tol)


@pytest.mark.parametrize("dim,k,ncc", [(2, 3, (4, 3)), (3, 2, (2, 2, 3)), (3, 5, (2, 1, 2))])
def test_coarse_nodes_are_exact(tpss, cuda, dim, k, ncc):
    """Fine nodes at a coarse cell's corners take its values as they are."""
    import torch
    N, cells = k + 1, int(np.prod(ncc))
    v = np.random.Generator(np.random.Philox(4)).uniform(-1.0, 1.0, (cells,) + (N,) * dim)
    corner = (slice(None),) + (0,) * dim
    v[corner] *= 1e-9
    up = torch.zeros(cells * 2 ** dim * N ** dim, dtype=torch.float64, device=cuda)
    tpss.prolongate_add(dim, k, ncc, up, torch.tensor(v.reshape(-1), dtype=torch.float64, device=cuda))
    # node 0 of the first child of every coarse cell
    fine = X.grid(up.cpu().numpy(), [2 * c for c in ncc], N)[(slice(None, None, 2 * N),) * dim]
    want = X.grid(v.reshape(-1), ncc, N)[(slice(None, None, N),) * dim]
    assert np.array_equal(fine, want)
