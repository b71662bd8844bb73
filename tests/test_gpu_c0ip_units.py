"""C0IP / FE_Q operator on vectors whose magnitudes differ from node to node, against an evaluation in extended
precision, value by value: the error over sum |row| |x| of the FP64 factorization.

Tolerance, in units of 2^-53, per direction: a row's integers are rounded by (terms / 4 + 2) 2^-57 of (largest row sum) x
(largest value of those the row contracts, up to a binade: twice); that value enters the bound with the row's smallest entry
at least, hence the factor (row sum / smallest entry). FP64's own part is some 2 (terms + 2). A unit that a
value outside the row has set shows at once: with values 1e12 times larger it is off by 1e8 and more."""
import numpy as np
import pytest

import extended as X

pytestmark = pytest.mark.gpu


def apply(P, x, cuda):
    import torch
    xs = torch.tensor(np.asarray(x, np.float64), dtype=torch.float64, device=cuda)
    y = torch.full_like(xs, float("nan"))
    P.vmult(y, xs)
    return y.cpu().numpy()


def vectors(k, nc, seed):
    n = nc * k - 1
    g = np.random.Generator(np.random.Philox(seed))
    u = g.uniform(-1.0, 1.0, (n, n))
    # the inside nodes of every fifth cell along x, y and both; each value by itself; three regions, two of which
    # the integers do not cover
    inside = np.array([((i + 1) // k) % 5 == 2 and (i + 1) % k != 0 for i in range(n)])
    stripe = np.where(inside, 1e12, 1.0)
    yield "x", u * stripe
    yield "y", u * stripe[:, None]
    yield "both", u * stripe * stripe[:, None]
    yield "values", u * 10.0 ** g.uniform(-12.0, 0.0, (n, n))
    yield "regions", u * np.ldexp(1.0, np.repeat([-900, 0, 850], n)[np.minimum(np.arange(n) * 3 // n, 2) * n])[:, None]


@pytest.mark.parametrize("k,nc", [(2, 13), (3, 9), (3, 16), (4, 9), (5, 8), (6, 8), (7, 8)])
def test_value_by_value(tpss, cuda, k, nc):
    P = tpss.C0IPBiharmonic(k, nc, nc)
    terms = 4 * k + 1
    spread = max(X.spread(B) for B in X.q_1d(k, nc))
    tol = 2 * (2 * (terms / 4 + 2) * spread / 16 + 2 * (terms + 2))
    for name, x in vectors(k, nc, 60 + k):
        ref, bound = X.c0ip(k, nc, x)
        assert X.worst(apply(P, x.reshape(-1), cuda), ref, bound) <= tol, (name, tol)
