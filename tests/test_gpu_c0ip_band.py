"""C0IP / FE_Q operator with integers: every degree, from two cells (each next to both boundaries) to more cells than
classes of rows, magnitudes the integers do not cover, infinities and zeros, against the numpy oracle.

Tolerance 1e-12 (relative max-norm): a contraction's error is 2^-57 of (row sum of the band) x (largest
value of its window), below FP64's own rounding, so the FP64 tolerance of the operator applies
unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def philox(seed, n):
    return np.random.Generator(np.random.Philox(seed)).uniform(-1.0, 1.0, n)


def apply(P, x, cuda):
    import torch
    xs = torch.tensor(x, dtype=torch.float64, device=cuda)
    y = torch.full_like(xs, float("nan"))
    P.vmult(y, xs)
    return y.cpu().numpy()


@pytest.fixture(scope="module")
def c0():
    from oracle import np_c0ip
    return np_c0ip


@pytest.mark.parametrize("problem", ["biharmonic", "poisson"])
@pytest.mark.parametrize("k,nc", [(2, 2), (2, 11), (3, 2), (3, 5), (3, 9), (4, 3), (4, 6), (5, 5), (6, 4), (7, 3)])
def test_sizes_and_scales(tpss, c0, cuda, k, nc, problem):
    kw = dict(problem=tpss.C0IPBiharmonic.Q_POISSON) if problem == "poisson" else {}
    P = tpss.C0IPBiharmonic(k, nc, nc, **kw)
    A = c0.level_matrix(k, nc, problem="poisson") if problem == "poisson" else c0.level_matrix(k, nc)
    x = philox(40 + k, A.shape[0])
    ref = A @ x
    # 2^+-270: inside the integers' range, 2^+-330: FP64 contractions
    for s in (1.0, 2.0 ** 270, 2.0 ** -270, 2.0 ** 330, 2.0 ** -330):
        assert rel_err(apply(P, x * s, cuda) / s, ref) <= 1e-12, s


def test_range_zeros_and_nan(tpss, c0, cuda):
    k, nc = 3, 10
    P = tpss.C0IPBiharmonic(k, nc, nc)
    A = c0.level_matrix(k, nc)
    n = nc * k - 1
    r = np.random.Generator(np.random.Philox(2))
    x = philox(1, n * n) * 10.0 ** r.uniform(-150.0, 100.0, n * n)
    assert rel_err(apply(P, x, cuda), A @ x) <= 1e-12
    assert not apply(P, np.zeros(n * n), cuda).any()
    x = philox(3, n * n)
    fine = apply(P, x, cuda).reshape(n, n)
    for bad in (np.inf, np.nan):
        x2 = x.copy().reshape(n, n)
        x2[2, 2] = bad
        got = apply(P, x2.reshape(-1), cuda).reshape(n, n)
        assert not np.isfinite(got[2, 2])
        # rows or columns two cells and more away
        far = 2 + 2 * k + k
        assert np.array_equal(got[far:, :], fine[far:, :]) and np.array_equal(got[:, far:], fine[:, far:])
