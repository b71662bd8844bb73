"""FP64 level transfer with integers: cells per block and remainders, every degree, magnitudes the integers do
not cover, infinities and zeros, against the CPU oracle.

Tolerance 1e-12 (relative max-norm): a pass's rounding is 2^-58 of the cell's largest value, below FP64's
own, so the FP64 tolerance of the transfer applies unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def philox(seed, n):
    return np.random.Generator(np.random.Philox(seed)).uniform(-1.0, 1.0, n)


def both(tpss, dim, k, ncc, coarse, fine, cuda):
    """(fine + P coarse, coarse + R fine)"""
    import torch
    c, f = (torch.tensor(v, dtype=torch.float64, device=cuda) for v in (coarse, fine))
    up, down = f.clone(), c.clone()
    tpss.prolongate_add(dim, k, ncc, up, c)
    tpss.restrict_add(dim, k, ncc, down, f)
    return up.cpu().numpy(), down.cpu().numpy()


def vectors(dim, k, ncc, seed):
    n = int(np.prod(ncc)) * (k + 1) ** dim
    return philox(seed, n), philox(seed + 1, n * 2 ** dim)


# one coarse cell; fewer and more cells than a block's share, odd counts
SIZES = [(2, 1, (1, 1)), (2, 1, (13, 5)), (2, 2, (7, 6)), (2, 3, (17, 3)), (2, 4, (5, 5)), (2, 5, (11, 2)), (2, 6, (3, 7)),
         (2, 7, (9, 2)), (3, 1, (3, 3, 2)), (3, 2, (2, 5, 3)), (3, 3, (1, 1, 1)), (3, 3, (5, 1, 2)), (3, 4, (3, 2, 3)),
         (3, 5, (2, 1, 3)), (3, 6, (2, 2, 1)), (3, 7, (1, 3, 2))]


@pytest.mark.parametrize("dim,k,ncc", SIZES)
def test_sizes_and_scales(tpss, oracle, cuda, dim, k, ncc):
    c, f = vectors(dim, k, ncc, 30 + k)
    up, down = oracle.prolongate_add(dim, k, ncc, c, f), oracle.restrict_add(dim, k, ncc, c, f)
    # 2^+-280: inside the integers' range, 2^+-320: FP64 passes
    for s in (1.0, 2.0 ** 280, 2.0 ** -280, 2.0 ** 320, 2.0 ** -320):
        u, d = both(tpss, dim, k, ncc, c * s, f * s, cuda)
        assert rel_err(u / s, up) <= 1e-12 and rel_err(d / s, down) <= 1e-12, s


@pytest.mark.parametrize("dim,k,ncc", [(2, 3, (6, 5)), (3, 4, (3, 2, 2))])
def test_range_zeros_and_nan(tpss, oracle, cuda, dim, k, ncc):
    nd = (k + 1) ** dim
    c, f = vectors(dim, k, ncc, 7)
    r = np.random.Generator(np.random.Philox(9))
    cw, fw = c * 10.0 ** r.uniform(-150.0, 100.0, c.size), f * 10.0 ** r.uniform(-150.0, 100.0, f.size)
    u, d = both(tpss, dim, k, ncc, cw, fw, cuda)
    assert rel_err(u, oracle.prolongate_add(dim, k, ncc, cw, fw)) <= 1e-12
    assert rel_err(d, oracle.restrict_add(dim, k, ncc, cw, fw)) <= 1e-12
    u, d = both(tpss, dim, k, ncc, np.zeros_like(c), np.zeros_like(f), cuda)
    assert not u.any() and not d.any()
    u, d = both(tpss, dim, k, ncc, np.zeros_like(c), f, cuda)
    assert np.array_equal(u, f)
    u0, d0 = both(tpss, dim, k, ncc, c, f, cuda)
    for bad in (np.inf, np.nan):
        c2, f2 = c.copy(), f.copy()
        c2[nd + nd // 2] = f2[nd // 2] = bad  # coarse cell 1; fine cell 0, a child of coarse cell 0
        u, d = both(tpss, dim, k, ncc, c2, f2, cuda)
        # fine cells 2 and 3 of the first row are children of coarse cell 1
        assert not np.isfinite(u[2 * nd:3 * nd]).all() and not np.isfinite(d[:nd]).all()
        assert np.array_equal(u[4 * nd:2 * ncc[0] * nd], u0[4 * nd:2 * ncc[0] * nd])
        assert np.array_equal(d[2 * nd:], d0[2 * nd:])
