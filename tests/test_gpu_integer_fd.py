"""FP64 fast-diagonalization kernels that contract on the integer pipe: block exponents, tile edges,
magnitudes the integers do not cover, infinities and zeros, against the CPU oracle.

Tolerance 1e-12 (relative max-norm): a contraction's error is 2^-58 of (row sum of the 1-D matrix) x
(largest value of its block), below FP64's own rounding, so the FP64 tolerance of the smoother applies
unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def philox(seed, n):
    return np.random.Generator(np.random.Philox(seed)).uniform(-1.0, 1.0, n)


def widths(nc, seed):
    r = np.random.Generator(np.random.Philox(seed))
    return [w / w.sum() for w in (r.uniform(0.5, 1.5, n) for n in nc)]


def make(tpss, dim, k, nc, pv=1, sv=0, h=None, cells=None, **ad):
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(
        dim=dim, degree=k, n_cells=nc, patch_variant=pv, smoother_variant=sv, cell_h=h, cell_dof_start=cells))
    op = tpss.LaplaceOperator(sh) if sv == 1 else None
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, op, tpss.SchwarzPreconditioner.AdditionalData(precision=0, **ad))
    return p


def apply(p, src, cuda):
    import torch
    s = torch.tensor(src, dtype=torch.float64, device=cuda)
    d = torch.full_like(s, float("nan"))
    p.vmult(d, s)
    return d.cpu().numpy()


# patch counts around one CTA's share and below it; even and odd 1-D sizes; one patch
COLOR = [(2, 1, (2, 2), 1, 0), (2, 3, (17, 9), 1, 0), (2, 7, (4, 3), 1, 1), (2, 6, (9, 5), 0, 0), (3, 1, (6, 5, 5), 1, 0),
         (3, 2, (5, 4, 3), 1, 1), (3, 4, (5, 3, 4), 1, 0), (3, 7, (2, 3, 2), 1, 0), (3, 2, (4, 5, 3), 0, 0),
         (3, 4, (3, 2, 3), 0, 1)]


@pytest.mark.parametrize("dim,k,nc,pv,sv", COLOR)
def test_color_kernel(tpss, oracle, cuda, dim, k, nc, pv, sv):
    src = philox(10 + k, int(np.prod(nc)) * (k + 1) ** dim)
    om = 0.4
    for h in (None, widths(nc, k)):  # mirror-symmetric 1-D problems, and none
        ref = oracle.schwarz_vmult(dim, k, nc, src, patch_variant=pv, smoother_variant=sv, omega=om, h=h)
        p = make(tpss, dim, k, nc, pv, sv, h, relaxation=om, kernel_variant=1)
        # 2^+-290: inside the integers' range, 2^+-320: FP64 passes
        for scale in (1.0, 2.0 ** 290, 2.0 ** -290, 2.0 ** 320, 2.0 ** -320):
            assert rel_err(apply(p, src * scale, cuda) / scale, ref) <= 1e-12, (h is None, scale)


def check_range_and_nan(tpss, oracle, cuda, dim, k, nc, **kw):
    """Values over 500 orders of magnitude, zeros, an infinity and a NaN."""
    cd = (k + 1) ** dim
    n = int(np.prod(nc)) * cd
    om = 0.4
    p = make(tpss, dim, k, nc, relaxation=om, **kw)
    src = philox(1, n) * 10.0 ** np.random.Generator(np.random.Philox(2)).uniform(-150.0, 100.0, n)
    assert rel_err(apply(p, src, cuda), oracle.schwarz_vmult(dim, k, nc, src, omega=om)) <= 1e-12
    assert not apply(p, np.zeros(n), cuda).any()
    one = np.zeros(n)
    one[n // 3] = 1e-3
    ref = oracle.schwarz_vmult(dim, k, nc, one, omega=om)
    got = apply(p, one, cuda)
    assert rel_err(got, ref) <= 1e-12 and not got[ref == 0.0].any()
    src = philox(3, n)
    fine = apply(p, src, cuda)
    for bad in (np.inf, np.nan):
        cell = int(np.prod(nc)) // 2
        src2 = src.copy()
        src2[cell * cd + cd // 2] = bad
        got = apply(p, src2, cuda).reshape(-1, cd)
        idx = np.indices(list(reversed(nc))).reshape(dim, -1)
        near = (np.abs(idx - idx[:, cell][:, None]) <= 1).all(axis=0)  # cells of the patches that hold the DoF
        assert not np.isfinite(got[near]).any()
        assert np.array_equal(got[~near], fine.reshape(-1, cd)[~near])


@pytest.mark.parametrize("dim,k,nc", [(2, 3, (9, 7)), (3, 2, (5, 4, 6)), (3, 4, (4, 4, 3))])
def test_color_kernel_range_and_nan(tpss, oracle, cuda, dim, k, nc):
    check_range_and_nan(tpss, oracle, cuda, dim, k, nc, kernel_variant=1)


# vertices along x around the tile of 8 (4 for k >= 5 in 3D) and cells around 7 (3); one patch; line
# counts below and above one CTA's 128; lines long enough to be cut into segments
SWEEP = [(2, 1, (2, 2)), (2, 3, (8, 5)), (2, 3, (9, 4)), (2, 4, (3, 70)), (2, 7, (15, 3)), (2, 2, (40, 3)), (3, 1, (2, 2, 2)),
         (3, 1, (16, 2, 9)), (3, 2, (7, 5, 4)), (3, 3, (4, 3, 21)), (3, 4, (9, 2, 3)), (3, 5, (5, 4, 2)), (3, 6, (2, 3, 2)),
         (3, 7, (4, 2, 2))]


@pytest.mark.parametrize("dim,k,nc", SWEEP)
def test_direction_sweep(tpss, oracle, cuda, dim, k, nc):
    """The direction-by-direction smoother (the default for FP64 additive vertex patches) against the
    oracle on uniform cells, and on all against the per-color kernel, which reads the same tables;
    unequal widths (with k = 7 too many entry combinations for tabulated reciprocals; their 1-D
    eigenproblems are so ill-conditioned that either kernel differs from the oracle's own
    eigensolver by up to 1.5e-11), permuted cells, RAS weights."""
    nd = (k + 1) ** dim
    src = philox(20 + k, int(np.prod(nc)) * nd)
    om = 0.37
    cells = np.random.Generator(np.random.Philox(5)).permutation(int(np.prod(nc))).astype(np.int64) * nd
    for h, cs, ras in ((None, None, False), (widths(nc, k), None, True), (widths(nc, k + 1), cells, False)):
        kw = dict(h=h, cells=cs, relaxation=om, use_ras_weights=ras)
        got = apply(make(tpss, dim, k, nc, **kw), src, cuda)
        if h is None:
            ref = oracle.schwarz_vmult(dim, k, nc, src, omega=om)
            assert rel_err(got, ref) <= 1e-12
        assert rel_err(got, apply(make(tpss, dim, k, nc, kernel_variant=1, **kw), src, cuda)) <= 1e-12
    p = make(tpss, dim, k, nc, relaxation=om)
    ref = oracle.schwarz_vmult(dim, k, nc, src, omega=om)
    for scale in (2.0 ** 290, 2.0 ** -290, 2.0 ** 320, 2.0 ** -320):
        assert rel_err(apply(p, src * scale, cuda) / scale, ref) <= 1e-12, scale


@pytest.mark.parametrize("dim,k,nc", [(2, 3, (9, 7)), (3, 2, (5, 4, 6)), (3, 4, (4, 4, 3))])
def test_direction_sweep_range_and_nan(tpss, oracle, cuda, dim, k, nc):
    check_range_and_nan(tpss, oracle, cuda, dim, k, nc)
