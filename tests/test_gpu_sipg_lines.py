"""FP64 SIPG operator, line by line with integers: tile edges along x, segments of the lines, faces between
cells of different widths, permuted cells, magnitudes the integers do not cover, infinities and zeros,
against the CPU oracle.

Tolerance 1e-12 (relative max-norm): a contraction's error is 2^-58 of (row sum of the 1-D matrix) x
(largest value of its pencil), below FP64's own rounding, so the FP64 tolerance of the operator applies
unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def philox(seed, n):
    return np.random.Generator(np.random.Philox(seed)).uniform(-1.0, 1.0, n)


def widths(nc, seed, few=False):
    """Random cell widths; few: of two values, so that equal and unequal neighbours occur."""
    r = np.random.Generator(np.random.Philox(seed))
    w = [r.choice([0.5, 1.25], n) if few else r.uniform(0.5, 1.5, n) for n in nc]
    return [v / v.sum() for v in w]


def make(tpss, dim, k, nc, h=None, cells=None, ip=1.0, **kw):
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(
        dim=dim, degree=k, n_cells=nc, patch_variant=1, cell_h=h, cell_dof_start=cells))
    return tpss.LaplaceOperator(sh, ip, **kw)


def apply(op, src, cuda):
    import torch
    s = torch.tensor(src, dtype=torch.float64, device=cuda)
    d = torch.full_like(s, float("nan"))
    op.vmult(d, s)
    assert np.array_equal(s.cpu().numpy(), src, equal_nan=True)
    return d.cpu().numpy()


# cells along x around a tile's 40 / (k + 1); single cells (both faces on the boundary); more than one
# block of 128 lines; long lines (several segments); every degree
SIZES = [(2, 1, (41, 2)), (2, 2, (13, 1)), (2, 3, (10, 33)), (2, 4, (1, 1)), (2, 5, (7, 70)), (2, 6, (6, 9)), (2, 7, (5, 300)),
         (3, 1, (21, 3, 2)), (3, 2, (14, 5, 1)), (3, 3, (9, 2, 7)), (3, 4, (8, 3, 40)), (3, 4, (1, 1, 1)), (3, 5, (6, 1, 3)),
         (3, 6, (3, 4, 2)), (3, 7, (6, 2, 2)),
         # the lower degrees above take the cell-wise kernel on levels of that size; these do not
         (2, 1, (41, 830)), (2, 2, (13, 320)), (3, 1, (21, 40, 30)), (3, 2, (14, 31, 10)), (3, 3, (9, 11, 9)), (3, 4, (1, 10, 9))]


@pytest.mark.parametrize("dim,k,nc", SIZES)
def test_sizes_and_widths(tpss, oracle, cuda, dim, k, nc):
    src = philox(20 + k, int(np.prod(nc)) * (k + 1) ** dim)
    for h in (None, widths(nc, k), widths(nc, k, True)):
        op = make(tpss, dim, k, nc, h, ip=1.5)
        ref = oracle.sipg_vmult(dim, k, nc, src, ip=1.5, h=h)
        # 2^+-280: inside the integers' range, 2^+-320: FP64 contractions
        for scale in (1.0, 2.0 ** 280, 2.0 ** -280, 2.0 ** 320, 2.0 ** -320):
            assert rel_err(apply(op, src * scale, cuda) / scale, ref) <= 1e-12, (h is None, scale)


@pytest.mark.parametrize("dim,k,nc", [(2, 3, (11, 6)), (3, 2, (5, 6, 4)), (3, 2, (15, 17, 17))])
def test_cell_order_and_penalty(tpss, oracle, cuda, dim, k, nc):
    n_cells, cd = int(np.prod(nc)), (k + 1) ** dim
    cells = np.random.Generator(np.random.Philox(5)).permutation(n_cells).astype(np.int64) * cd
    src = philox(6, n_cells * cd)
    h = widths(nc, 7)
    op = make(tpss, dim, k, nc, h, cells, penalty_mode=tpss.Penalty.kp1sq)
    ref = oracle.sipg_vmult(dim, k, nc, src, h=h, cell_start=cells, penalty="kp1sq")
    assert rel_err(apply(op, src, cuda), ref) <= 1e-12


@pytest.mark.parametrize("dim,k,nc", [(2, 4, (9, 7)), (3, 3, (5, 4, 6)), (3, 3, (10, 9, 10))])
def test_range_zeros_and_nan(tpss, oracle, cuda, dim, k, nc):
    cd = (k + 1) ** dim
    n = int(np.prod(nc)) * cd
    op = make(tpss, dim, k, nc)
    src = philox(1, n) * 10.0 ** np.random.Generator(np.random.Philox(2)).uniform(-150.0, 100.0, n)
    assert rel_err(apply(op, src, cuda), oracle.sipg_vmult(dim, k, nc, src)) <= 1e-12
    assert not apply(op, np.zeros(n), cuda).any()
    one = np.zeros(n)
    one[n // 3] = 1e-3
    ref = oracle.sipg_vmult(dim, k, nc, one)
    assert rel_err(apply(op, one, cuda), ref) <= 1e-12
    src = philox(3, n)
    fine = apply(op, src, cuda)
    cell = int(np.prod(nc)) // 2
    x = [cell % nc[0], cell // nc[0] % nc[1], cell // (nc[0] * nc[1])]
    for bad in (np.inf, np.nan):
        src2 = src.copy()
        src2[cell * cd + cd // 2] = bad
        got = apply(op, src2, cuda).reshape(-1, cd)
        assert not np.isfinite(got[cell]).all()
        # cells that share neither a face nor an edge's layer with it stay as they are
        for c in range(got.shape[0]):
            y = [c % nc[0], c // nc[0] % nc[1], c // (nc[0] * nc[1])]
            if max(abs(a - b) for a, b in zip(x, y)) > 1:
                assert np.array_equal(got[c], fine.reshape(-1, cd)[c])


def test_two_streams(tpss, oracle, cuda):
    """One operator applied on two streams in turn: the second call waits for the first's scratch."""
    import torch
    dim, k, nc = 3, 3, (24, 24, 24)
    op = make(tpss, dim, k, nc)
    n = int(np.prod(nc)) * (k + 1) ** dim
    src = [torch.tensor(philox(i, n), dtype=torch.float64, device=cuda) for i in range(2)]
    want = []
    for s in src:
        want.append(torch.empty_like(s))
        op.vmult(want[-1], s)
    got = [torch.empty_like(s) for s in src]
    streams = [torch.cuda.Stream(device=cuda) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(5):
        for st, g, s in zip(streams, got, src):
            with torch.cuda.stream(st):
                g.zero_()
                op.vmult(g, s)
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert torch.equal(w, g)
