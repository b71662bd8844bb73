"""Vectors of very large and very small magnitudes: scaled by a power of two inside the integers' range the FP64 operator, the
transfers and the C0IP operator give the scaled result to the bit; beyond it FP64 contractions take over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cases(tpss, cuda):
    import torch

    def rand(n):
        return torch.tensor(np.random.Generator(np.random.Philox(n)).uniform(-1.0, 1.0, n), dtype=torch.float64, device=cuda)

    for dim, k, nc in ((2, 4, (12, 13)), (3, 5, (5, 4, 5))):
        sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=1))
        op = tpss.LaplaceOperator(sh)
        yield rand(sh.n_dofs()), op.vmult
    for dim, k, nc in ((2, 3, (7, 5)), (3, 4, (2, 3, 2))):
        n = int(np.prod(nc)) * (k + 1) ** dim

        def up(d, s, a=(dim, k, nc)):
            d.zero_()
            tpss.prolongate_add(*a, d, s[:s.numel() // 2 ** a[0]].contiguous())

        def down(d, s, a=(dim, k, nc)):
            c = torch.zeros(s.numel() // 2 ** a[0], dtype=torch.float64, device=cuda)
            tpss.restrict_add(*a, c, s)
            d.zero_()
            d[:c.numel()] = c

        yield rand(n * 2 ** dim), up
        yield rand(n * 2 ** dim), down
    P = tpss.C0IPBiharmonic(3, 9, 9)
    yield rand(P.n_dofs()), P.vmult


def test_scaled(tpss, cuda):
    import torch
    for s, f in cases(tpss, cuda):
        want, got = torch.empty_like(s), torch.empty_like(s)
        f(want, s)
        for e in (-700, -400, 400, 700):
            f(got, s * 2.0 ** e)
            assert torch.equal(got * 2.0 ** -e, want), e
        for e in (-900, 900):
            f(got, s * 2.0 ** e)
            assert (got * 2.0 ** -e - want).abs().max() <= 1e-12 * want.abs().max(), e
