"""Error of the FP64 kernels that contract with integers against extended precision, in the root mean square over
the result's (the smoother: value by value over the bound of fast diagonalization), on random and on slowly varying
vectors of one magnitude.

Tolerances in units of u = 2^-53, from the roundings to FP64 alone; the integer contractions have to stay below them:
  operator   4 u: one rounding per pass and array (3), and the sums over the faces
  transfer   3 u: one rounding per pass
  C0IP      4 k u: the bands are sums of k + 1 quadrature terms, whose second derivatives are products of k - 1 factors
  smoother  4 dim (N + 2) u: 2 dim contractions of N values, and as much for the eigenvectors and eigenvalues in FP64"""
import numpy as np
import pytest

import extended as X

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def vectors(n, seed):
    g = np.random.Generator(np.random.Philox(seed))
    yield g.uniform(-1.0, 1.0, n)
    yield 1.0 + 0.01 * g.uniform(-1.0, 1.0, n)


def dev(x, cuda):
    import torch
    return torch.tensor(np.asarray(x, np.float64), dtype=torch.float64, device=cuda)


def layout(tpss, dim, k, nc, patch=1):
    return tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=patch))


@pytest.mark.parametrize("dim,k,nc", [(2, 3, (24, 25)), (2, 5, (9, 11)), (2, 6, (9, 8)), (2, 7, (8, 7)), (3, 3, (11, 11, 10)),
                                      (3, 4, (3, 10, 9)), (3, 5, (5, 4, 5)), (3, 7, (4, 3, 4))])
def test_operator(tpss, cuda, dim, k, nc):
    import torch
    op = tpss.LaplaceOperator(layout(tpss, dim, k, nc))
    for u in vectors(int(np.prod(nc)) * (k + 1) ** dim, k):
        d = torch.empty(u.size, dtype=torch.float64, device=cuda)
        op.vmult(d, dev(u, cuda))
        assert X.rms(d.cpu().numpy(), X.sipg(k, nc, u)[0]) <= 4 * U


@pytest.mark.parametrize("dim,k,ncc", [(2, 1, (9, 7)), (2, 4, (5, 5)), (2, 7, (5, 2)), (3, 1, (5, 4, 3)), (3, 2, (2, 5, 3)),
                                       (3, 4, (3, 2, 3)), (3, 7, (1, 3, 2))])
def test_transfer(tpss, cuda, dim, k, ncc):
    import torch
    n = int(np.prod(ncc)) * (k + 1) ** dim
    for c, f in zip(vectors(n, k), vectors(n * 2 ** dim, k + 10)):
        up, down = (torch.zeros(m, dtype=torch.float64, device=cuda) for m in (f.size, c.size))
        tpss.prolongate_add(dim, k, ncc, up, dev(c, cuda))
        tpss.restrict_add(dim, k, ncc, down, dev(f, cuda))
        assert X.rms(up.cpu().numpy(), X.transfer(k, ncc, c, False)[0]) <= 3 * U
        assert X.rms(down.cpu().numpy(), X.transfer(k, ncc, f, True)[0]) <= 3 * U


@pytest.mark.parametrize("k,nc", [(2, 24), (3, 16), (4, 12), (5, 10), (6, 8), (7, 6)])
def test_c0ip(tpss, cuda, k, nc):
    import torch
    P = tpss.C0IPBiharmonic(k, nc, nc)
    for x in vectors((nc * k - 1) ** 2, 5 * k):
        y = torch.empty(x.size, dtype=torch.float64, device=cuda)
        P.vmult(y, dev(x, cuda))
        assert X.rms(y.cpu().numpy(), X.c0ip(k, nc, x)[0]) <= 4 * k * U


@pytest.mark.parametrize("patch,variant", [("vertex", 0), ("vertex", 1), ("cell", 0)])
@pytest.mark.parametrize("dim,k,nc", [(2, 2, (7, 6)), (2, 3, (6, 5)), (2, 5, (5, 4)), (2, 7, (4, 4)), (3, 1, (4, 5, 4)), (3, 2, (3, 4, 3)),
                                      (3, 3, (3, 3, 2))])
def test_smoother(tpss, cuda, dim, k, nc, patch, variant):
    """variant: 0 the default kernel, 1 one launch per color."""
    import torch
    sh = layout(tpss, dim, k, nc, getattr(tpss.PatchVariant, patch))
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, None, tpss.SchwarzPreconditioner.AdditionalData(relaxation=1.0, precision=tpss.Precision.fp64,
                                                                     kernel_variant=variant))
    n = 2 if patch == "vertex" else 1
    for u in vectors(sh.n_dofs(), k):
        d = torch.empty(u.size, dtype=torch.float64, device=cuda)
        p.vmult(d, dev(u, cuda))
        assert X.worst(d.cpu().numpy(), *X.smoother(k, nc, u, n)) <= 4 * dim * (n * (k + 1) + 2)
