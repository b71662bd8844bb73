"""Levels far longer in one direction than a grid's second dimension (65,535): FP64 operator and additive
smoother against the CPU oracle, with the FP64 tolerance 1e-12 (relative max-norm) of the other sizes.

Along y and z a line has at most 65,535 segments; along x the tiles alone number more than that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def run(tpss, cuda, dim, k, nc, what):
    import torch
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=1))
    src = np.random.Generator(np.random.Philox(1)).uniform(-1.0, 1.0, sh.n_dofs())
    s = torch.tensor(src, dtype=torch.float64, device=cuda)
    d = torch.full_like(s, float("nan"))
    if what == "operator":
        tpss.LaplaceOperator(sh).vmult(d, s)
    else:
        p = tpss.SchwarzPreconditioner()
        p.initialize(sh, None, tpss.SchwarzPreconditioner.AdditionalData(relaxation=0.25, precision=tpss.Precision.fp64))
        p.vmult(d, s)
    return src, d.cpu().numpy()


@pytest.mark.parametrize("dim,k,nc", [(2, 1, (2, 70000)), (2, 2, (1, 66000)), (3, 1, (2, 1, 66000)), (2, 1, (1320000, 1))])
def test_operator(tpss, oracle, cuda, dim, k, nc):
    src, got = run(tpss, cuda, dim, k, nc, "operator")
    assert rel_err(got, oracle.sipg_vmult(dim, k, nc, src)) <= 1e-12


@pytest.mark.parametrize("dim,k,nc", [(2, 1, (2, 70000)), (3, 1, (2, 2, 66000)), (2, 1, (460000, 2))])
def test_smoother(tpss, oracle, cuda, dim, k, nc):
    src, got = run(tpss, cuda, dim, k, nc, "smoother")
    assert rel_err(got, oracle.schwarz_vmult(dim, k, nc, src, patch_variant=1, omega=0.25)) <= 1e-12
