"""A level of two cells per direction has one vertex patch: the default FP64 smoother takes the per-color kernel's single
launch there, and with it its result to the bit, within the FP64 tolerance 1e-12 of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("k", [1, 3, 4])
def test_one_launch(tpss, oracle, cuda, dim, k):
    import torch
    nc = (2,) * dim
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=1))
    src = np.random.Generator(np.random.Philox(k)).uniform(-1.0, 1.0, sh.n_dofs())
    s, out = torch.tensor(src, dtype=torch.float64, device=cuda), []
    for variant in (0, 1):
        p = tpss.SchwarzPreconditioner()
        p.initialize(sh, None, tpss.SchwarzPreconditioner.AdditionalData(
            relaxation=0.25, precision=tpss.Precision.fp64, kernel_variant=variant))
        out.append(torch.full_like(s, float("nan")))
        p.vmult(out[-1], s)
    assert torch.equal(out[0], out[1])
    ref = oracle.schwarz_vmult(dim, k, nc, src, patch_variant=1, omega=0.25)
    assert np.abs(out[0].cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
