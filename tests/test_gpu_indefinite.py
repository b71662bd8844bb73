"""FP64 smoothers whose local problems are indefinite (ip_factor 0.1): no integer contractions; each kernel against the
dense local inverses of the same tables.

Tolerance 1e-12 (relative max-norm), the FP64 tolerance of the smoothers."""
import numpy as np
import pytest

import extended as X

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patch,variant", [("vertex", 0), ("vertex", 1), ("cell", 0)])
@pytest.mark.parametrize("dim,k,nc", [(2, 1, (5, 6)), (2, 3, (6, 5)), (2, 4, (5, 5)), (2, 7, (4, 4)), (3, 1, (4, 5, 4)), (3, 2, (3, 4, 3)),
                                      (3, 3, (3, 3, 2))])
def test_local_inverses(tpss, cuda, dim, k, nc, patch, variant):
    import torch
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(
        dim=dim, degree=k, n_cells=nc, patch_variant=getattr(tpss.PatchVariant, patch)))
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, None, tpss.SchwarzPreconditioner.AdditionalData(
        relaxation=0.5, precision=tpss.Precision.fp64, ip_factor=0.1, kernel_variant=variant))
    lower = sh.patches()[0]
    inv = tpss.precond_local_inverse(p, 0, len(lower), device=cuda).cpu().numpy()
    n = (2 if patch == "vertex" else 1) * (k + 1)
    u = np.random.Generator(np.random.Philox(k)).uniform(-1.0, 1.0, sh.n_dofs())
    g = X.grid(u, nc, k + 1).astype(float)
    out = np.zeros_like(g)
    for B, low in zip(inv, lower):
        at = tuple(slice(low[d] * (k + 1), low[d] * (k + 1) + n) for d in reversed(range(dim)))
        out[at] += 0.5 * (B @ g[at].reshape(-1)).reshape((n,) * dim)
    d = torch.empty(u.size, dtype=torch.float64, device=cuda)
    p.vmult(d, torch.tensor(u, dtype=torch.float64, device=cuda))
    ref = X.ungrid(out, nc, k + 1)
    assert np.abs(d.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
