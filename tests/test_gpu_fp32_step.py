"""SchwarzSmoother steps with an FP32 smoother: the residual is that of the cell-wise operator, to the bit.

An operator that found no room for its line arrays runs the cell-wise kernel; steps with it are the reference. (A residual
with another rounding in its last FP64 bits rounds to another FP32 value now and then: 20 steps moved x by 1e-9.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_residual_is_cellwise(tpss, cuda):
    import torch
    dim, k, nc = 3, 4, (24, 24, 24)
    sh = tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=dim, degree=k, n_cells=nc, patch_variant=1))
    n = sh.n_dofs()
    g = np.random.Generator(np.random.Philox(2))
    x0, b = (torch.tensor(g.uniform(-1.0, 1.0, n), dtype=torch.float64, device=cuda) for _ in range(2))

    def steps(op):
        p = tpss.SchwarzPreconditioner()
        p.initialize(sh, op, tpss.SchwarzPreconditioner.AdditionalData(relaxation=0.15, precision=tpss.Precision.fp32))
        s = tpss.SchwarzSmoother()
        s.initialize(op, p, tpss.SchwarzSmoother.AdditionalData(number_of_smoothing_steps=20))
        x = x0.clone()
        s.step(x, b)
        return x

    with_arrays = tpss.LaplaceOperator(sh)
    got = steps(with_arrays)
    keep = 40 << 20  # the line arrays take 55 MB
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = []
    while torch.cuda.mem_get_info()[0] > keep + (8 << 20):
        fill.append(torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device=cuda))
    without = tpss.LaplaceOperator(sh)
    del fill
    torch.cuda.empty_cache()
    y = [torch.empty_like(b) for _ in range(2)]
    with_arrays.vmult(y[0], b)
    without.vmult(y[1], b)
    assert not torch.equal(y[0], y[1])
    assert torch.equal(got, steps(without))
