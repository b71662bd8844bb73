"""Line arrays of the FP64 operator and smoother: allocated with their handle, so that a first application costs no
allocation and takes the same route inside a stream capture; where the device has no room, decided once."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIM, K, NC = 3, 4, (24, 24, 24)


def layout(tpss, nc=NC):
    return tpss.SubdomainHandler(tpss.SubdomainHandler.AdditionalData(dim=DIM, degree=K, n_cells=nc, patch_variant=1))


def smoother(tpss, sh, **kw):
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, None, tpss.SchwarzPreconditioner.AdditionalData(relaxation=0.15, precision=tpss.Precision.fp64, **kw))
    return p


class Shallow:
    """A shallow copy made through the C interface."""

    def __init__(self, tpss, p):
        self.lib, self.parent, self.h = tpss.load(), p, C.c_void_p()
        d = p._desc(p.get_additional_data())
        assert self.lib.tpss_precond_create_shallow(p.handle, C.byref(d), C.byref(self.h)) == 0

    def vmult(self, dst, src):
        import torch
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert self.lib.tpss_precond_vmult(self.h, C.c_void_p(dst.data_ptr()), C.c_void_p(src.data_ptr()), stream) == 0

    def __del__(self):
        self.lib.tpss_precond_destroy(self.h)


def make(tpss, what, sh):
    if what == "operator":
        return tpss.LaplaceOperator(sh)
    p = smoother(tpss, sh)
    return Shallow(tpss, p) if what == "shallow" else p


def vectors(cuda, n):
    import torch
    s = torch.tensor(np.random.Generator(np.random.Philox(2)).uniform(-1.0, 1.0, n), dtype=torch.float64, device=cuda)
    return s, torch.full_like(s, float("nan"))


@pytest.mark.parametrize("what", ["operator", "smoother", "shallow"])
def test_first_application_allocates_nothing(tpss, cuda, what):
    import torch
    sh = layout(tpss)
    s, d = vectors(cuda, sh.n_dofs())
    make(tpss, what, sh).vmult(d, s)  # loads the kernels' code
    torch.cuda.synchronize()
    h = make(tpss, what, sh)
    free = torch.cuda.mem_get_info()[0]
    h.vmult(d, s)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free


@pytest.mark.parametrize("what", ["operator", "smoother", "shallow"])
def test_captured_before_and_after_the_first_application(tpss, cuda, what):
    import torch
    sh = layout(tpss)
    s, want = vectors(cuda, sh.n_dofs())
    make(tpss, what, sh).vmult(want, s)
    h, got = make(tpss, what, sh), torch.full_like(s, float("nan"))
    for _ in range(2):
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            h.vmult(got, s)
        got.fill_(float("nan"))
        g.replay()
        assert torch.equal(got, want)
        got.fill_(float("nan"))
        h.vmult(got, s)
        assert torch.equal(got, want)


def test_smoother_on_two_streams(tpss, cuda):
    """One FP64 smoother applied on two streams in turn: the second call waits for the first's line arrays."""
    import torch
    sh = layout(tpss)
    p = smoother(tpss, sh)
    src = [vectors(cuda, sh.n_dofs())[0] * f for f in (1.0, -3.0)]
    want = [torch.empty_like(s) for s in src]
    for w, s in zip(want, src):
        p.vmult(w, s)
    got = [torch.empty_like(s) for s in src]
    streams = [torch.cuda.Stream(device=cuda) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(5):
        for st, g, s in zip(streams, got, src):
            with torch.cuda.stream(st):
                g.zero_()
                p.vmult(g, s)
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        assert torch.equal(w, g)


def test_no_room(tpss, cuda):
    """With 40 MB left on the device neither the operator's arrays (55 MB) nor the smoother's (126 MB) fit. The handles work
    without, within the FP64 tolerance, try no allocation again, and keep their route when there is room."""
    import torch
    sh = layout(tpss)
    s, d = vectors(cuda, sh.n_dofs())
    want = []
    for what in ("operator", "smoother"):
        make(tpss, what, sh).vmult(d, s)
        want.append(d.clone())
    # code of the kernels that do without line arrays
    small = layout(tpss, (2, 2, 2))
    a, b = vectors(cuda, small.n_dofs())
    tpss.LaplaceOperator(small).vmult(b, a)
    smoother(tpss, small, kernel_variant=1).vmult(b, a)
    smoother(tpss, sh, kernel_variant=1).vmult(d, s)
    keep = 40 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = []
    while torch.cuda.mem_get_info()[0] > keep + (8 << 20):
        fill.append(torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device=cuda))
    handles = [make(tpss, what, sh) for what in ("operator", "smoother")]
    free = torch.cuda.mem_get_info()[0]
    got = []
    for h, w in zip(handles, want):
        h.vmult(d, s)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        got.append(d.cpu().numpy())
        assert np.abs(got[-1] - w.cpu().numpy()).max() <= 1e-12 * w.abs().max().item()
        assert not np.array_equal(got[-1], w.cpu().numpy())  # another kernel's rounding
    del fill
    torch.cuda.empty_cache()
    for h, g in zip(handles, got):
        h.vmult(d, s)
        assert np.array_equal(d.cpu().numpy(), g)
