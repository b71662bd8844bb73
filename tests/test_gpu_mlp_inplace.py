"""MLP.forward into its own input (as many outputs as inputs): with one layer, whose product reads the input
while it writes the output, and with hidden layers."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [0, 1, 3])
@pytest.mark.parametrize("rows", [300, 20000])
def test_output_over_input(tpss, cuda, layers, rows):
    import torch
    m = tpss.MLP(96, 96, 64, layers, seed=3)
    x = torch.tensor(np.random.Generator(np.random.Philox(1)).uniform(-1, 1, (rows, 96)), dtype=torch.float32, device=cuda)
    y = m.forward(x)
    for _ in range(3):
        z = x.clone()
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert tpss.load().tpss_mlp_forward(m.handle, C.c_void_p(z.data_ptr()), rows, C.c_void_p(z.data_ptr()), stream) == 0
        assert torch.equal(y, z)
