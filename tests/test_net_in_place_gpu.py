"""Predictions written over their own inputs equal those written elsewhere, bit for bit: the network's
kernels are the same, whether the output rows are narrower than the input rows, as wide or wider, and
whether the two buffers begin together or a part of a row apart."""
import ctypes

import pytest

import casim_b200 as cb
from casim_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_out,depth,rows,shift", [(20, 20, 2, 384, 0), (63, 20, 4, 148 * 128 + 128, 0), (16, 60, 1, 1280, 0),
                                                         (40, 40, 2, 1280, 12), (7, 5, 16, 256, 0)])
def test_forward_in_place(cuda_device, n_in, n_out, depth, rows, shift):
    import torch
    net = sg.Surrogate(n_in, n_out, width=128, depth=depth, seed=n_in)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, n_in), generator=g, device="cuda")
    want = net.forward(x)
    buf = torch.zeros(shift + rows * max(n_in, n_out), device="cuda")
    buf[shift:shift + rows * n_in] = x.reshape(-1)
    torch.cuda.synchronize()
    p = buf.data_ptr()
    st = cb.lib().casim_b200_sg_forward(net.h, ctypes.c_void_p(p + 4 * shift), rows, ctypes.c_void_p(p))
    assert st == cb.OK
    assert torch.equal(buf[:rows * n_out].reshape(rows, n_out), want)
    net.close()
