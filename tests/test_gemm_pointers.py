"""casim_b200_sg_gemm's pointers: an output on any float boundary gets the product that an aligned one
gets, bit for bit; operands off their 16-byte boundary, or an output off a float's, are refused
before anything reaches the device (pointers that are never followed: no GPU needed)."""
import ctypes

import pytest

import casim_b200 as cb


@pytest.mark.parametrize("a,b,c", [(4096 + 8, 8192, 16384), (4096, 8192 + 2, 16384), (4096, 8192, 16384 + 2)])
def test_misaligned_pointers_are_refused(a, b, c):
    p = ctypes.c_void_p
    assert cb.lib().casim_b200_sg_gemm(p(a), p(b), 128, 16, 64, p(c)) == cb.EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(128, 16, 64), (256, 256, 128)])
def test_output_on_any_float(cuda_device, M, N, K):
    import torch
    from casim_b200 import surrogate as sg
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    want = sg.gemm(a, b)
    for off in (1, 2, 3):
        buf = torch.full((M * N + 8,), -1.0, device="cuda")
        torch.cuda.synchronize()
        st = cb.lib().casim_b200_sg_gemm(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), M, N, K,
                                         ctypes.c_void_p(buf.data_ptr() + 4 * off))
        assert st == cb.OK
        assert torch.equal(buf[off:off + M * N].reshape(M, N), want)
        assert (buf[:off] == -1).all() and (buf[off + M * N:] == -1).all()
