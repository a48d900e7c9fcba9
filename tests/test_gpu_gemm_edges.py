"""The GEMM's row-wise epilogue at the edges of its 128-row tiles, its column
tiles and its 32 x 32 turns, with and without bias, ReLU and a split K,
against FP32 products of the same bf16 operands.  Both sides sum exact
products in FP32, so they differ by at most the rounding of K additions:
K * 2^-24 of the sum of the products' magnitudes."""

import ctypes as C

import pytest

from kinectfusion_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,relu", [
    (1, 1, 8, 0), (127, 15, 24, 1), (128, 16, 64, 0), (129, 17, 72, 1), (31, 33, 2048, 0), (33, 63, 1032, 1),
    (160, 65, 40, 1), (257, 127, 288, 0), (64, 129, 1280, 1), (5000, 288, 32, 0), (38000, 257, 32, 1),
])
def test_gemm_edges(m, n, k, relu):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(n, generator=g, device="cuda")
    c = torch.full((m + 1, n), 7.0, device="cuda")  # one row more: nothing past the product is written
    abi.check(abi.load().kf_gemm_bf16(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr()),
                                      m, n, k, C.c_void_p(bias.data_ptr()), relu, None))
    want = a.double() @ b.double().T + bias.double()
    scale = a.double().abs() @ b.double().abs().T + bias.double().abs()
    if relu:
        want = want.clamp(min=0)
    assert ((c[:m].double() - want).abs() <= (k + 2) * 2.0 ** -24 * scale).all()
    assert (c[m] == 7.0).all()
