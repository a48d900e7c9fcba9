"""Two outputs of the GEMM's epilogue and of its split-K reduction:

* products without a bias, with and without ReLU, direct and split, against
  FP64 products of the same bf16 operands: both sides sum exact products, so
  they differ by at most the rounding of K additions, K * 2^-24 of the sum of
  the products' magnitudes;
* the bf16 copy that the learner's layers read: its forward pass equals, bit
  for bit, the same layers taken one by one through kf_gemm_bf16 with the FP32
  activations rounded to bf16 outside.  The first dense layer's GEMM is split
  along K at the smaller batches and not at the largest."""

import ctypes as C

import numpy as np
import pytest

import kf_learn_oracle as lo
from kinectfusion_b200 import abi, learned

pytestmark = pytest.mark.gpu


def gemm(a, b, bias, relu):
    import torch
    c = torch.full((a.shape[0] + 1, b.shape[0]), 7.0, device="cuda")  # one row more: nothing past the product is written
    abi.check(abi.load().kf_gemm_bf16(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr()),
                                      a.shape[0], b.shape[0], a.shape[1],
                                      None if bias is None else C.c_void_p(bias.data_ptr()), relu, None))
    assert (c[-1] == 7.0).all()
    return c[:-1]


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 1, 8), (129, 17, 72), (31, 33, 2048), (128, 64, 64), (257, 127, 288),
                                   (64, 129, 1280), (5000, 288, 32)])
def test_without_bias(m, n, k, relu):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16)
    want = a.double() @ b.double().T
    if relu:
        want = want.clamp(min=0)
    scale = a.double().abs() @ b.double().abs().T
    assert ((gemm(a, b, None, relu).double() - want).abs() <= (k + 2) * 2.0 ** -24 * scale).all()


@pytest.mark.parametrize("batch", [8, 72, 9472])
def test_bf16_copy_is_the_rounded_result(batch):
    import torch
    params = lo.init_params(13)
    net = learned.Learner(batch, seed=1)
    net.set_params(params)
    weights, biases = lo.unpack(params)
    x = (0.5 * torch.randn(batch, 60, 80, 2, generator=torch.Generator(device="cuda").manual_seed(batch),
                           device="cuda")).to(torch.bfloat16)
    h = x
    for layer in range(6):
        if layer < 4:
            cin, cout, _, _, hout, wout, k, kpad = lo.CONV[layer]
            pad = torch.nn.functional.pad(h.reshape(batch, *lo.CONV[layer][2:4], cin), (0, 0, 1, 1, 1, 1))
            col = torch.zeros(batch, hout, wout, kpad, dtype=torch.bfloat16, device="cuda")
            for ky in range(3):
                for kx in range(3):
                    col[..., ky * 3 + kx:k:9] = pad[:, ky:ky + 2 * hout:2, kx:kx + 2 * wout:2, :]
            h = col.reshape(batch * hout * wout, kpad)
        else:
            h = h.reshape(batch, -1)
        w = torch.from_numpy(np.ascontiguousarray(weights[layer])).cuda().to(torch.bfloat16)
        y = gemm(h.contiguous(), w, torch.from_numpy(np.ascontiguousarray(biases[layer])).cuda(), int(layer < 5))
        h = y.to(torch.bfloat16)
    got = net.forward(x)
    torch.cuda.synchronize()
    assert torch.equal(got, y) and bool((y != 0).any())
