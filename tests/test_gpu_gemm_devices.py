"""The GEMM's shared-memory limit is set on every device it runs on, from
whichever thread gets there first."""

import ctypes as C
import threading

import pytest

from kinectfusion_b200 import abi

pytestmark = pytest.mark.gpu

SHAPES = [(130, 16, 64), (130, 32, 64), (130, 64, 64), (200, 128, 128), (600, 300, 256)]


def products(device):
    """Whether each tile width's product is the FP32 one, on `device`."""
    import torch
    torch.cuda.set_device(device)
    ok = []
    for m, n, k in SHAPES:
        g = torch.Generator(device="cuda").manual_seed(m + n + k)
        a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
        b = torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16)
        c = torch.empty(m, n, device="cuda")
        abi.check(abi.load().kf_gemm_bf16(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr()),
                                          m, n, k, None, 0, None))
        want = a.double() @ b.double().T
        scale = a.double().abs() @ b.double().abs().T
        ok.append(bool(((c.double() - want).abs() <= (k + 2) * 2.0 ** -24 * scale).all()))
    return ok


def test_threads_on_one_device():
    results = [None] * 4
    threads = [threading.Thread(target=lambda i=i: results.__setitem__(i, products(0))) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert results == [[True] * len(SHAPES)] * 4


def test_a_second_device():
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    assert products(0) == [True] * len(SHAPES)
    assert products(1) == [True] * len(SHAPES)
    assert products(0) == [True] * len(SHAPES)
