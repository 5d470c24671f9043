"""Bit 1 of nvfp4_b200_gemv_config: a GEMV right behind the kernel that writes its weights, on every kernel that can take it."""
import ctypes

import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu

M, K = 17408, 5120


def two(lib, p, s, x, y):
    return lib.launch_nvfp4_gemv2(ptr(p), ptr(s), ptr(x[0]), ptr(x[1]), ptr(y), M, K, stream())


def two_interleaved(lib, p, s, x, y):
    return lib.launch_nvfp4_gemv2i(ptr(p), ptr(s), ptr(x), ptr(y), M, K, stream())


def plain(lib, p, s, x, y):
    return lib.launch_nvfp4_gemv_v8(ptr(p), ptr(s), ptr(x), ptr(y), M, K, stream())


def fused(entry):
    return lambda lib, p, s, x, y: getattr(lib, entry)(ptr(p), ptr(s), ptr(x), ptr(y), M, K, 0, ctypes.c_void_p(0), 1e-6, 0,
                                                       ctypes.c_void_p(0), stream())


@pytest.mark.parametrize("call", [two, two_interleaved, plain, fused("launch_nvfp4_gemv_fused"),
                                  fused("launch_nvfp4_gemv_step")],
                         ids=["gemv2", "gemv2i", "v8", "fused", "step"])
def test_weights_written_by_the_kernel_in_front(lib, call):
    # A row copy (launch_embed_rows) lets its successor start at once; without the bit the GEMV's first stages of weights
    # would be those that were there before.
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    weights = torch.randint(0, 256, (2 * M, K // 2), dtype=torch.uint8, device="cuda", generator=g)     # two matrices
    rows = [torch.arange(i * M, (i + 1) * M, dtype=torch.int64, device="cuda") for i in range(2)]
    x = torch.randn((2, K), device="cuda", generator=g).half()
    p = torch.zeros((M, K // 2), dtype=torch.uint8, device="cuda")
    s = torch.randint(118, 123, (M * K // 16,), dtype=torch.uint8, device="cuda", generator=g)
    write = lambda i: lib.launch_embed_rows(ptr(weights), ptr(rows[i]), ptr(p), M, K // 4, 2 * M, stream())
    y = torch.zeros((2, M), dtype=torch.float16, device="cuda")
    want = []
    for i in range(2):
        assert write(i) == 0
        torch.cuda.synchronize()
        assert torch.equal(p, weights[i * M:(i + 1) * M])
        assert call(lib, p, s, x, y) == 0
        torch.cuda.synchronize()
        want.append(y.clone())
    assert not torch.equal(*want)
    assert lib.nvfp4_b200_gemv_config(0, 0, 2) == 0
    try:
        for i in (0, 1, 0, 1):
            assert write(i) == 0 and call(lib, p, s, x, y) == 0
            torch.cuda.synchronize()
            assert torch.equal(y, want[i])
    finally:
        assert lib.nvfp4_b200_gemv_config(0, 0, 0) == 0
