"""Scale bytes at the ends of their range (0 is zero, 255 is infinity, 254 is 2^127) on the tensor-core GEMVs, whose matrix
instruction reads 0 as 2^-127 and 255 as NaN: the same rows as the register-streaming kernel's."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_codec_oracle as oc
from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu


def call(lib, entry, d_p, d_s, d_x, out, M, K):
    if entry == "launch_nvfp4_gemv2":
        return lib.launch_nvfp4_gemv2(ptr(d_p), ptr(d_s), ptr(d_x), ptr(d_x[1]), ptr(out), M, K, stream())
    if entry == "launch_nvfp4_gemv2i":
        return lib.launch_nvfp4_gemv2i(ptr(d_p), ptr(d_s), ptr(d_x.t().contiguous()), ptr(out), M, K, stream())
    return lib.launch_nvfp4_gemv_v8(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, stream())


@pytest.mark.parametrize("entry", ["launch_nvfp4_gemv_v8", "launch_nvfp4_gemv2", "launch_nvfp4_gemv2i"])
def test_ends_of_the_range(lib, entry):
    M, K = 8202, 5120
    rng = np.random.default_rng(8)
    p = rng.integers(0, 256, (M, K // 2), dtype=np.uint8)
    s = rng.integers(118, 123, (M, K // 16), dtype=np.uint8)
    at = rng.integers(0, K // 16, M)
    kind = np.arange(M) % 5                                  # 0: byte 0, 1: 254, 2: 255, 3: 255 over zeros, 4: usual
    for k, byte in ((0, 0), (1, 254), (2, 255), (3, 255)):
        rows = np.nonzero(kind == k)[0]
        s[rows, at[rows]] = byte
        if k == 3:
            p[rows[:, None], at[rows][:, None] * 8 + np.arange(8)] = 0
    x = (rng.integers(-64, 65, (2, K)) / 8).astype(np.float16)       # a block's sum is exact in any order, so its sign is too
    d_p, d_s, d_x = dev(p), dev(s), dev(x)
    two = entry != "launch_nvfp4_gemv_v8"
    got, plain = (torch.zeros((1 + two, M), dtype=torch.float16, device="cuda") for _ in range(2))
    assert call(lib, entry, d_p, d_s, d_x, got, M, K) == 0
    assert lib.nvfp4_b200_gemv_config(4, 0, 0) == 0          # a forced warp count keeps to the register-streaming kernel
    try:
        assert call(lib, entry, d_p, d_s, d_x, plain, M, K) == 0
    finally:
        assert lib.nvfp4_b200_gemv_config(0, 0, 0) == 0
    torch.cuda.synchronize()
    got, plain = got.cpu().numpy().astype(np.float64), plain.cpu().numpy().astype(np.float64)
    assert np.isnan(plain[:, kind == 3]).all() and np.isinf(plain[:, kind == 2]).mean() > 0.99
    assert np.isinf(plain[:, kind == 1]).mean() > 0.99 and np.isfinite(plain[:, (kind == 0) | (kind == 4)]).all()
    assert np.array_equal(np.isnan(got), np.isnan(plain)) and np.array_equal(got[np.isinf(plain)], plain[np.isinf(plain)])
    fin = np.isfinite(plain)
    assert oc.rel_error_floored(got[fin], plain[fin]).max() <= 2e-3
    assert lib.nvfp4_gemv_tc_status(0) == 0
