"""Activations with infinities and NaN on the one-activation tensor-core GEMV, whose digits cannot hold them: every entry, with the
RMSNorm in front, the residual or silu(gate) * up behind, and the two-matrix launch, gives what IEEE arithmetic gives."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import nvfp4_codec_oracle as oc
from tests.gpu_util import dev, ptr, stream

pytestmark = pytest.mark.gpu


def weights(M, K):
    rng = np.random.default_rng(M + K)
    return rng.integers(0, 256, (M, K // 2), dtype=np.uint8), rng.integers(118, 123, (M, K // 16), dtype=np.uint8)


def same(got, want):
    """NaN where the truth has NaN, the same infinities, and the rounding of the output elsewhere."""
    got, want = got.cpu().numpy().astype(np.float64), np.asarray(want, np.float64)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf])
    fin = np.isfinite(want)
    if fin.any():
        assert oc.rel_error_floored(got[fin], want[fin]).max() <= 2e-3


# the last row tile is ragged; a value in the first, an inner and the last stage of K
@pytest.mark.parametrize("entry,M,K", [("launch_nvfp4_gemv_step", 5122, 6144), ("launch_nvfp4_gemv_fused", 8202, 5120),
                                       ("launch_nvfp4_gemv_v8", 8202, 5120)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("at", [0, 2111, -1])
def test_rows_are_those_of_ieee_arithmetic(lib, entry, M, K, bad, at):
    p, s = weights(M, K)
    rng = np.random.default_rng(3)
    x, h = rng.standard_normal(K).astype(np.float16), rng.standard_normal(M).astype(np.float16)
    x[at] = bad
    h[:] = np.where(rng.random(M) < 0.01, np.float16("-inf"), h)
    d_p, d_s, d_x, d_h = dev(p), dev(s), dev(x), dev(h)
    out = torch.zeros(M, dtype=torch.float16, device="cuda")
    with np.errstate(invalid="ignore"):
        y = oc.decode_f64(p, s)[:, at] * float(bad)          # the rest of the sum is finite
        if entry.endswith("v8"):
            assert lib.launch_nvfp4_gemv_v8(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, stream()) == 0
            want = y
        else:
            assert getattr(lib, entry)(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, 0, ctypes.c_void_p(0), 1e-6, 1, ptr(d_h),
                                       stream()) == 0
            want = h.astype(np.float64) + y
    torch.cuda.synchronize()
    same(out, want)
    assert lib.nvfp4_gemv_tc_status(0) == 0


def test_rows_whose_weights_there_are_zero(lib):
    # 0 * inf = NaN, also where a whole block of weights is zero or its scale byte is 0
    M, K = 8202, 5120
    p, s = weights(M, K)
    rng = np.random.default_rng(6)
    p[::2, 160:168] = rng.choice([0, 0x88, 0x80, 0x08], (p[::2].shape[0], 8))     # +0 and -0
    s[1::2, 20] = 0
    x = rng.standard_normal((2, K)).astype(np.float16)
    x[:, 325] = np.inf
    d_p, d_s, d_x = dev(p), dev(s), dev(x)
    out = torch.zeros((3, M), dtype=torch.float16, device="cuda")
    assert lib.launch_nvfp4_gemv_v8(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, stream()) == 0
    assert lib.launch_nvfp4_gemv2(ptr(d_p), ptr(d_s), ptr(d_x), ptr(d_x[1]), ptr(out[1]), M, K, stream()) == 0
    torch.cuda.synchronize()
    assert torch.isnan(out[:, ::2]).all()
    # (a scale byte of 0 is zero, as in every other kernel of the library)
    assert torch.isnan(out[:, 1::2]).all()


def test_norm_in_front_and_activation_behind(lib):
    # a finite activation whose normalised value overflows fp16: an infinity that only the multiplied vector holds
    M, K = 8192, 5120
    p, s = weights(M, K)
    rng = np.random.default_rng(4)
    x, w1 = rng.standard_normal(K).astype(np.float16), np.ones(K, np.float32)
    w1[1234] = 1e9
    d_p, d_s, d_x, d_w = dev(p), dev(s), dev(x), dev(w1)
    col = oc.decode_f64(p, s)[:, 1234]
    with np.errstate(invalid="ignore"):
        y = col * np.inf * np.sign(float(x[1234]))
        out = torch.zeros(M, dtype=torch.float16, device="cuda")
        assert lib.launch_nvfp4_gemv_fused(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, 1, ptr(d_w), 1e-6, 0,
                                           ctypes.c_void_p(0), stream()) == 0
        torch.cuda.synchronize()
        same(out, y)
        out = torch.zeros(M // 2, dtype=torch.float16, device="cuda")
        assert lib.launch_nvfp4_gemv_fused(ptr(d_p), ptr(d_s), ptr(d_x), ptr(out), M, K, 1, ptr(d_w), 1e-6, 2,
                                           ctypes.c_void_p(0), stream()) == 0
        torch.cuda.synchronize()
        g, u = y.reshape(-1, 2, 8)[:, 0], y.reshape(-1, 2, 8)[:, 1]
        same(out, (np.where(np.isneginf(g), np.nan, g) * u).reshape(-1))     # silu(-inf) = -inf / inf
    # an infinite activation: its mean of squares is infinite, the others become 0 and it becomes NaN
    x[77] = np.inf
    out = torch.zeros(M, dtype=torch.float16, device="cuda")
    assert lib.launch_nvfp4_gemv_fused(ptr(d_p), ptr(d_s), ptr(dev(x)), ptr(out), M, K, 1, ptr(d_w), 1e-6, 0,
                                       ctypes.c_void_p(0), stream()) == 0
    torch.cuda.synchronize()
    assert torch.isnan(out).all()


def test_mlp_block(lib):
    hidden, inter = 2560, 8192
    gp, gs = weights(2 * inter, hidden)
    dp, ds = weights(hidden, inter)
    rng = np.random.default_rng(5)
    h0, w1 = rng.standard_normal(hidden).astype(np.float16), np.ones(hidden, np.float32)
    w1[99] = 1e9
    mats = [dev(a) for a in (gp, gs, dp, ds)]
    d_w = dev(w1)
    results = []
    for one in (True, False):
        h, act = dev(h0), torch.zeros(inter, dtype=torch.float16, device="cuda")
        if one:
            rc = lib.launch_nvfp4_mlp_tc(*(ptr(m) for m in mats), ptr(h), ptr(act), ptr(d_w), 1e-6, inter, hidden, stream())
        else:
            rc = lib.launch_nvfp4_gemv_tc_fused(ptr(mats[0]), ptr(mats[1]), ptr(h), ptr(act), 2 * inter, hidden, 1, ptr(d_w),
                                                1e-6, 2, ctypes.c_void_p(0), stream())
            rc |= lib.launch_nvfp4_gemv_tc_fused(ptr(mats[2]), ptr(mats[3]), ptr(act), ptr(h), hidden, inter, 0,
                                                 ctypes.c_void_p(0), 1e-6, 1, ptr(h), stream())
        assert rc == 0
        torch.cuda.synchronize()
        results.append((act.cpu().numpy(), h.cpu().numpy()))
    assert not np.isfinite(results[0][0]).any() and not np.isfinite(results[0][1]).any()
    for a, b in zip(*results):
        assert np.array_equal(a, b, equal_nan=True)
    assert lib.nvfp4_gemv_tc_status(0) == 0
