"""Two activations through the tensor-core GEMV: shapes from one stage and one row to all K splits, both layouts of the
activations, extreme values, and launches on several streams."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_codec_oracle as oc
from tests.gpu_util import dev, gemv2, gemv2i, ptr, stream

pytestmark = pytest.mark.gpu


def weights(M, K, seed=0):
    rng = np.random.default_rng(seed + M + K)
    return rng.integers(0, 256, (M, K // 2), dtype=np.uint8), rng.integers(118, 123, (M, K // 16), dtype=np.uint8)


def check(y, p, s, a):
    ref = oc.gemv_f64(p, s, a)
    assert oc.rel_error_floored(y, ref).max() <= 1e-3       # the fp16 rounding of the output is 4.9e-4


# K splits of 1 to 8 CTAs, ragged row tiles, splits that do not divide the stages; then shapes around the line to the other
# kernel (K of 11 and 12 stages, too many tiles for one round)
@pytest.mark.parametrize("M,K", [(3000, 3584), (6144, 5120), (5120, 6144), (700, 17408), (5120, 17408), (10240, 3072),
                                 (13000, 3072), (20000, 3072), (37000, 3072), (4000, 2816), (40000, 3072), (1, 256), (1000, 768)])
def test_two_activations(lib, M, K):
    p, s = weights(M, K)
    rng = np.random.default_rng(1)
    a0 = rng.standard_normal(K).astype(np.float16)
    a1 = (rng.standard_normal(K) * 2.0 ** rng.integers(-12, 6, K)).astype(np.float16)
    a1[:16] = 0
    a1[16:32] = np.float16(6e-8)                             # subnormal
    rc, y = gemv2(lib, p, s, a0, a1)
    assert rc == 0
    check(y[0], p, s, a0)
    check(y[1], p, s, a1)
    rc, y2 = gemv2i(lib, p, s, a0, a1)
    assert rc == 0 and np.array_equal(y.view(np.uint16), y2.view(np.uint16))
    rc, swapped = gemv2(lib, p, s, a1, a0)
    assert rc == 0 and np.array_equal(swapped[0].view(np.uint16), y[1].view(np.uint16))
    assert np.array_equal(swapped[1].view(np.uint16), y[0].view(np.uint16))
    assert lib.nvfp4_gemv_tc_status(0) == 0


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("at", [0, 777, 5119])
def test_an_activation_that_is_not_finite(lib, bad, at):
    # what IEEE arithmetic gives: a row is +-inf or NaN by its weight there, the other activation is untouched
    M, K = 2050, 5120
    p, s = weights(M, K)
    rng = np.random.default_rng(2)
    a0, a1 = rng.standard_normal(K).astype(np.float16), rng.standard_normal(K).astype(np.float16)
    rc, clean = gemv2(lib, p, s, a0, a1)
    assert rc == 0
    b1 = a1.copy()
    b1[at] = bad
    rc, y = gemv2(lib, p, s, a0, b1)
    assert rc == 0 and np.array_equal(y[0].view(np.uint16), clean[0].view(np.uint16))
    w = oc.decode_f64(p, s)[:, at]
    with np.errstate(invalid="ignore"):
        want = w * bad                                       # 0 * inf = NaN
    assert np.array_equal(np.isnan(y[1]), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(y[1][ok].astype(np.float64), want[ok])


def test_streams_share_nothing(lib):
    jobs = []
    for i, (M, K) in enumerate([(5120, 17408), (1024, 5120), (17408, 5120), (6144, 5120)]):
        p, s = weights(M, K, i)
        x = np.random.default_rng(i).standard_normal((2, K)).astype(np.float16)
        jobs.append((M, K, dev(p), dev(s), dev(x), torch.zeros((2, M), dtype=torch.float16, device="cuda"), torch.cuda.Stream()))

    def call(M, K, p, s, x, out):
        assert lib.launch_nvfp4_gemv2(ptr(p), ptr(s), ptr(x), ptr(x[1]), ptr(out), M, K, stream()) == 0

    want = []
    for *j, st in jobs:
        call(*j)
        torch.cuda.synchronize()
        want.append(j[-1].clone())
        j[-1].zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for *j, st in jobs:
            with torch.cuda.stream(st):
                call(*j)
    torch.cuda.synchronize()
    for (*j, st), w in zip(jobs, want):
        assert torch.equal(j[-1], w)
    assert lib.nvfp4_gemv_tc_status(0) == 0
