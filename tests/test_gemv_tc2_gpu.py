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


# K splits of 1 to 8 CTAs on the tensor-core kernel, ragged row tiles, splits that do not divide the stages; then shapes that
# the other kernel keeps (split 0): one round of row tiles with a short K, one tile an SM, two rounds, three with no split,
# K of 11 stages, too many tiles for one round of clusters, the smallest
@pytest.mark.parametrize("M,K,split", [(3000, 8192, 8), (3000, 5376, 7), (5500, 6144, 6), (6144, 5120, 5), (5120, 6144, 6),
                                       (5120, 17408, 6), (8000, 5120, 4), (8900, 4096, 4), (9216, 4096, 3), (10240, 4096, 3),
                                       (13000, 6144, 2), (17000, 3072, 2), (28000, 3072, 1), (37000, 3072, 1),
                                       (3000, 3584, 0), (6144, 3072, 0), (700, 17408, 0), (2368, 5120, 0), (10240, 3072, 0),
                                       (12288, 5120, 0), (20000, 3072, 0), (25000, 2816, 0), (40000, 3072, 0), (1, 256, 0),
                                       (1000, 768, 0)])
def test_two_activations(lib, M, K, split):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert lib.nvfp4_gemv_tc2_split(M, K) == split
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
    M, K = 2450, 5120
    assert lib.nvfp4_gemv_tc2_split(M, K) > 0
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
        assert (lib.nvfp4_gemv_tc2_split(M, K) > 0) == (M > 1024)
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
