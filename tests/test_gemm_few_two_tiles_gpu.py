"""The W4A16 GEMM of 129 to 256 tokens on narrow matrices (two column tiles of the few-token kernel) against float64."""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,n,K", [
    (128, 129, 256),        # one row tile, one stage, one token in the second column tile
    (300, 200, 512),        # ragged rows and tokens
    (2560, 193, 1024),      # the widest with a short K; a token past 64 in the second tile
    (5120, 136, 6144),      # K split over three
    (4608, 200, 3072),      # 72 tiles, which clusters of four CTAs do not hold
    (5376, 255, 3072),      # the widest of all
    (1000, 256, 17408),     # K split over eight
])
def test_against_float64(lib, M, n, K):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + n + K)
    p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.randint(118, 123, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
    x = torch.randn((n, K), device="cuda", generator=g).half()
    n8 = (n + 7) // 8 * 8
    xt = torch.zeros((K, n8), dtype=torch.float16, device="cuda")
    xt[:, :n] = x.t()
    codes = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    codes = torch.cat([codes, -codes])
    w = torch.stack([codes[(p & 15).long()], codes[(p >> 4).long()]], -1).view(M, K)
    w = w * torch.exp2(s.double() - 127).repeat_interleave(16, 1)
    want, size = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    # products are exact; fp32 sums of K terms lose at most 2^-20 of the sum of magnitudes here, the
    # result is rounded to fp16 once, with a residual added twice
    bound = want.abs() * 2 ** -11 + size * 2 ** -20 + 2 ** -24
    plain = None
    for flags in (0, 1, 2, 3, 6, 7):
        act, ld = (x, K) if flags & 1 else (xt, n8)
        shape = (n, M) if flags & 2 else (M, n8)
        old = torch.randn(shape, device="cuda", generator=g).half()
        out = torch.cat([old.flatten(), torch.full((64,), 7.0, dtype=torch.float16, device="cuda")])
        assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(act), ld, ptr(out), shape[1], M, n, K, flags, stream()) == 0
        torch.cuda.synchronize()
        assert lib.nvfp4_gemm_status(0) == 0
        assert (out[-64:] == 7).all()
        got = out[:-64].view(shape)
        if not flags & 2:
            assert (got[:, n:] == 0).all()
            got = got[:, :n].t()
        extra, ref = 0, want
        if flags & 4:
            ref = want + old.double()
            extra = ref.abs() * 2 ** -11
        assert ((got.double() - ref).abs() <= (bound + extra) * 1.001).all(), flags
        if not flags & 4:                                  # the layouts differ in nothing else
            assert plain is None or torch.equal(plain, got)
            plain = got.clone()
    if n == n8:
        out = torch.zeros((M, n), dtype=torch.float16, device="cuda")
        assert lib.launch_nvfp4_gemmtc_v5(ptr(p), ptr(s), ptr(xt), ptr(out), M, n, K, stream()) == 0
        torch.cuda.synchronize()
        assert torch.equal(out.t(), plain)
