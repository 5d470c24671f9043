"""The FP4 GEMM on CTA pairs at the sizes where its tiles (256 rows x 192 or 256 tokens), its boxes of scale bytes (four
stages of 256 k), its ring and its stores end: bit-identical to the single-CTA kernel, which the oracle pins."""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu


def operands(M, K, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + 3 * K + 7 * n)
    r = lambda lo, hi, *s: torch.randint(lo, hi, s, dtype=torch.uint8, device="cuda", generator=g)
    return r(0, 256, M, K // 2), r(102, 122, M, K // 16), r(0, 256, n, K // 2), r(102, 122, n, K // 16)


def run(lib, ops, M, K, n, ld, config):
    lib.nvfp4_b200_gemm_fp4_config(config)
    try:
        out = torch.full(((M + 1) * ld,), float("nan"), dtype=torch.float16, device="cuda")
        p, s, ap, a_s = ops
        assert lib.launch_nvfp4_gemm_fp4(ptr(p), ptr(s), ptr(ap), ptr(a_s), ptr(out), M, n, K, ld, stream()) == 0
        torch.cuda.synchronize()
        return out.view(torch.int16)
    finally:
        lib.nvfp4_b200_gemm_fp4_config(3)


# K: one stage (a box whose other places stay empty), 2, 3, 5, 9 and 20 stages; M and n at the edges of tiles and of 32;
# pitches of the output that TMA stores take (a multiple of 8) and do not take; many tiles a pair (the last three)
@pytest.mark.parametrize("M,K,n,ld", [(256, 256, 192, 192), (129, 256, 129, 136), (257, 512, 193, 193), (130, 768, 385, 392),
                                      (300, 1280, 256, 256), (512, 2304, 257, 264), (5120, 1024, 200, 203),
                                      (640, 5120, 1000, 1000), (20000, 256, 400, 400), (9000, 1280, 1111, 1112),
                                      (2048, 768, 8192, 8192)])
@pytest.mark.parametrize("tile", [192, 256])
def test_pairs_equal_the_single_cta_kernel(lib, M, K, n, ld, tile):
    ops = operands(M, K, n)
    want = run(lib, ops, M, K, n, ld, 0)
    got = run(lib, ops, M, K, n, ld, 4 | (32 if tile == 192 else 16))
    assert torch.equal(want, got)
    rows = want.view(M + 1, ld)
    nan = torch.full((1,), float("nan"), dtype=torch.float16).view(torch.int16).item()
    assert (rows[M] == nan).all() and (rows[:M, n:] == nan).all()          # nothing past the last row or token
    assert lib.nvfp4_gemm_fp4_status(0) == 0


# Few deep tiles: K in parts.  From 65 tokens on pairs add the parts that the single-CTA kernel's CTAs have, in the same order;
# parts that do not divide K, one row tile, several column tiles, an output that TMA stores do not take.
@pytest.mark.parametrize("M,K,n,ld", [(128, 10240, 65, 72), (100, 10496, 129, 136), (1024, 10240, 128, 128),
                                      (5120, 10240, 256, 256), (5120, 17408, 200, 203), (300, 12288, 1000, 1000)])
def test_few_deep_tiles_run_on_pairs(lib, M, K, n, ld):
    ops = operands(M, K, n)
    want = run(lib, ops, M, K, n, ld, 1)
    for _ in range(3):
        assert torch.equal(run(lib, ops, M, K, n, ld, 3), want)
    rows = want.view(M + 1, ld)
    nan = torch.full((1,), float("nan"), dtype=torch.float16).view(torch.int16).item()
    assert (rows[M] == nan).all() and (rows[:M, n:] == nan).all()
    assert lib.nvfp4_gemm_fp4_status(0) == 0


@pytest.mark.parametrize("M,K,n", [(1024, 17408, 100), (1024, 17408, 200)])
def test_few_deep_tiles_against_float64(lib, M, K, n):
    # Scale bytes over 12 binades on both sides, so that sums do not fit fp32.  The tensor core truncates the sum that it
    # adds to: eight parts of K leave an eighth of the truncations of one accumulation over all of it, so at most half
    # of the results that are not the correctly rounded ones.
    g = torch.Generator(device="cuda")
    g.manual_seed(M + n)
    r = lambda lo, hi, *s: torch.randint(lo, hi, s, dtype=torch.uint8, device="cuda", generator=g)
    ops = r(0, 256, M, K // 2), r(110, 122, M, K // 16), r(0, 256, n, K // 2), r(110, 122, n, K // 16)
    lut = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    lut = torch.cat([lut, -lut])

    def decode(p, s):
        w = lut[torch.stack([p & 15, p >> 4], -1).view(p.shape[0], -1).long()]
        return w * torch.exp2(s.double() - 127).repeat_interleave(16, 1)

    want = (decode(*ops[:2]) @ decode(*ops[2:]).t()).half()
    ld = (n + 7) // 8 * 8
    wrong = {c: (run(lib, ops, M, K, n, ld, c).view(torch.float16).view(M + 1, ld)[:M, :n] != want).double().mean().item()
             for c in (0, 3)}
    assert wrong[3] <= 0.5 * wrong[0], wrong
