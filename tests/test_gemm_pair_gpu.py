"""The W4A16 GEMM on CTA pairs (more than 128 tokens) against float64 at the edges of its tiles."""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def pairs_for_every_shape(lib):
    lib.nvfp4_b200_gemm_config(7)            # by default short K goes to 256-row tiles where those fill the GPU
    yield
    lib.nvfp4_b200_gemm_config(3)


@pytest.mark.parametrize("M,n,K", [
    (256, 129, 256),        # one pair, one weight stage, one token past the few-token kernel
    (257, 192, 512),        # a pair with one row in its first CTA only; exactly one 192-token tile
    (128, 193, 1280),       # second CTA without rows; ring of stages used more than once
    (6000, 257, 2304),      # one token past a tile of 256
    (5120, 512, 1024),      # 192-token tiles (60 pairs), the last one ragged
    (20000, 520, 256),      # 256-token tiles, several rounds of pairs
])
@pytest.mark.parametrize("flags", [0, 1, 2, 3, 6, 7])
def test_against_float64(lib, M, n, K, flags):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + n + K)
    p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.randint(118, 123, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
    x = torch.randn((n, K), device="cuda", generator=g).half()
    n8 = (n + 7) // 8 * 8
    if flags & 1:
        act, ld_act = x, K
    else:
        act, ld_act = torch.zeros((K, n8), dtype=torch.float16, device="cuda"), n8
        act[:, :n] = x.t()
    shape, ld_out = ((n, M), M) if flags & 2 else ((M, n8), n8)
    old = torch.randn(shape, device="cuda", generator=g).half()
    out = torch.cat([old.flatten(), torch.full((64,), 7.0, dtype=torch.float16, device="cuda")])
    rc = lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(act), ld_act, ptr(out), ld_out, M, n, K, flags, stream())
    torch.cuda.synchronize()
    assert rc == 0 and lib.nvfp4_gemm_status(0) == 0
    assert (out[-64:] == 7).all()
    got = out[:-64].view(shape).double()
    if not flags & 2:
        assert (got[:, n:] == 0).all()          # padded tokens are zero activations
        got = got[:, :n].t()

    codes = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    codes = torch.cat([codes, -codes])
    w = torch.stack([codes[(p & 15).long()], codes[(p >> 4).long()]], -1).view(M, K)
    w = w * torch.exp2(s.double() - 127).repeat_interleave(16, 1)
    want, size = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    # products are exact; fp32 sums of K terms lose at most 2^-20 of the sum of magnitudes here, the
    # result is rounded to fp16 once, with a residual added twice
    bound = want.abs() * 2 ** -11 + size * 2 ** -20 + 2 ** -24
    if flags & 4:
        want = want + old.double()
        bound = bound + want.abs() * 2 ** -11
    assert ((got - want).abs() <= bound * 1.001).all(), ((got - want).abs() / bound).max().item()


@pytest.mark.parametrize("M,n,K", [
    (20000, 520, 512), (20000, 520, 2560), (20000, 520, 5120),      # tiles, tiles or pairs by output layout, pairs
    (10240, 1000, 256), (4096, 2048, 1024),                         # last rounds nearly empty and full
])
@pytest.mark.parametrize("flags", [0, 1, 2, 3, 6, 7])
def test_the_choice_does_not_show(lib, M, n, K, flags):
    # whichever kernel the shape and the output layout get: the same bits
    g = torch.Generator(device="cuda")
    g.manual_seed(M + K)
    p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.randint(118, 123, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
    n8 = (n + 7) // 8 * 8
    act = torch.randn((n, K) if flags & 1 else (K, n8), device="cuda", generator=g).half()
    shape = (n, M) if flags & 2 else (M, n8)
    old = torch.randn(shape, device="cuda", generator=g).half()
    outs = []
    for config in (7, 3, 1):
        lib.nvfp4_b200_gemm_config(config)
        outs.append(old.clone())
        assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(act), act.shape[1], ptr(outs[-1]), shape[1], M, n, K,
                                              flags, stream()) == 0
    torch.cuda.synchronize()
    assert lib.nvfp4_gemm_status(0) == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
