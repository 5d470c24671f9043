"""Chunk attention on the tensor cores against float64 and, for infinities and NaN, against the
decode kernel run once per token."""
import numpy as np
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu
D = 256


def _inputs(n, p0, hq, hkv, max_len, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, gate = r(n, hq * D).half(), r(n, hq * D).half()
    keys, vals = r(hkv, max_len, D).half(), r(hkv, max_len, D).half()
    # rows no token of the chunk may see hold whatever was there before
    keys[:, p0 + n:] = float("nan")
    vals[:, p0 + n:] = float("inf")
    return q, gate, keys, vals


def _run(lib, q, keys, vals, p0, n, gate, hq, hkv, scale):
    out = torch.full((n, hq * D), 7.0, dtype=torch.float16, device="cuda")
    rc = lib.launch_attn_prefill(ptr(q), ptr(keys), ptr(vals), p0 + 1, n, ptr(gate), ptr(out),
                                 keys.shape[1], hq, hkv, scale, stream())
    torch.cuda.synchronize()
    assert rc == 0 and lib.nvfp4_gemm_status(0) == 0
    return out


@pytest.mark.parametrize("n,p0,hq,hkv,max_len,scale", [
    (64, 0, 2, 1, 64, 1 / 16),          # one key step, half masked
    (65, 63, 2, 1, 200, 1 / 16),        # one token past a tile; last key = first of a step
    (21, 235, 24, 4, 256, 1 / 16),      # one tile of 126 rows, keys split in two
    (22, 300, 24, 4, 512, 1 / 4),       # ragged second tile; peaked weights, growing maxima
    (1, 4095, 24, 4, 4096, 1 / 16),     # one token, keys split as far as they go
    (130, 0, 5, 5, 130, 1 / 16),        # no shared heads: 128 + 2 tokens
    (43, 1000, 9, 3, 1100, 1.0),        # 42 tokens a tile; weights on very few keys
    (512, 3488, 24, 4, 4100, 1 / 16),   # the last chunk of a long document
    (1024, 0, 6, 1, 1024, 1 / 16),
    (64, 0, 12, 6, 64, 1 / 16),         # (the first two shapes with enough heads for this kernel)
    (65, 63, 12, 6, 200, 1 / 16),
])
def test_against_float64(lib, n, p0, hq, hkv, max_len, scale):
    q, gate, keys, vals = _inputs(n, p0, hq, hkv, max_len, n + p0)
    out = _run(lib, q, keys, vals, p0, n, gate, hq, hkv, scale)
    again = _run(lib, q, keys, vals, p0, n, gate, hq, hkv, scale)
    assert torch.equal(out, again)
    L = p0 + n
    mask = torch.arange(L, device="cuda")[None, :] > (p0 + torch.arange(n, device="cuda"))[:, None]
    for h in range(hq):
        k, v = keys[h // (hq // hkv), :L].double(), vals[h // (hq // hkv), :L].double()
        s = (q[:, h * D:(h + 1) * D].double() @ k.T * scale).masked_fill(mask, -float("inf"))
        o = torch.softmax(s, -1) @ v
        sg = torch.sigmoid(gate[:, h * D:(h + 1) * D].double()).half()
        want = (o.half().double() * sg.double())
        got = out[:, h * D:(h + 1) * D].double()
        # one fp16 step in the rounded sum and one in the product, and the fp32 sums: a score of
        # size |s| carries |s| 2^-22, which moves its weight by as much
        bound = want.abs() * 2 ** -9 + v.abs().max() * (2 ** -20 + s[~mask].abs().max() * 2 ** -21)
        assert ((got - want).abs() <= bound).all(), (h, ((got - want).abs() / bound).max().item())


@pytest.mark.parametrize("hq,hkv", [(6, 2), (12, 4)])           # one query at a time; tensor cores
def test_infinities_and_nan_as_the_decode_kernel(lib, hq, hkv):
    # a later token's value never reaches an earlier one, an unmasked one does as in fp32
    n, p0, scale = 70, 130, 1 / 16
    q, gate, keys, vals = _inputs(n, p0, hq, hkv, 256, 3)
    vals[0, 150, 3] = float("inf")
    vals[0, 170, 5] = -float("inf")
    vals[1, 190, 7] = float("nan")
    keys[1, 160, 0] = float("inf")
    keys[1, 180] = 60000.0
    out = _run(lib, q, keys, vals, p0, n, gate, hq, hkv, scale).cpu().numpy()
    for t in range(n):
        ln = torch.tensor([p0 + t + 1], dtype=torch.int64, device="cuda")
        o = torch.zeros(hq * D, dtype=torch.float16, device="cuda")
        qt, gt = q[t].contiguous(), gate[t].contiguous()
        assert lib.launch_attn_decode_heads(ptr(qt), ptr(keys), ptr(vals), ptr(ln), ptr(gt), ptr(o), 256,
                                            hq, hkv, scale, stream()) == 0
        want = o.cpu().numpy()
        assert np.array_equal(np.isnan(out[t]), np.isnan(want)), t
        assert np.array_equal(np.isinf(out[t]), np.isinf(want)), t
        fin = np.isfinite(want)
        assert np.allclose(out[t][fin].astype(np.float64), want[fin].astype(np.float64), rtol=2 ** -9, atol=2 ** -14), t


@pytest.mark.parametrize("n,p0", [(512, 512), (512, 1536), (512, 3488), (256, 3800)])
def test_accumulation_stays_short(lib, n, p0):
    # Tensor-core sums truncate: 2 MMAs per 16 keys lose 2^-24 of the sum each on average.  Over at most 1024
    # keys a CTA that is 128 losses, half of them from a sum that has still to grow: 2^-18, and against the
    # fp16 step (2^-10 to 2^-11 of the value) 4 to 8 outputs in 1000 then round the other way, next to 2 or
    # 3 from the scores.  (All keys in one accumulation: 16 to 25 in 1000 at 2500 to 4000 keys.)
    hq, hkv, scale = 24, 4, 1 / 16
    q, gate, keys, vals = _inputs(n, p0, hq, hkv, p0 + n, n + p0)
    out = _run(lib, q, keys, vals, p0, n, gate, hq, hkv, scale)
    mask = torch.arange(p0 + n, device="cuda")[None, :] > (p0 + torch.arange(n, device="cuda"))[:, None]
    other = 0
    for h in range(hq):
        k, v = keys[h // 6].double(), vals[h // 6].double()
        sl = slice(h * D, (h + 1) * D)
        o = torch.softmax((q[:, sl].double() @ k.T * scale).masked_fill(mask, -float("inf")), -1) @ v
        other += (out[:, sl] != (o.half().double() * torch.sigmoid(gate[:, sl].double()).half().double()).half()).sum().item()
    assert other <= 0.011 * out.numel(), other / out.numel()


@pytest.mark.parametrize("n,p0,hq,hkv,same", [
    (64, 0, 6, 1, True), (46, 46, 12, 2, True), (24, 150, 24, 4, True), (128, 0, 1, 1, True),
    (64, 0, 24, 4, False), (32, 98, 24, 4, False), (16, 300, 6, 1, False),
])
def test_few_heads_keep_the_decode_kernels_bits(lib, n, p0, hq, hkv, same):
    # both sides of the line below which a chunk goes through the kernel with the decode kernel's arithmetic
    q, gate, keys, vals = _inputs(n, p0, hq, hkv, p0 + n, n)
    out = _run(lib, q, keys, vals, p0, n, gate, hq, hkv, 1 / 16)
    want = torch.empty_like(out)
    for t in range(n):
        ln = torch.tensor([p0 + t + 1], dtype=torch.int64, device="cuda")
        qt, gt = q[t].contiguous(), gate[t].contiguous()
        assert lib.launch_attn_decode_heads(ptr(qt), ptr(keys), ptr(vals), ptr(ln), ptr(gt), ptr(want[t]), p0 + n,
                                            hq, hkv, 1 / 16, stream()) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, want) == same
    # one fp16 step in the rounded sum and one in the product, sums in another order (see above; scores below 8)
    bound = want.double().abs() * 2 ** -9 + 2 * vals.double().abs().max() * (2 ** -20 + 8 * 2 ** -21)
    assert ((out.double() - want.double()).abs() <= bound).all()
