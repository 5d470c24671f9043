"""The chunk kernels of the Gated DeltaNet and the row-wise silu-mul at the sizes where their tiles
end: blocks of 4 tokens, operand stages of 16, conv strips of 2 or 8 tokens, 2- or 8-token accesses."""
import numpy as np
import pytest
import torch

from oracle import fused_ops_oracle as fo
from tests.gpu_util import dev, ptr, stream, ulp_diff_f16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nv,n", [(1, 1, 2), (1, 2, 4), (2, 6, 5), (3, 3, 16), (1, 2, 17), (5, 5, 19), (1, 3, 67), (1, 1, 131)])
@pytest.mark.parametrize("strong", [False, True])
def test_deltanet_chunk_against_float64(lib, nk, nv, n, strong):
    # strong: decays down to e^-60 a token, which underflow over a block
    rng = np.random.default_rng(nk + 10 * nv + 100 * n)
    f16 = np.float16
    C = (2 * nk + nv) * 128
    ld = C + nv * 128 + 2 * nv
    ld += (-ld) % 4
    x = rng.standard_normal((n, ld)).astype(f16)
    a0 = C + nv * 128 + nv
    if strong:
        x[:, a0:a0 + nv] = rng.uniform(-6, 6, (n, nv)).astype(f16)
    conv_w = (rng.standard_normal((C, 4)) * 0.5).astype(f16)
    conv_state = rng.standard_normal((C, 4)).astype(f16)
    A_log = np.log(rng.uniform(0.1, 16, nv)).astype(f16)
    dt_bias = np.ones(nv, dtype=f16)
    norm_w = (1 + 0.1 * rng.standard_normal(128)).astype(f16)
    state = (rng.standard_normal((nv, 128, 128)) * 0.1).astype(np.float32)

    # token by token in float64 between the fp16 rounding points (conv output, beta, o)
    cs, S = conv_state.copy(), state.astype(np.float64)
    want_o = np.empty((n, nv, 128))
    for t in range(n):
        scr, cs = fo.dn_conv(x[t, :C], conv_w, cs)
        scr = np.asarray(scr, dtype=np.float64)
        for h in range(nv):
            kh = h // (nv // nk)
            q, k = scr[kh * 128:][:128], scr[(nk + kh) * 128:][:128]
            v = scr[2 * nk * 128 + h * 128:][:128]
            q = q / np.sqrt((q * q).sum() + 1e-6) / np.sqrt(128)
            k = k / np.sqrt((k * k).sum() + 1e-6)
            beta = np.float64(f16(1 / (1 + np.exp(-np.float64(x[t, C + nv * 128 + h])))))
            eg = np.exp(-np.exp(np.float64(A_log[h])) * np.log1p(np.exp(np.float64(x[t, a0 + h]) + 1.0)))
            Sh = S[h] * eg
            S[h] = Sh + np.outer((v - Sh @ k) * beta, k)
            want_o[t, h] = S[h] @ q
    o16 = want_o.astype(f16).astype(np.float64)
    xn = (o16 / np.sqrt((o16 ** 2).mean(-1, keepdims=True) + 1e-6)).astype(f16)
    z = x[:, C:C + nv * 128].astype(np.float64).reshape(n, nv, 128)
    want = ((xn * norm_w).astype(f16).astype(np.float64) * (z / (1 + np.exp(-z)))).astype(f16).reshape(n, -1)

    d_cs, d_S = dev(conv_state), dev(state)
    d_x, d_w, d_A, d_dt, d_nw = dev(x), dev(conv_w), dev(A_log), dev(dt_bias), dev(norm_w)
    nbytes = lib.nvfp4_dn_prefill_work_bytes(n, nk, nv)
    work = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")       # NaN everywhere
    out = torch.zeros((n, nv * 128), dtype=torch.float16, device="cuda")
    rc = lib.launch_dn_prefill(ptr(d_x), ld, ptr(d_w), ptr(d_cs), ptr(d_A), ptr(d_dt), ptr(d_nw),
                               ptr(d_S), ptr(work), nbytes, ptr(out), n, nk, nv, 1e-6, stream())
    torch.cuda.synchronize()
    assert rc == 0
    assert np.array_equal(d_cs.cpu().numpy().view(np.uint16), cs.view(np.uint16))
    # a conv output on the edge of an fp16 step moves a token's k, q or v by 2^-11 of itself
    assert np.abs(d_S.cpu().numpy() - S).max() <= 2e-3 * np.abs(S).max()
    steps = ulp_diff_f16(out.cpu().numpy(), want)
    assert (steps <= 1).mean() > 0.97, (steps.max(), (steps <= 1).mean())


def test_deltanet_chunk_keeps_a_bad_token_from_earlier_ones(lib):
    # token 6 (third of its block) has an infinite v: tokens 0..5 are what they are without it
    rng = np.random.default_rng(0)
    nk, nv, n = 1, 1, 9
    C, ld = 384, 384 + 128 + 4
    x = rng.standard_normal((n, ld)).astype(np.float16)
    outs = []
    for bad in (False, True):
        xb = x.copy()
        if bad:
            xb[6, 256:384] = np.inf
        d = [dev(a) for a in (xb, np.full((C, 4), 0.5, np.float16), np.zeros((C, 4), np.float16),
                              np.zeros(1, np.float16), np.zeros(1, np.float16), np.ones(128, np.float16),
                              np.zeros((1, 128, 128), np.float32))]
        nbytes = lib.nvfp4_dn_prefill_work_bytes(n, nk, nv)
        work = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
        out = torch.zeros((n, 128), dtype=torch.float16, device="cuda")
        assert lib.launch_dn_prefill(ptr(d[0]), ld, ptr(d[1]), ptr(d[2]), ptr(d[3]), ptr(d[4]), ptr(d[5]),
                                     ptr(d[6]), ptr(work), nbytes, ptr(out), n, nk, nv, 1e-6, stream()) == 0
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0][:6], outs[1][:6]) and np.isfinite(outs[1][:6]).all()
    assert not np.isfinite(outs[1][6:]).any()


@pytest.mark.parametrize("inter,N,shift", [(8, 1, 0), (24, 13, 0), (8, 8, 0), (64, 264, 0), (16, 16, 2), (16, 18, 0), (16, 18, 1),
                                           (2048, 7, 0), (2048, 10, 0), (2048, 512, 0), (2048, 512, 1), (512, 2048, 0),
                                           (1192, 515, 0)])    # many short rows, long rows, in each width
def test_silu_mul_rows_with_ragged_and_unaligned_rows(lib, inter, N, shift):
    rng = np.random.default_rng(inter + N)
    gu = (rng.standard_normal((2 * inter, N)) * 3).astype(np.float16)
    d_gu = torch.zeros(2 * inter * N + shift, dtype=torch.float16, device="cuda")[shift:]
    d_gu.copy_(torch.from_numpy(gu.reshape(-1)))
    act = torch.full((inter * N + 8,), 7.0, dtype=torch.float16, device="cuda")
    assert lib.launch_silu_mul_rows(ptr(d_gu), ptr(act), inter, N, stream()) == 0
    torch.cuda.synchronize()
    g = gu.reshape(inter // 8, 2, 8, N)
    want = fo.silu_mul(g[:, 0].reshape(-1), g[:, 1].reshape(-1))
    got = act.cpu().numpy()
    assert ulp_diff_f16(got[:inter * N], want.reshape(-1)).max() <= 1 and (got[inter * N:] == 7).all()


@pytest.mark.parametrize("n,shift", [((1 << 19) - 1, 0), (1 << 19, 0), ((1 << 19) + 5, 0), (1 << 20, 1), (2048 * 300 + 2047, 0)])
def test_silu_mul_of_long_vectors(lib, n, shift):
    rng = np.random.default_rng(n)
    g = (rng.standard_normal(n) * 3).astype(np.float16)
    u = rng.standard_normal(n).astype(np.float16)
    d_g = torch.zeros(n + shift, dtype=torch.float16, device="cuda")[shift:]
    d_g.copy_(torch.from_numpy(g))
    d_u = dev(u)
    out = torch.full((n + 8,), 7.0, dtype=torch.float16, device="cuda")
    assert lib.launch_silu_mul(ptr(d_g), ptr(d_u), ptr(out), n, stream()) == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert ulp_diff_f16(got[:n], fo.silu_mul(g, u)).max() <= 1 and (got[n:] == 7).all()


@pytest.mark.parametrize("hq,hkv,n", [(1, 1, 1), (5, 1, 3), (24, 4, 9), (9, 3, 2),
                                      (24, 4, 10), (1, 1, 100), (5, 1, 60), (9, 3, 30)])
def test_attn_prep_of_a_chunk_equals_token_by_token(lib, hq, hkv, n):
    # a CTA a head; then, with more tokens, eight heads a CTA: fewer, exactly and more than fill one
    rng = np.random.default_rng(hq + n)
    max_len, p0, ld = 140, 31, hq * 512 + hkv * 512 + 24
    qkv = dev(rng.standard_normal((n, ld)).astype(np.float16))
    w = [dev((1 + 0.1 * rng.standard_normal(256)).astype(np.float32)) for _ in range(2)]
    tab = [dev(rng.uniform(-1, 1, (max_len, 256)).astype(np.float16)) for _ in range(2)]
    new = lambda *s: torch.full(s, 7.0, dtype=torch.float16, device="cuda")
    a = [new(n, hq * 256), new(n, hq * 256), new(hkv, max_len, 256), new(hkv, max_len, 256)]
    b = [t.clone() for t in a]
    args = [ptr(t) for t in w + tab]
    assert lib.launch_attn_prep_tokens(ptr(qkv), ld, *args, p0, n, *[ptr(t) for t in a], hq, hkv, max_len, 1e-6,
                                       stream()) == 0
    for t in range(n):
        pos = torch.tensor([p0 + t], dtype=torch.int64, device="cuda")
        row = qkv[t].contiguous()
        assert lib.launch_attn_prep(ptr(row), *args, ptr(pos), ptr(b[0][t]), ptr(b[1][t]), ptr(b[2]), ptr(b[3]), hq,
                                    hkv, max_len, 1e-6, stream()) == 0
        torch.cuda.synchronize()
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 3, 9, 130])
def test_deltanet_chunk_with_inputs_at_any_element(lib, n, shift):
    # x a view that starts at an odd element of a wider row (every access to it is legal at 2 bytes):
    # the same values, the same bits
    rng = np.random.default_rng(n + shift)
    nk, nv = 2, 4
    C = (2 * nk + nv) * 128
    width = C + nv * 128 + 2 * nv
    ld = width + 8
    x = rng.standard_normal((n, width)).astype(np.float16)
    results = []
    for at in (0, shift):
        room = torch.zeros(n * ld + 8, dtype=torch.float16, device="cuda")
        rows = room[at:at + n * ld].view(n, ld)
        rows[:, :width] = dev(x)
        args = [dev(np.random.default_rng(1).standard_normal(s).astype(np.float16)) for s in ((C, 4), (C, 4), nv, nv, 128)]
        state = dev(np.random.default_rng(2).standard_normal((nv, 128, 128)).astype(np.float32))
        nbytes = lib.nvfp4_dn_prefill_work_bytes(n, nk, nv)
        work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        out = torch.zeros((n, nv * 128), dtype=torch.float16, device="cuda")
        assert lib.launch_dn_prefill(ptr(rows), ld, *[ptr(a) for a in args], ptr(state), ptr(work), nbytes, ptr(out), n,
                                     nk, nv, 1e-6, stream()) == 0
        torch.cuda.synchronize()
        results.append((out, state, args[1]))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 6, 7, 17])
def test_deltanet_state_after_an_infinite_last_value(lib, n):
    # The last token of a chunk that ends inside a block of four: S = S e^g + k delta with delta infinite
    # leaves infinities of k's sign, whatever the block's empty places hold.
    rng = np.random.default_rng(n)
    C, ld = 384, 384 + 128 + 4
    x = rng.standard_normal((n, ld)).astype(np.float16)
    x[n - 1, 256:384] = np.inf
    d = [dev(a) for a in (x, np.full((C, 4), 0.5, np.float16), np.zeros((C, 4), np.float16), np.zeros(1, np.float16),
                          np.zeros(1, np.float16), np.ones(128, np.float16), np.zeros((1, 128, 128), np.float32))]
    nbytes = lib.nvfp4_dn_prefill_work_bytes(n, 1, 1)
    work = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")
    out = torch.zeros((n, 128), dtype=torch.float16, device="cuda")
    assert lib.launch_dn_prefill(ptr(d[0]), ld, ptr(d[1]), ptr(d[2]), ptr(d[3]), ptr(d[4]), ptr(d[5]), ptr(d[6]), ptr(work),
                                 nbytes, ptr(out), n, 1, 1, 1e-6, stream()) == 0
    torch.cuda.synchronize()
    acc = (x[max(0, n - 4):, 128:256].astype(np.float64) * 0.5).sum(0)          # k before its (positive) silu and norm
    state = d[6].cpu().numpy()[0]
    assert np.isinf(state).all() and (np.sign(state) == np.sign(acc)).all()
