"""Gated DeltaNet over a chunk in blocks of 64 tokens (tensor cores): block edges, every number of row groups per CTA, strong
and absent decay, and values that are not finite."""
import numpy as np
import pytest
import torch

from tests.gpu_util import ptr, stream, ulp_diff_f16

pytestmark = pytest.mark.gpu


def inputs(nk, nv, n, decay, seed=0):
    """Conv weights (0, 0, 0, 1) and inputs of 24 and more make silu and the fp16 rounding exact: q, k and v are x."""
    g = torch.Generator().manual_seed(seed + 1000 * nv + n)
    C = (2 * nk + nv) * 128
    ld = C + nv * 128 + 2 * nv
    ld += -ld % 4
    x = torch.randn(n, ld, generator=g)
    x[:, :C] = torch.randint(24, 80, (n, C), generator=g).float()
    x[:, 2 * nk * 128:C] += torch.randint(0, 900, (n, nv * 128), generator=g).float()
    a = x[:, C + nv * 129:C + nv * 130]
    if decay == "strong":
        a.uniform_(-6, 6, generator=g)
    A_log = torch.full((nv,), -9.0) if decay == "none" else torch.log(torch.rand(nv, generator=g) * 8 + 0.05)
    conv_w = torch.zeros(C, 4)
    conv_w[:, 3] = 1
    t = dict(x=x, conv_w=conv_w, conv_state=torch.zeros(C, 4), A_log=A_log, dt_bias=torch.ones(nv), norm_w=torch.ones(128))
    t = {k: v.half().cuda() for k, v in t.items()}
    t["state"] = (torch.randn(nv, 128, 128, generator=g) * 20).cuda()
    return t, ld


def run(lib, t, ld, nk, nv, n):
    state, conv_state = t["state"].clone(), t["conv_state"].clone()
    nbytes = lib.nvfp4_dn_prefill_work_bytes(n, nk, nv)
    work = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")            # NaN everywhere
    out = torch.zeros((n, nv * 128), dtype=torch.float16, device="cuda")
    assert lib.launch_dn_prefill(ptr(t["x"]), ld, ptr(t["conv_w"]), ptr(conv_state), ptr(t["A_log"]), ptr(t["dt_bias"]),
                                 ptr(t["norm_w"]), ptr(state), ptr(work), nbytes, ptr(out), n, nk, nv, 1e-6, stream()) == 0
    torch.cuda.synchronize()
    return state, out


def reference(t, nk, nv, n, dtype):
    x = t["x"].to(dtype)
    C = (2 * nk + nv) * 128
    unit = lambda v: v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)
    rep = lambda v: v.repeat_interleave(nv // nk, 1)
    q = rep(unit(x[:, :nk * 128].view(n, nk, 128)) / 128 ** 0.5)
    k = rep(unit(x[:, nk * 128:2 * nk * 128].view(n, nk, 128)))
    v = x[:, 2 * nk * 128:C].view(n, nv, 128)
    z = x[:, C:C + nv * 128].view(n, nv, 128)
    beta = torch.sigmoid(x[:, C + nv * 128:C + nv * 129]).half().to(dtype)
    g = -torch.exp(t["A_log"].to(dtype)) * torch.nn.functional.softplus(x[:, C + nv * 129:C + nv * 130] + 1.0)
    S, o = t["state"].to(dtype), torch.empty(n, nv, 128, dtype=dtype, device="cuda")
    for i in range(n):
        S = S * torch.exp(g[i])[:, None, None]
        delta = beta[i][:, None] * (v[i] - torch.einsum("hrd,hd->hr", S, k[i]))
        S = S + delta[:, :, None] * k[i][:, None, :]
        o[i] = torch.einsum("hrd,hd->hr", S, q[i])
    xn = o.half().to(dtype)
    xn = (xn / torch.sqrt((xn * xn).mean(-1, keepdim=True) + 1e-6)).half().to(dtype)
    return S, (xn * z / (1 + torch.exp(-z))).half().view(n, -1)


# one, two, three and four row groups per CTA (the last head part of three is short), and more CTAs than SMs; chunks
# that end with a block, one token into it, one before its end
@pytest.mark.parametrize("nk,nv,n", [(1, 1, 256), (2, 6, 257), (3, 12, 319), (5, 20, 160), (10, 20, 193), (20, 40, 100),
                                     (8, 40, 127), (8, 40, 128), (56, 56, 64), (28, 56, 65), (10, 80, 129)])
@pytest.mark.parametrize("decay", ["usual", "strong", "none"])
def test_blocks_of_64_against_float64(lib, nk, nv, n, decay):
    t, ld = inputs(nk, nv, n, decay)
    if decay == "strong":                                    # one token that clears the state: e^-inf
        t["x"][n // 2, (2 * nk + nv) * 128 + nv * 129:(2 * nk + nv) * 128 + nv * 130] = float("inf")
    S, out = run(lib, t, ld, nk, nv, n)
    want_S, want = reference(t, nk, nv, n, torch.float64)
    plain_S, _ = reference(t, nk, nv, n, torch.float32)
    # What fp32 gives token by token, and 16 roundings more.  (The keys are all positive here, so nearly parallel, and
    # without decay a state forgets little: its fp32 error is far above its roundings, and differs by the order of sums.)
    err = lambda a: (a.double() - want_S).norm() / want_S.norm()
    assert err(S) <= 3 * err(plain_S) + 2 ** -20, (err(S), err(plain_S))
    steps = ulp_diff_f16(out.cpu().numpy(), want.cpu().numpy())
    assert (steps <= 1).mean() > 0.98 and (steps <= 3).mean() > 0.999, ((steps <= 1).mean(), steps.max())


def test_a_token_that_is_not_finite_stays_out_of_earlier_ones(lib):
    nk, nv, n, bad = 8, 40, 140, 70
    t, ld = inputs(nk, nv, n, "usual")
    S0, clean = run(lib, t, ld, nk, nv, n)
    C = (2 * nk + nv) * 128
    t["x"][bad, 2 * nk * 128 + 5] = float("inf")             # v: row 5 of head 0
    S1, out = run(lib, t, ld, nk, nv, n)
    assert torch.equal(out[:64], clean[:64])                 # blocks before
    # the block's tokens before it (head 0's outputs there are taken token by token: at most a rounding of o and of the
    # normalised o away), and everything of the other heads
    assert torch.isfinite(out[:bad]).all()
    assert ulp_diff_f16(out[64:bad, :128].cpu().numpy(), clean[64:bad, :128].cpu().numpy()).max() <= 3
    assert torch.equal(out[:, 128:], clean[:, 128:])
    assert not torch.isfinite(out[bad, 5]) and not torch.isfinite(out[bad + 1:, :128]).any()   # (the gated norm spreads NaN)
    assert not torch.isfinite(S1[0, 5]).any() and torch.isfinite(S1[1:]).all() and torch.isfinite(S1[0, 16:]).all()
    assert torch.equal(S0[1:], S1[1:])
    # a query that is not finite is its own token's alone (and, through the conv's zero weights, that of the three after it)
    t["x"][bad, 2 * nk * 128 + 5] = 30.0
    t["x"][bad, 3] = float("nan")
    S2, out = run(lib, t, ld, nk, nv, n)
    assert torch.isfinite(S2).all() and not torch.isfinite(out[bad, :128]).any()
    assert torch.isfinite(out[:bad]).all() and torch.isfinite(out[bad + 4:]).all()
    # a key: nothing of its heads is finite from there on, everything before it is
    t["x"][bad, 3] = 30.0
    t["x"][bad, nk * 128 + 3] = float("nan")
    S3, out = run(lib, t, ld, nk, nv, n)
    assert torch.isfinite(out[:bad]).all() and not torch.isfinite(out[bad:, :128 * (nv // nk)]).any()
    assert torch.isfinite(out[:, 128 * (nv // nk):]).all()
