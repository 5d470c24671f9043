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
                                     (8, 40, 127), (8, 40, 128), (56, 56, 64), (28, 56, 65), (10, 80, 129),
                                     # (those of them that four tokens at a time take, a little longer)
                                     (3, 12, 321), (20, 40, 112), (28, 56, 97)])
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
    # every head, and every head's output of every token (three fp16 steps of each value are 3 * 2^-11 of the row, halved
    # and doubled within a binade)
    norm = lambda a: a.flatten(1).norm(dim=1)
    assert (norm(S.double() - want_S) <= 3 * norm(plain_S.double() - want_S) + 2 ** -20 * norm(want_S)).all()
    rows = lambda a: a.double().view(n * nv, 128).norm(dim=1)
    assert (rows(out.double() - want.double()) <= 2 ** -8 * rows(want)).all()
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


def real_inputs(nk, nv, n, seed):
    """What a decoder layer meets: small conv weights, decays of e^-0.001 to e^-20 and more, a state in use."""
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g)
    C = (2 * nk + nv) * 128
    ld = C + nv * 128 + 2 * nv
    t = dict(x=r(n, ld), conv_w=r(C, 4) * 0.02, conv_state=r(C, 4), A_log=torch.log(torch.rand(nv, generator=g) * 16 + 1e-3),
             dt_bias=torch.ones(nv), norm_w=torch.ones(128))
    t = {k: v.half().cuda() for k, v in t.items()}
    t["state"] = (r(nv, 128, 128) * 0.1).cuda()
    return t, ld


def float64_state(t, ld, conv_out, nk, nv, n):
    """The state after the chunk in 64 bits, from the fp16 conv outputs and the fp16 beta."""
    C = (2 * nk + nv) * 128
    x, co = t["x"].double(), conv_out.double()
    unit = lambda v: (v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(nv // nk, 1)
    k = unit(co[:, nk * 128:2 * nk * 128].view(n, nk, 128))
    v = co[:, 2 * nk * 128:].view(n, nv, 128)
    beta = torch.sigmoid(x[:, C + nv * 128:C + nv * 129]).half().double()
    g = -torch.exp(t["A_log"].double()) * torch.nn.functional.softplus(x[:, C + nv * 129:] + t["dt_bias"].double())
    S = t["state"].double()
    for i in range(n):
        S = S * torch.exp(g[i])[:, None, None]
        delta = beta[i][:, None] * (v[i] - torch.einsum("hrd,hd->hr", S, k[i]))
        S = S + delta[:, :, None] * k[i][:, None, :]
    return S


@pytest.mark.parametrize("kind,n", [("usual", 100), ("usual", 512), ("slow", 200), ("alike", 200)])
def test_error_is_that_of_the_token_by_token_form(lib, kind, n):
    # The same chunk at once (blocks of 64) and in pieces that the kernel of four tokens at a time takes (64 tokens of 48 heads),
    # both against 64 bits.  Everything that both share is exact: q, k and v are chosen, conv weights (0, 0, 0, 1) and inputs
    # of 24 and more, or 0, pass the conv and silu unchanged; beta is 1/2 or 1.
    nk, nv = 16, 48
    t, ld = real_inputs(nk, nv, n, 7 + n)
    C = (2 * nk + nv) * 128
    g = torch.Generator().manual_seed(n)
    t["conv_w"].zero_()
    t["conv_w"][:, 3] = 1
    x = torch.randint(24, 200, (n, C), generator=g).float()
    if kind != "alike":                      # a key or query has a third of its values, so that they are far from parallel
        x[:, :2 * nk * 128] *= (torch.rand(n, 2 * nk * 128, generator=g) < 0.33)
    t["x"][:, :C] = x.half().cuda()
    b = torch.where(torch.rand(n, nv, generator=g) < 0.5, 0.0, 30.0)
    t["x"][:, C + nv * 128:C + nv * 129] = b.half().cuda()
    if kind != "usual":
        t["A_log"].fill_(-7.0)
    want = float64_state(t, ld, t["x"][:, :C], nk, nv, n)
    once, _ = run(lib, t, ld, nk, nv, n)
    pieces = dict(t)
    for i in range(0, n, 64):
        m = min(64, n - i)
        state, conv_state = pieces["state"].clone(), pieces["conv_state"].clone()
        nbytes = lib.nvfp4_dn_prefill_work_bytes(m, nk, nv)
        work, out = torch.empty(nbytes, dtype=torch.uint8, device="cuda"), torch.empty(m * nv * 128, dtype=torch.float16, device="cuda")
        assert lib.launch_dn_prefill(ptr(t["x"][i:]), ld, ptr(t["conv_w"]), ptr(conv_state), ptr(t["A_log"]), ptr(t["dt_bias"]),
                                     ptr(t["norm_w"]), ptr(state), ptr(work), nbytes, ptr(out), m, nk, nv, 1e-6, stream()) == 0
        pieces.update(state=state, conv_state=conv_state)
    torch.cuda.synchronize()
    err = lambda a: ((a.double() - want).norm() / want.norm()).item()
    # the errors are averages over 786432 values of a few dozen roundings each: 10 % is far outside their spread
    assert err(once) <= 1.1 * err(pieces["state"]), (err(once), err(pieces["state"]))


def test_small_tokens_beside_large_ones(lib):
    # A token of 60000s, one that clears the state, then tokens of 2^-8 and less with hardly any decay: operands that share a
    # row's scale with the large token, and everything that is left at the end is small.
    nk, nv, n = 16, 48, 128
    t, ld = real_inputs(nk, nv, n, 11)
    C = (2 * nk + nv) * 128
    g = torch.Generator().manual_seed(12)
    t["conv_w"].zero_()
    t["conv_w"][:, 3] = 1
    x = torch.randint(24, 200, (n, C), generator=g).float()
    x[:, :2 * nk * 128] *= (torch.rand(n, 2 * nk * 128, generator=g) < 0.33)
    x[:, 2 * nk * 128:] = torch.randn(n, nv * 128, generator=g) * 2.0 ** -9
    x[::64, 2 * nk * 128:] = 60000
    t["x"][:, :C] = x.half().cuda()
    t["x"][:, C + nv * 128:C + nv * 129] = 30.0
    t["x"][:, C + nv * 129:] = 0.0
    t["x"][1::64, C + nv * 129:] = 60000.0
    t["A_log"].fill_(-7.0)
    S, _ = run(lib, t, ld, nk, nv, n)
    # silu of the small values as the kernel rounds it: fp32, then fp16 (a value that falls the other way is 2^-11 of itself off,
    # and there are few: 1e-5 of the state)
    co = t["x"][:, :C].clone()
    v = co[:, 2 * nk * 128:].float()
    co[:, 2 * nk * 128:] = (v / (1 + torch.exp(-v))).half()
    want = float64_state(t, ld, co, nk, nv, n)
    worst = ((S.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)).max().item()
    assert worst <= 1e-5, worst


def test_workspace_grows_with_the_chunk(lib):
    # a workspace sized for the longest chunk serves the shorter ones, whichever of the two forms takes them
    for nk, nv in ((16, 48), (16, 64), (14, 56), (10, 40), (8, 24), (5, 20), (4, 12), (1, 1)):
        sizes = [lib.nvfp4_dn_prefill_work_bytes(n, nk, nv) for n in range(1, 700)]
        assert all(a <= b for a, b in zip(sizes, sizes[1:])), (nk, nv)
