"""The performance cases of this framework: what its users run on one GPU, with real sizes.

Every case goes through a public entry point: ``DecodeEngine`` (``prefill``, ``capture``, ``step``),
the bridge's ``QLinear``, or the C ABI bound by ``nvfp4_v100_b200._lib``.  The shapes are those of
the 27B hybrid decoder that ``ModelConfig`` defaults to (hidden 5120, MLP 17408, 24 query / 4 KV
heads x 256, DeltaNet 16 / 48 heads x 128, vocabulary 248320), with seeded random weights.

``listed`` gives the cases, ``draw`` one more of the same ranges, ``prepare`` what a program holds
before the call (weights uploaded, graph captured, inputs in device memory), ``run`` one pass.
"""
import ctypes
import math

import numpy as np
import torch

from nvfp4_v100_b200 import _lib
from nvfp4_v100_b200.engine import DecodeEngine, ModelConfig

HIDDEN, INTER, VOCAB = 5120, 17408, 248320
# (rows, columns) of the linear layers as the container stores them, one entry per matrix
ATTENTION = [(12288, HIDDEN), (1024, HIDDEN), (1024, HIDDEN), (HIDDEN, 6144)]
DELTANET = [(10240, HIDDEN), (6144, HIDDEN), (48, HIDDEN), (48, HIDDEN), (HIDDEN, 6144)]
MLP = [(INTER, HIDDEN), (INTER, HIDDEN), (HIDDEN, INTER)]
PROJECTIONS = [(1024, HIDDEN), (6144, HIDDEN), (HIDDEN, 6144), (10240, HIDDEN), (12288, HIDDEN),
               (INTER, HIDDEN), (HIDDEN, INTER)]


def listed():
    return [
        # generating text with the whole 27B decoder: one token per replay of the step graph, after
        # the usual 512-token prompt and deep in a long conversation
        {"name": "decode_ctx512", "kind": "decode", "layers": 64, "context": 512},
        {"name": "decode_ctx3500", "kind": "decode", "layers": 64, "context": 3500},
        # time to the first token: a chat turn of a few words, the usual prompt, and a document.
        # 16 of the 64 layers: all blocks of four layers are alike, and every cache and state is
        # returned for comparison
        {"name": "prompt_27", "kind": "prompt", "layers": 16, "tokens": 27, "chunk": 512},
        {"name": "prompt_511", "kind": "prompt", "layers": 16, "tokens": 511, "chunk": 512},
        {"name": "prompt_4000", "kind": "prompt", "layers": 16, "tokens": 4000, "chunk": 512},
        # a program that keeps its own model code and captures the 497 matrix-vector products of
        # one token in a graph: the headline bandwidth workload
        {"name": "gemv_497", "kind": "gemv_mix", "layers": 64},
        # the smallest call of the drop-in layer: one key projection of one token, launched eagerly
        {"name": "linear_1_token", "kind": "linear", "m": 1024, "k": HIDDEN, "tokens": 1},
        # the drop-in layers of one MLP block: two tokens (draft verification), a small ragged batch
        # of sequences decoded together, and a prompt chunk
        {"name": "mlp_2_tokens", "kind": "mlp", "tokens": 2},
        {"name": "mlp_21_tokens", "kind": "mlp", "tokens": 21},
        {"name": "mlp_2048_tokens", "kind": "mlp", "tokens": 2048},
        # FP4 activations quantised on the fly: prefill of 4 x 2048 tokens
        {"name": "w4a4_8192_tokens", "kind": "w4a4", "m": INTER, "k": HIDDEN, "tokens": 8192},
        # writing a container: quantising one MLP matrix on the device
        {"name": "quantise", "kind": "quantise", "m": INTER, "k": HIDDEN},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "gemv_mix", "linear", "mlp", "w4a4", "quantise"])
    if kind == "decode":
        return {"kind": kind, "layers": 4 * rng.randint(4, 16), "context": _log_uniform(rng, 16, 3500)}
    if kind == "prompt":
        return {"kind": kind, "layers": 4 * rng.randint(1, 4), "tokens": _log_uniform(rng, 8, 4000),
                "chunk": rng.choice([256, 512, 512, 1024])}
    if kind == "gemv_mix":
        return {"kind": kind, "layers": 4 * rng.randint(2, 16)}
    if kind == "linear":
        m, k = rng.choice(PROJECTIONS)
        return {"kind": kind, "m": m, "k": k, "tokens": rng.choice([1, 1, 2, _log_uniform(rng, 3, 2048)])}
    if kind == "mlp":
        return {"kind": kind, "tokens": _log_uniform(rng, 1, 2048)}
    if kind == "w4a4":
        m, k = rng.choice(PROJECTIONS[1:])
        return {"kind": kind, "m": m, "k": k, "tokens": _log_uniform(rng, 32, 8192)}
    return {"kind": kind, "m": rng.randint(64, INTER), "k": 16 * rng.randint(64, HIDDEN // 16)}


# ----------------------------------------------------------------------------------- helpers
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} rc={rc}")


def _quantised(lib, g, m, k):
    """An [m, k] matrix of N(0, 0.02^2) weights as NVFP4 bytes."""
    w = (torch.randn((m, k), device="cuda", generator=g) * 0.02).half()
    p = torch.empty(m * k // 2, dtype=torch.uint8, device="cuda")
    s = torch.empty(m * k // 16, dtype=torch.uint8, device="cuda")
    _ok(lib.launch_nvfp4_encode(_ptr(w), _ptr(p), _ptr(s), m, k, _stream()), "encode")
    return p, s


def _activations(g, tokens, k):
    return torch.randn((tokens, k), device="cuda", generator=g).half()


def _engine(layers, max_len, seed):
    eng = DecodeEngine(ModelConfig(n_layers=layers, vocab=VOCAB, max_len=max_len), device="cuda")
    eng.load_random(seed=seed)
    eng.reset(0)
    return eng


def _states(eng):
    """Every cache and recurrent state of the engine (its own buffers)."""
    names = {True: ("keys", "values"), False: ("conv_state", "state")}
    return [L.extra[n] for L in eng.layers for n in names[L.attn]]


# ----------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    lib = _lib.load()
    g = _generator(seed)
    rng = np.random.default_rng(seed)
    s = {"kind": case["kind"], "lib": lib}
    kind = case["kind"]
    if kind == "decode":
        n = case["context"]
        eng = _engine(case["layers"], (n + 128) // 64 * 64, seed)
        for L in eng.layers:                # what the prompt left: caches up to n, states
            e = L.extra
            if L.attn:
                e["keys"][:, :n].normal_(generator=g)
                e["values"][:, :n].normal_(generator=g)
            else:
                e["conv_state"].normal_(generator=g)
                e["state"].normal_(std=0.1, generator=g)
        eng.pos.fill_(n)
        eng.len.fill_(n + 1)
        eng.capture()
        s.update(eng=eng, n=n, token=int(rng.integers(0, VOCAB)))
    elif kind == "prompt":
        n = case["tokens"]
        eng = _engine(case["layers"], (n + 128) // 64 * 64, seed)
        eng.capture()
        s.update(eng=eng, tokens=[int(t) for t in rng.integers(0, VOCAB, n)], chunk=case["chunk"])
    elif kind == "gemv_mix":
        shapes = []
        for i in range(case["layers"]):
            shapes += (ATTENTION if i % 4 == 3 else DELTANET) + MLP
        shapes.append((VOCAB, HIDDEN))
        pad = lambda n: (n + 127) // 128 * 128
        x = torch.empty(sum(pad(k) for _, k in shapes), dtype=torch.float16, device="cuda")
        x.normal_(generator=g)
        y = torch.zeros(sum(pad(m) for m, _ in shapes), dtype=torch.float16, device="cuda")
        calls, at_x, at_y = [], 0, 0
        for m, k in shapes:
            p = torch.randint(0, 256, (m * k // 2,), dtype=torch.uint8, device="cuda", generator=g)
            c = torch.randint(118, 123, (m * k // 16,), dtype=torch.uint8, device="cuda", generator=g)
            calls.append((p, c, x[at_x:], y[at_y:], m, k))
            at_x, at_y = at_x + pad(k), at_y + pad(m)

        def step():
            for p, c, a, o, m, k in calls:
                _ok(lib.launch_nvfp4_gemv_v8(_ptr(p), _ptr(c), _ptr(a), _ptr(o), m, k, _stream()), "gemv")

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        s.update(graph=graph, calls=calls, x=x, y=y)
    elif kind in ("linear", "mlp"):
        from nvfp4_v100_b200.pipeline._qwen38_infer import QLinear

        shapes = MLP if kind == "mlp" else [(case["m"], case["k"])]
        mats = [_quantised(lib, g, m, k) for m, k in shapes]
        s["mats"] = mats
        s["layers"] = [QLinear(p.data_ptr(), c.data_ptr(), m, k) for (p, c), (m, k) in zip(mats, shapes)]
        s["x"] = _activations(g, case["tokens"], shapes[0][1])
    elif kind == "w4a4":
        m, k, n = case["m"], case["k"], case["tokens"]
        n8 = (n + 7) // 8 * 8
        s["w"] = _quantised(lib, g, m, k)
        s["x"] = _activations(g, n, k)
        s["out"] = torch.zeros((m, n8), dtype=torch.float16, device="cuda")
        s["work"] = torch.empty(k * n8, dtype=torch.float16, device="cuda")
        s["dims"] = (m, n, k)
    elif kind == "quantise":
        m, k = case["m"], case["k"]
        s["w"] = (torch.randn((m, k), device="cuda", generator=g) * 0.02).half()
        s["p"] = torch.empty((m, k // 2), dtype=torch.uint8, device="cuda")
        s["s"] = torch.empty((m, k // 16), dtype=torch.uint8, device="cuda")
        s["dims"] = (m, k)
    else:
        raise ValueError(kind)
    return s


# --------------------------------------------------------------------------------------- run
def run(state):
    kind, lib = state["kind"], state["lib"]
    if kind == "decode":
        # one token at the end of the context; the position is set again so that any number of
        # passes decodes the same place
        eng = state["eng"]
        eng.pos.fill_(state["n"])
        eng.len.fill_(state["n"] + 1)
        eng.tok.fill_(state["token"])
        eng.step()
        return [eng.logits] + [L.extra["state"] for L in eng.layers if not L.attn]
    if kind == "prompt":
        eng, tokens = state["eng"], state["tokens"]
        eng.reset(tokens[0])
        eng.prefill(tokens[:-1], chunk=state["chunk"])
        eng.tok.fill_(tokens[-1])
        eng.step()
        return [eng.logits] + _states(eng)
    if kind == "gemv_mix":
        state["graph"].replay()
        return state["y"]
    if kind == "linear":
        return state["layers"][0](state["x"])
    if kind == "mlp":
        gate, up, down = state["layers"]
        a, b = gate(state["x"]), up(state["x"])
        h = torch.empty_like(a)
        _ok(lib.launch_silu_mul(_ptr(a), _ptr(b), _ptr(h), a.numel(), _stream()), "silu_mul")
        return down(h)
    if kind == "w4a4":
        m, n, k = state["dims"]
        p, c = state["w"]
        _ok(lib.launch_nvfp4_gemm_w4a4(_ptr(p), _ptr(c), _ptr(state["x"]), _ptr(state["out"]),
                                       _ptr(state["work"]), m, n, k, _stream()), "gemm_w4a4")
        return state["out"]
    m, k = state["dims"]
    _ok(lib.launch_nvfp4_encode(_ptr(state["w"]), _ptr(state["p"]), _ptr(state["s"]), m, k, _stream()),
        "encode")
    return [state["p"], state["s"]]


# ------------------------------------------------------------------------------ work, tolerance
def _matrix(m, k):
    return m * k * 9 // 16


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        layers = case["layers"]
        n_att, n_dn = layers // 4, layers - layers // 4
        params = (n_att * sum(m * k for m, k in ATTENTION) + n_dn * sum(m * k for m, k in DELTANET)
                  + layers * sum(m * k for m, k in MLP))
        weights = params * 9 // 16
        head = _matrix(VOCAB, HIDDEN)
        kv_row = 2 * 4 * 256 * 2                      # bytes of one position's keys and values
        dn_state = 48 * 128 * 128 * 4 + 10240 * 4 * 2
        if kind == "decode":
            n = case["context"]
            return {"bytes": weights + head + n_att * (n + 2) * kv_row + n_dn * 2 * dn_state
                             + 2 * HIDDEN + 2 * VOCAB,
                    "flops": 2 * params + 2 * VOCAB * HIDDEN + n_att * 24 * 256 * 4 * (n + 1)
                             + n_dn * 48 * 128 * 128 * 6}
        n = case["tokens"]
        # the prompt's products, then the step of its last token (which reads the weights again);
        # caches and states written once per prompt, cleared before it
        return {"bytes": 2 * weights + head + n_att * 3 * n * kv_row + n_dn * 4 * dn_state + 2 * n * HIDDEN,
                "flops": 2 * params * n + 2 * VOCAB * HIDDEN + n_att * 24 * 256 * 2 * n * (n + 1)
                         + n_dn * 48 * 128 * 128 * 6 * n}
    if kind == "gemv_mix":
        shapes = [(VOCAB, HIDDEN)]
        for i in range(case["layers"]):
            shapes += (ATTENTION if i % 4 == 3 else DELTANET) + MLP
        return {"bytes": sum(_matrix(m, k) + 2 * m + 2 * k for m, k in shapes),
                "flops": sum(2 * m * k for m, k in shapes)}
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["tokens"]
        return {"bytes": _matrix(m, k) + 2 * n * (m + k), "flops": 2 * m * k * n}
    if kind == "mlp":
        n = case["tokens"]
        return {"bytes": sum(_matrix(m, k) for m, k in MLP) + 4 * n * HIDDEN,
                "flops": sum(2 * m * k * n for m, k in MLP)}
    if kind == "w4a4":
        m, k, n = case["m"], case["k"], case["tokens"]
        return {"bytes": _matrix(m, k) + 2 * n * (m + k), "flops": 2 * m * k * n}
    m, k = case["m"], case["k"]
    return {"bytes": m * k * 2 + _matrix(m, k), "flops": 0}


def tolerance(case):
    """Measured by taking the sums in another order (the other GEMV kernel, other prompt chunks):
    fp16 roundings between layers then fall differently and random weights carry that on, up to
    1.1e-2 after 64 layers and 4e-3 after 16 (largest single values 5e-2); one product alone moves by
    7e-6, an fp16 step (1e-3) at its largest."""
    kind = case["kind"]
    if kind == "quantise":
        return "exact"
    if kind == "decode":
        return {"rel": 0.03, "max": 0.25}
    if kind == "prompt":
        return {"rel": 0.016, "max": 0.25}
    return {"rel": 3e-4, "max": 5e-3}
