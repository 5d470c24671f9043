"""Bridge between the third-party Qwen3.5 model code and this repository's sm_100a library.

The module answers to the public names of the reference's ``pipeline/_qwen38_infer.py`` (every
acceptance script of the reference imports them, experiments/_qwen38_p9_acc.py:21-27), so a script
written against the reference runs against this package unchanged:

  bindings      ``load_gemv`` ``load_v5`` ``GEMV`` ``V5`` ``GEMV_T1`` ``set_gemv_t1``
  weights       ``open_container`` ``upload_nvfp4`` ``PackedEmb`` ``QEmbedding`` ``QLinear``
                ``st_name`` ``patch_linears`` ``fill_rest`` ``rebuild_rope`` ``build_model``
  decode state  ``ensure_kv_stage`` ``snap_decode_state`` ``restore_decode_state``
                ``refresh_deltanet_state`` ``prefill``
  operators     ``patch_fused_deltanet`` ``patch_attn_decode`` ``patch_rmsnorm`` ``patch_rope``
                ``patch_mlp_silu_mul``   (the last two: experiments/_qwen38_p9_fuse.py:48-116)
  step graph    ``GraphDecoder`` ``GraphDecoder2``

How it is built here (the reference's behaviour in brackets where it differs):
  * one shared library, bound once through ``nvfp4_v100_b200._lib`` with its signature table
    [six DLLs, ``argtypes`` set at every call site]; ``kernels/<name>.dll`` aliases exist and are
    checked, so ``ctypes.CDLL`` on the reference's file names keeps working;
  * weight bytes are copied to the device straight from the memory-mapped container [file reads
    into host byte strings first];
  * the embedding table lives in device memory and rows are gathered there — a 2.5 GB table is
    small next to 180 GB of HBM [host table, row decoded on the CPU and copied per token];
  * every operator substitution is a small callable object that remembers the module's own
    forward and falls back to it for any shape the fused kernel does not cover;
  * head counts come from the module, so tensor-parallel shards and small test models work; the
    27B head counts take the reference-named entry points, others the ``*_heads`` variants;
  * a failed launch raises ``RuntimeError`` with the return code.
"""
from __future__ import annotations

import ctypes
import json
import mmap
import os

import numpy as np
import torch
import torch.nn as nn

from .. import _lib

BASE = os.path.dirname(os.path.abspath(__file__))
KDIR = os.path.join(os.path.dirname(BASE), "kernels")
MODEL_DIR = os.environ.get("NVFP4_MODEL_DIR", "")
UPLOAD_BYTES = [0]          # running total, as the reference keeps it (a one-element list)

_vp = ctypes.c_void_p
_DLL_NAMES = ("nvfp4_gemv.dll", "nvfp4_cuda_v5.dll", "nvfp4_rmsnorm.dll", "nvfp4_attn_decode.dll",
              "nvfp4_rope_silu.dll", "nvfp4_dn_fused.dll")


# ------------------------------------------------------------------------------------ bindings
def _bound_library(alias: str):
    """The library, after checking that the reference's file name for it resolves."""
    if alias not in _DLL_NAMES:
        raise ValueError(alias)
    if not os.path.exists(os.path.join(KDIR, alias)):
        raise RuntimeError(f"{os.path.join(KDIR, alias)} is missing: "
                           "run `python -m nvfp4_v100_b200.build` (there is no CPU fallback)")
    return _lib.load()


def load_gemv():
    return _bound_library("nvfp4_gemv.dll")


def load_v5():
    return _bound_library("nvfp4_cuda_v5.dll")


GEMV = load_gemv()
V5 = load_v5()
H2D = GEMV.gpu_memcpy_h2d
_T1_ENTRIES = {"v1": "launch_nvfp4_gemv", "v8": "launch_nvfp4_gemv_v8"}
GEMV_T1 = getattr(GEMV, _T1_ENTRIES.get(os.environ.get("VF_GEMV", "v8"), _T1_ENTRIES["v8"]))


def set_gemv_t1(name):
    """Choose the entry point QLinear uses for one token: 'v1' or 'v8' (KeyError otherwise)."""
    global GEMV_T1
    GEMV_T1 = getattr(GEMV, _T1_ENTRIES[name])
    return GEMV_T1


# the current stream's handle without a Python Stream object (1.5 us of every call); None: not offered
_RAW_STREAM = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_handle() -> int:
    if _RAW_STREAM is None:
        return torch.cuda.current_stream().cuda_stream
    return _RAW_STREAM(torch.cuda.current_device())


def _cur_stream():
    return _vp(_stream_handle())


def _p(t: torch.Tensor):
    return _vp(t.data_ptr())


def _ok(rc: int, what: str):
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")


def _kind(layer) -> str:
    # the reference's transformers calls the attribute block_type, the installed one layer_type
    k = getattr(layer, "layer_type", None)
    return k if k is not None else getattr(layer, "block_type")


# ------------------------------------------------------------------------------------- weights
class _Container:
    """``nvfp4_packed.bin`` mapped read-only; a matrix is a byte range of the map."""

    def __init__(self, directory: str):
        self.directory = directory
        self._fh = open(os.path.join(directory, "nvfp4_packed.bin"), "rb")
        size = os.fstat(self._fh.fileno()).st_size
        self._map = mmap.mmap(self._fh.fileno(), 0, access=mmap.ACCESS_READ) if size else None
        self.view = np.frombuffer(self._map, dtype=np.uint8) if size else np.zeros(0, np.uint8)

    def close(self):
        self.view = None
        if self._map is not None:
            self._map.close()
        self._fh.close()


_OPEN = {"container": None}


def open_container(model_dir=None):
    where = model_dir or MODEL_DIR
    if not where:
        raise RuntimeError("no model directory: pass model_dir or set NVFP4_MODEL_DIR")
    cur = _OPEN["container"]
    if cur is None or cur.directory != where:
        if cur is not None:
            cur.close()
        _OPEN["container"] = _Container(where)
    return _OPEN["container"]


def upload_nvfp4(entry):
    """Index entry -> (device address of the packed bytes, device address of the scale bytes).

    Two allocations, because callers own and free the two addresses independently (the
    reference's pair fusion does: experiments/_qwen38_p7_pair.py:115-118); each is filled by one
    synchronous copy whose source is the memory-mapped container itself, so no intermediate host
    copy of the matrix is made (reference: pipeline/_qwen38_infer.py:91-101)."""
    box = _OPEN["container"]
    if box is None:
        raise RuntimeError("open_container() first")
    addresses = []
    for what in ("packed", "scales"):
        nbytes, at = int(entry[what + "_bytes"]), int(entry[what + "_off"])
        dst = GEMV.gpu_malloc(nbytes)
        if not dst:
            raise MemoryError(f"gpu_malloc({nbytes}) for the {what} bytes")
        _ok(H2D(dst, box.view[at:at + nbytes].ctypes.data, nbytes), "gpu_memcpy_h2d")
        UPLOAD_BYTES[0] += nbytes
        addresses.append(dst)
    return tuple(addresses)


def _byte_table() -> np.ndarray:
    """All 256 packed bytes -> the two fp32 code-point values they hold (low nibble first)."""
    mag = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=np.float32)
    b = np.arange(256)
    lo = np.where(b & 0x08, -mag[b & 7], mag[b & 7])
    hi = np.where(b & 0x80, -mag[(b >> 4) & 7], mag[(b >> 4) & 7])
    return np.stack([lo, hi], axis=1).astype(np.float32)


class PackedEmb:
    """NVFP4 embedding table kept packed (memory-mapped ``.npy`` pair); indexing dequantises the
    requested rows to fp16 on the host with the codec's arithmetic: value = code point x
    2^(scale byte - 127), computed in float64 and rounded once to fp16."""
    CP = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=np.float32)

    def __init__(self, path_p, path_s):
        self.packed = np.load(path_p, mmap_mode="r")
        self.scales = np.load(path_s, mmap_mode="r")
        self.shape = (self.packed.shape[0], 2 * self.packed.shape[1])
        self._pairs = _byte_table()

    def __getitem__(self, idx):
        one_row = np.isscalar(idx) or (torch.is_tensor(idx) and idx.ndim == 0)
        rows = np.atleast_1d(np.asarray(idx.cpu() if torch.is_tensor(idx) else idx)).ravel()
        vals = self._pairs[np.asarray(self.packed[rows])]              # (n, K/2, 2)
        vals = vals.reshape(len(rows), -1, 16).astype(np.float64)
        factor = np.ldexp(1.0, np.asarray(self.scales[rows]).astype(np.int32) - 127)
        out = (vals * factor[..., None]).astype(np.float16).reshape(len(rows), -1)
        return torch.from_numpy(out[0] if one_row else out)


class QEmbedding(nn.Module):
    """Token embedding.  ``weight_cpu`` is the host table the reference's callers index
    (``GraphDecoder.step(tok, model.model.embed_tokens.weight_cpu)``).  The table is also copied to
    the device once — as fp16, or as its packed and scale bytes when it is a ``PackedEmb`` — and
    lookups are gathered (and dequantised by ``launch_nvfp4_decode_rows``) there."""

    def __init__(self, weight_cpu):
        super().__init__()
        self.weight_cpu = weight_cpu
        self.num_embeddings, self.embedding_dim = weight_cpu.shape
        self._table = None

    def device_table(self):
        if self._table is None:
            w = self.weight_cpu
            if torch.is_tensor(w):
                self._table = w.to(device="cuda", dtype=torch.float16)
            else:                                     # PackedEmb: keep it packed on the device too
                self._table = (torch.from_numpy(np.ascontiguousarray(w.packed)).cuda(),
                               torch.from_numpy(np.ascontiguousarray(w.scales)).cuda())
        return self._table

    def forward(self, ids):
        table = self.device_table()
        flat = ids.reshape(-1).to(device="cuda", dtype=torch.int64)
        if torch.is_tensor(table):
            return table.index_select(0, flat).view(*ids.shape, -1)
        packed, scales = table
        out = torch.empty((flat.numel(), self.embedding_dim), dtype=torch.float16, device="cuda")
        for lo in range(0, flat.numel(), 32768):
            part = flat[lo:lo + 32768]
            _ok(GEMV.launch_nvfp4_decode_rows(_p(packed), _p(scales), _p(part), _p(out[lo:]),
                                              part.numel(), self.embedding_dim,
                                              self.num_embeddings, _cur_stream()),
                "launch_nvfp4_decode_rows")
        return out.view(*ids.shape, -1)


class QLinear(nn.Module):
    """A Linear whose weight is NVFP4 bytes in device memory (``d_p`` packed, ``d_s`` scales).
    One token runs the GEMV entry point, two tokens the two-activation GEMV, more the tensor-core
    GEMM, which takes and returns token-minor matrices (reference: pipeline/_qwen38_infer.py:144-184)."""

    def __init__(self, d_p, d_s, M, K, bias=None):
        super().__init__()
        self.d_p, self.d_s, self.M, self.K = d_p, d_s, M, K
        self.bias = bias

    # (pointers and the stream go to the bound entry points as plain integers: one projection of one
    # token is 3.6 us of GPU time and was 16 us of host time)
    def _one(self, x, y):
        rc = GEMV_T1(self.d_p, self.d_s, x.data_ptr(), y.data_ptr(), self.M, self.K, _stream_handle())
        if rc:
            _ok(rc, "gemv")

    def _two(self, x, y):
        p = x.data_ptr()
        rc = GEMV.launch_nvfp4_gemv2(self.d_p, self.d_s, p, p + 2 * self.K, y.data_ptr(), self.M, self.K,
                                     _stream_handle())
        if rc:
            _ok(rc, "gemv2")

    def _many(self, x, tokens):
        # x is [tokens, K] and the caller wants [tokens, M]: the token-major entry reads and writes
        # exactly that (bit-identical to transposing around launch_nvfp4_gemmtc_v5, which is what
        # the reference does: pipeline/_qwen38_infer.py:175-181).  -2 = a shape or pointer the
        # tensor-core kernel does not take: then the reference-shaped call below.
        y = torch.empty((tokens, self.M), dtype=torch.float16, device=x.device)
        rc = V5.launch_nvfp4_gemm_w4a16_ex(self.d_p, self.d_s, x.data_ptr(), self.K, y.data_ptr(), self.M,
                                           self.M, tokens, self.K, 3, _stream_handle())
        if rc == 0:
            return y
        if rc != -2:
            _ok(rc, "gemm")
        # The tensor-core kernel takes token counts that are multiples of 8 (16-byte rows for
        # its TMA loads); any other count would fall to the CUDA-core kernel, orders of magnitude
        # slower.  So the token-minor matrices are padded with zero columns and the result is cut
        # back (the reference's wmma kernel takes any count: kernels/nvfp4_cuda_v5.cu:406-422).
        padded = (tokens + 7) // 8 * 8
        if padded == tokens:
            xt = x.t().contiguous()                                   # [K, tokens]
        else:
            xt = torch.zeros((self.K, padded), dtype=torch.float16, device=x.device)
            xt[:, :tokens] = x.t()
        yt = torch.empty((self.M, padded), dtype=torch.float16, device=x.device)
        _ok(V5.launch_nvfp4_gemmtc_v5(self.d_p, self.d_s, _p(xt), _p(yt), self.M, padded, self.K,
                                      _cur_stream()), "gemm")
        return yt[:, :tokens].t().contiguous()

    def forward(self, x):
        rows = x.dim() == 2 and x.shape[1] == self.K
        flat = x if rows else x.reshape(-1, self.K)
        if flat.dtype is not torch.float16:
            flat = flat.half()
        if not flat.is_contiguous():
            flat = flat.contiguous()
        tokens = flat.shape[0]
        if tokens == 0:
            raise IndexError("QLinear: no tokens")
        if tokens <= 2:
            y = torch.empty((tokens, self.M), dtype=torch.float16, device=x.device)
            (self._one if tokens == 1 else self._two)(flat, y)
        else:
            y = self._many(flat, tokens)
        if self.bias is not None:
            y = y + self.bias
        # the view is also the check of the feature width: reshape alone takes any multiple of K
        return y if rows else y.view(*x.shape[:-1], self.M)


def st_name(name):
    """Name of a skeleton parameter in the checkpoint: the text model sits under
    ``model.language_model``; ``lm_head`` keeps its name."""
    head, sep, tail = name.partition(".")
    return f"model.language_model.{tail}" if (head == "model" and sep) else name


def _set_submodule(root, dotted: str, new):
    owner_path, _, leaf = dotted.rpartition(".")
    setattr(root.get_submodule(owner_path) if owner_path else root, leaf, new)


def patch_linears(model, index, misc):
    """Swap every ``nn.Linear`` whose weight is in the container index for a ``QLinear``;
    returns how many were swapped."""
    have = set(misc.files)
    targets = [(n, m) for n, m in model.named_modules() if isinstance(m, nn.Linear)]
    done = 0
    for dotted, lin in targets:
        entry = index.get(st_name(dotted + ".weight"))
        if entry is None:
            print(f"  [warn] no container entry for {dotted}.weight; module left untouched")
            continue
        bias = None
        if lin.bias is not None:
            key = st_name(dotted + ".bias")
            bias = (torch.from_numpy(misc[key]).half().cuda() if key in have
                    else torch.zeros(lin.bias.shape, dtype=torch.float16, device="cuda"))
        _set_submodule(model, dotted, QLinear(*upload_nvfp4(entry), entry["M"], entry["K"], bias=bias))
        done += 1
    return done


def fill_rest(model, misc, embed):
    """Load what is not a quantised matrix (norm weights, conv kernels, A_log, dt_bias, ...) from
    the misc archive.  Returns (number filled, names without a source)."""
    have = set(misc.files)
    n, missing = 0, []
    for name, param in model.named_parameters():
        if "embed_tokens" in name:
            if embed is not None:
                param.data.copy_(torch.as_tensor(np.asarray(embed)).half())
                n += 1
            continue
        key = st_name(name)
        if key not in have:
            missing.append(key)
            continue
        param.data.copy_(torch.from_numpy(misc[key]).half().reshape(param.shape))
        n += 1
    return n, missing


def rebuild_rope(model):
    """``to_empty`` leaves the rotary module's non-persistent buffers uninitialised: take them
    from a freshly constructed module.  Returns the number of modules repaired."""
    from transformers.models.qwen3_5.modeling_qwen3_5 import Qwen3_5TextRotaryEmbedding as Rotary

    fixed = 0
    for mod in model.modules():
        if not isinstance(mod, Rotary):
            continue
        donor = Rotary(mod.config, torch.device("cuda"))
        for attr in ("inv_freq", "original_inv_freq", "attention_scaling"):
            setattr(mod, attr, getattr(donor, attr))
        fixed += 1
    return fixed


def build_model(model_dir=None):
    """Directory with ``config.json`` + container -> (config, model): the third-party model
    skeleton with every Linear replaced by a QLinear and the remaining parameters loaded."""
    from transformers.models.qwen3_5.configuration_qwen3_5 import Qwen3_5TextConfig
    from transformers.models.qwen3_5.modeling_qwen3_5 import Qwen3_5ForCausalLM

    where = model_dir or MODEL_DIR
    open_container(where)

    def path(name):
        return os.path.join(where, name)

    with open(path("config.json"), encoding="utf-8") as fh:
        cfg = Qwen3_5TextConfig(**json.load(fh))
    with open(path("nvfp4_index.json"), encoding="utf-8") as fh:
        index = json.load(fh)
    misc = np.load(path("fp32_misc.npz"))
    with torch.device("meta"):                     # no storage until the weights are known
        model = Qwen3_5ForCausalLM(cfg).half()

    packed_pair = (path("nvfp4_embed_packed.npy"), path("nvfp4_embed_scales.npy"))
    default_mode = "nvfp4" if all(os.path.exists(p) for p in packed_pair) else "fp16"
    if os.environ.get("VF_EMBED", default_mode) == "nvfp4":
        table = PackedEmb(*packed_pair)
    else:
        table = torch.from_numpy(np.array(np.load(path("fp16_embed.npy"), mmap_mode="r")))
    model.model.embed_tokens = QEmbedding(table)

    swapped = patch_linears(model, index, misc)
    model.to_empty(device="cuda")
    filled, missing = fill_rest(model, misc, None)
    ropes = rebuild_rope(model)
    model.eval()
    torch.cuda.synchronize()
    print(f"  {swapped} Linear -> QLinear, {filled} other parameters, {ropes} rotary modules, "
          f"{UPLOAD_BYTES[0] / 1e9:.2f} GB of NVFP4 on the device", flush=True)
    if missing:
        print("  no source for:", missing[:10], flush=True)
    return cfg, model


# -------------------------------------------------------------------------------- decode state
def prefill(model, cache, ids, chunk=512):
    """Feed the prompt in chunks (more than two tokens per call, so every QLinear runs the GEMM);
    returns the greedy first token.  Reference flow: pipeline/_qwen38_infer.py:796-809."""
    total = ids.shape[1]
    logits = None
    with torch.no_grad():
        for lo in range(0, total, chunk):
            hi = min(total, lo + chunk)
            logits = model(ids[:, lo:hi], past_key_values=cache, use_cache=True, logits_to_keep=1,
                           cache_position=torch.arange(lo, hi, device="cuda")).logits
    return int(logits[0, -1].argmax())


_STAGE = {}


def ensure_kv_stage(model, max_len):
    """A device buffer large enough for one layer's keys (kv_heads x max_len x head_dim fp16),
    grown on demand and shared by all callers."""
    cfg = model.config
    heads = getattr(cfg, "num_key_value_heads", None) or cfg.num_attention_heads
    dim = getattr(cfg, "head_dim", None) or cfg.hidden_size // cfg.num_attention_heads
    need = heads * max_len * dim
    if _STAGE.get("elems", 0) < need:
        _STAGE["buf"] = torch.empty(need, dtype=torch.float16, device="cuda")
        _STAGE["elems"] = need
    return _STAGE["buf"]


def _attention_layers(model, cache):
    for i, layer in enumerate(model.model.layers):
        if _kind(layer) == "full_attention":
            yield i, layer.self_attn, cache.layers[i]


def _linear_layers(model, cache):
    for i, layer in enumerate(model.model.layers):
        if _kind(layer) == "linear_attention":
            yield i, layer.linear_attn, cache.layers[i]


def snap_decode_state(model, cache, prompt_len):
    """Host copy of what graph warm-up and capture disturb in the attention layers: the first
    ``prompt_len`` cache positions and the length counter.  [(layer, keys, values, length)]"""
    return [(i, slot.keys[:, :, :prompt_len].cpu(), slot.values[:, :, :prompt_len].cpu(),
             slot.cumulative_length.cpu())
            for i, _, slot in _attention_layers(model, cache)]


def restore_decode_state(model, cache, snap, prompt_len):
    for i, keys, values, length in snap:
        slot = cache.layers[i]
        slot.keys[:, :, :prompt_len].copy_(keys)
        slot.values[:, :, :prompt_len].copy_(values)
        slot.cumulative_length.copy_(length)


def _load_deltanet_state(mod, slot):
    # the cache keeps the recurrent state as [head][key][value]; the kernel wants [head][value][key]
    mod._vf_S.view(slot.recurrent_states[0].shape).copy_(slot.recurrent_states[0].transpose(1, 2))
    mod._vf_conv.copy_(slot.conv_states[0].reshape(-1))               # [channel][tap]


def refresh_deltanet_state(model, cache):
    """After another prefill into the same cache: reload the fused kernel's state buffers."""
    for _, mod, slot in _linear_layers(model, cache):
        _load_deltanet_state(mod, slot)


# ----------------------------------------------------------------------------------- operators
def _keep_original(mod, slot_name):
    """Remember ``mod.forward`` under ``slot_name`` the first time a module is patched."""
    if not hasattr(mod, slot_name):
        setattr(mod, slot_name, mod.forward)
    return getattr(mod, slot_name)


class _DeltaNetStep:
    """forward() of a linear-attention layer for one or two tokens: four projections, then per
    token one fused conv + gated delta rule + gated norm launch, then the output projection."""

    def __init__(self, mod, lib, keep_backup):
        self.mod, self.lib = mod, lib
        self.original = _keep_original(mod, "_vf_orig")
        channels, nv = mod.conv_dim, mod.num_v_heads
        dev = "cuda"
        mod._vf_conv = torch.zeros(channels * 4, dtype=torch.float16, device=dev)
        mod._vf_S = torch.zeros(nv * 128 * 128, dtype=torch.float32, device=dev)
        mod._vf_S_bak = torch.zeros_like(mod._vf_S) if keep_backup else None
        mod._vf_conv_bak = torch.zeros_like(mod._vf_conv) if keep_backup else None
        mod._vf_fast = True
        self.scratch = torch.zeros(channels, dtype=torch.float32, device=dev)
        self.outs = [torch.zeros(nv * 128, dtype=torch.float16, device=dev) for _ in range(2)]
        self.taps = mod.conv1d.weight.detach().reshape(channels, 4).half().contiguous()
        norm = mod.norm
        self.eps = float(getattr(norm, "variance_epsilon", getattr(norm, "eps", 1e-6)))
        self.reference_heads = (mod.num_k_heads, nv) == (16, 48)

    def _launch(self, mixed, z, b, a, out):
        m = self.mod
        ptrs = [_p(t) for t in (mixed, z, b, a, self.taps, m._vf_conv, m.A_log, m.dt_bias,
                                m.norm.weight, m._vf_S, self.scratch, out)]
        if self.reference_heads:
            rc = self.lib.launch_dn_fused(*ptrs, self.eps, _cur_stream())
        else:
            rc = self.lib.launch_dn_fused_heads(*ptrs, m.num_k_heads, m.num_v_heads, self.eps,
                                                _cur_stream())
        _ok(rc, "launch_dn_fused")

    def __call__(self, hidden_states, cache_params=None, attention_mask=None, **kw):
        tokens = hidden_states.shape[1]
        if tokens > 2:
            return self.original(hidden_states, cache_params=cache_params,
                                 attention_mask=attention_mask, **kw)
        m = self.mod
        proj = [f(hidden_states)[0] for f in (m.in_proj_qkv, m.in_proj_z, m.in_proj_b, m.in_proj_a)]
        if m._vf_S_bak is not None:          # state before this call, for a rejected draft token
            m._vf_S_bak.copy_(m._vf_S)
            m._vf_conv_bak.copy_(m._vf_conv)
        for t in range(tokens):
            self._launch(*(x[t].contiguous() for x in proj), self.outs[t])
        y = self.outs[0] if tokens == 1 else torch.stack(self.outs)
        return m.out_proj(y.view(1, tokens, -1))


def patch_fused_deltanet(model, cache, mtp=True):
    """Give every linear-attention layer the fused decode step.  Must run AFTER a prefill: the
    conv window and the recurrent state are taken from the cache.  ``mtp`` keeps a backup of the
    state taken at the start of each call.  Returns the patched modules; their ``_vf_conv`` /
    ``_vf_S`` tensors are the live state (reference: pipeline/_qwen38_infer.py:425-510)."""
    lib = _bound_library("nvfp4_dn_fused.dll")
    patched = []
    for _, mod, slot in _linear_layers(model, cache):
        mod.forward = _DeltaNetStep(mod, lib, mtp)
        _load_deltanet_state(mod, slot)
        patched.append(mod)
    return patched


class _AttentionStep:
    """forward() of a full-attention layer for one token: projections, q/k norm, rotary and the
    cache update stay with the model code; scores, softmax, weighted sum and the output gate are
    one fused launch reading the cache in place."""

    def __init__(self, mod, slot, lib, max_len):
        self.mod, self.slot, self.lib, self.max_len = mod, slot, lib, int(max_len)
        self.original = _keep_original(mod, "_vf_attn_orig")
        mod._vf_attn = True
        cfg = mod.config
        self.hq, self.hkv = cfg.num_attention_heads, cfg.num_key_value_heads
        self.ctx = torch.zeros(self.hq * mod.head_dim, dtype=torch.float16, device="cuda")

    def __call__(self, hidden_states, position_embeddings=None, attention_mask=None,
                 past_key_values=None, **kw):
        if hidden_states.shape[1] != 1 or past_key_values is None:
            return self.original(hidden_states, position_embeddings=position_embeddings,
                                 attention_mask=attention_mask, past_key_values=past_key_values,
                                 **kw)
        from transformers.models.qwen3_5 import modeling_qwen3_5 as hf

        m, dim = self.mod, self.mod.head_dim
        # q_proj emits, per head, [query | gate]
        per_head = m.q_proj(hidden_states).view(1, 1, self.hq, 2 * dim)
        q = m.q_norm(per_head[..., :dim]).transpose(1, 2)
        gate = per_head[..., dim:].reshape(-1).contiguous()
        k = m.k_norm(m.k_proj(hidden_states).view(1, 1, self.hkv, dim)).transpose(1, 2)
        v = m.v_proj(hidden_states).view(1, 1, self.hkv, dim).transpose(1, 2)
        q, k = hf.apply_rotary_pos_emb(q, k, *position_embeddings)
        keys, values = past_key_values.update(k, v, m.layer_idx)
        q = q.contiguous()
        head = (_p(q), _p(keys), _p(values), _p(self.slot.cumulative_length), _p(gate), _p(self.ctx))
        if (self.hq, self.hkv) == (24, 4):
            rc = self.lib.launch_attn_decode(*head, self.max_len, float(m.scaling), _cur_stream())
        else:
            rc = self.lib.launch_attn_decode_heads(*head, self.max_len, self.hq, self.hkv,
                                                   float(m.scaling), _cur_stream())
        _ok(rc, f"launch_attn_decode (layer {m.layer_idx})")
        return m.o_proj(self.ctx.view(1, 1, -1)), None


def patch_attn_decode(model, cache, max_len=3072):
    """Give every full-attention layer the fused single-token attention.  ``max_len`` is the
    cache's length (row pitch of its key/value tensors).  Returns the patched modules."""
    lib = _bound_library("nvfp4_attn_decode.dll")
    patched = []
    for _, mod, slot in _attention_layers(model, cache):
        mod.forward = _AttentionStep(mod, slot, lib, max_len)
        patched.append(mod)
    return patched


class _NormStep:
    """Zero-centred RMSNorm of fp16 rows, one launch: f16(f32(x) * rsqrt(mean(x^2) + eps) * (1 + w))."""

    def __init__(self, mod, lib):
        self.mod, self.lib = mod, lib
        self.original = _keep_original(mod, "_vf_norm_orig")
        mod._vf_norm = True
        self.one_plus_w = (mod.weight.float() + 1.0).contiguous()
        self.out = None

    def __call__(self, x):
        width = x.shape[-1]
        rows = x.numel() // width if width else 0
        single_token = x.dim() < 2 or x.shape[1] == 1
        if not (single_token and rows > 0 and x.dtype == torch.float16 and x.stride(-1) == 1):
            return self.original(x)                                   # prefill, odd layouts
        if self.out is None or self.out.shape != (rows, width):
            self.out = torch.empty((rows, width), dtype=torch.float16, device=x.device)
        _ok(self.lib.launch_rmsnorm(_p(x), x.stride(-2), _p(self.one_plus_w), _p(self.out), rows,
                                    width, float(self.mod.eps), _cur_stream()), "launch_rmsnorm")
        return self.out.view(x.shape)


def patch_rmsnorm(model):
    """Route every ``Qwen3_5RMSNorm`` through the fused kernel at decode shapes (hidden-size rows
    and the strided per-head q/k norms).  Returns the patched modules."""
    lib = _bound_library("nvfp4_rmsnorm.dll")
    patched = [m for m in model.modules() if type(m).__name__ == "Qwen3_5RMSNorm"]
    for mod in patched:
        mod.forward = _NormStep(mod, lib)
    return patched


def patch_rope():
    """Replace the model code's module-level ``apply_rotary_pos_emb`` by the fused q+k kernel for
    the decode case (batch 1, one token, 256 rotated dims, fp16); every other call goes to the
    original, kept as ``modeling_qwen3_5._vf_rope_orig``."""
    from transformers.models.qwen3_5 import modeling_qwen3_5 as hf

    lib = _bound_library("nvfp4_rope_silu.dll")
    if getattr(hf, "_vf_rope_orig", None) is None:
        hf._vf_rope_orig = hf.apply_rotary_pos_emb
    plain = hf._vf_rope_orig

    def rotary(q, k, cos, sin, unsqueeze_dim=1):
        decode_shape = (q.dim() == 4 and q.shape[0] == 1 and q.shape[2] == 1 and
                        q.shape[3] == 256 and cos.shape[-1] == 256)
        if not (decode_shape and q.dtype == k.dtype == torch.float16):
            return plain(q, k, cos, sin, unsqueeze_dim=unsqueeze_dim)
        q_in, k_in = q.contiguous(), k.contiguous()
        table = [t.reshape(-1).half().contiguous() for t in (cos, sin)]
        q_out, k_out = torch.empty_like(q_in), torch.empty_like(k_in)
        _ok(lib.launch_rope_qk(_p(q_in), _p(k_in), _p(table[0]), _p(table[1]), _p(q_out), _p(k_out),
                               q.shape[1], k.shape[1], _cur_stream()), "launch_rope_qk")
        return q_out, k_out

    hf.apply_rotary_pos_emb = rotary
    return rotary


class _MlpStep:
    """down(silu(gate(x)) * up(x)) for one token with the activation and product in one launch."""

    def __init__(self, mod, lib):
        self.mod, self.lib = mod, lib
        self.original = _keep_original(mod, "_vf_mlp_orig")
        mod._vf_mlp = True
        self.act = None

    def __call__(self, x):
        if x.numel() != x.shape[-1] or x.dtype != torch.float16:
            return self.original(x)
        m = self.mod
        gate, up = m.gate_proj(x), m.up_proj(x)
        if self.act is None or self.act.numel() != gate.numel():
            self.act = torch.empty(gate.numel(), dtype=torch.float16, device=x.device)
        _ok(self.lib.launch_silu_mul(_p(gate), _p(up), _p(self.act), gate.numel(), _cur_stream()),
            "launch_silu_mul")
        return m.down_proj(self.act.view(gate.shape))


def patch_mlp_silu_mul(model):
    lib = _bound_library("nvfp4_rope_silu.dll")
    patched = [m for m in model.modules() if type(m).__name__ == "Qwen3_5MLP"]
    for mod in patched:
        mod.forward = _MlpStep(mod, lib)
    return patched


# ---------------------------------------------------------------------------------- step graph
class GraphDecoder:
    """One decode step of the (patched) model as a CUDA graph: forward, logits copy, argmax and
    the cache-position increment are all inside the capture; a replay needs only the next token's
    embedding row and the rotary position.

    Construction runs ``n_warmup`` eager steps and the capture itself, each of which advances the
    cache and the DeltaNet state: snapshot before, restore after, then ``reset_pos()``.
    ``static_pos`` lets several decoders share one device-side position tensor.
    Reference: pipeline/_qwen38_infer.py:653-729."""

    def __init__(self, model, cache, first_pos, hid, n_warmup=3, static_pos=None, use_pos4=True):
        dev = "cuda"
        self.first_pos = self.rope_pos = first_pos
        self._own_pos = static_pos is None
        self.static_pos = (torch.tensor([first_pos, first_pos + 1], device=dev)
                           if static_pos is None else static_pos)
        self.pos2 = self.static_pos[:1].view(1)              # cache_position: a live view
        self.pos4 = torch.zeros(4, 1, 1, dtype=torch.long, device=dev)   # rotary position ids
        self.static_embeds = torch.zeros(1, 1, hid, dtype=torch.float16, device=dev)
        self.static_logits = torch.zeros(1, model.lm_head.M, dtype=torch.float16, device=dev)
        self.static_next = torch.zeros(1, dtype=torch.long, device=dev)
        self.pin = torch.empty(hid, dtype=torch.float16, pin_memory=True)
        self._tables = {}                                     # id(host table) -> device copy
        extra = {"position_ids": self.pos4} if use_pos4 else {}

        def body():
            logits = model(inputs_embeds=self.static_embeds, past_key_values=cache, use_cache=True,
                           cache_position=self.pos2, **extra).logits[:, -1, :]
            self.static_logits.copy_(logits)
            self.static_next.copy_(logits.argmax(dim=-1))
            self.static_pos.add_(1)

        self._one_step = body
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(side):
            for _ in range(n_warmup):
                self.pos4.fill_(int(self.static_pos[0]))
                body()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(self.graph):
            body()

    def set_pos(self, p):
        self.first_pos = self.rope_pos = p
        self.static_pos.copy_(torch.tensor([p, p + 1]))

    def reset_pos(self):
        self.set_pos(self.first_pos)

    def _embedding_row(self, tok_id, emb_w):
        if torch.is_tensor(emb_w) and emb_w.dtype == torch.float16:
            key = id(emb_w)
            if key not in self._tables:                       # dense table: one upload, then
                self._tables[key] = emb_w.to("cuda")          # every row is a device-side copy
            self.static_embeds.view(-1).copy_(self._tables[key][tok_id])
        else:                                                 # packed table: host decode
            self.pin.copy_(emb_w[tok_id])
            self.static_embeds.view(-1).copy_(self.pin, non_blocking=True)

    def _replay(self, tok_id, emb_w):
        self._embedding_row(tok_id, emb_w)
        self.pos4.fill_(self.rope_pos)
        self.graph.replay()
        self.rope_pos += 1

    def step(self, tok_id, emb_w):
        self._replay(tok_id, emb_w)
        return int(self.static_next.item())

    def step_logits(self, tok_id, emb_w):
        self._replay(tok_id, emb_w)
        return int(self.static_next.item()), self.static_logits


class GraphDecoder2:
    """Two tokens per replay, for speculative verification: the graph runs the model on
    [tokA, tokB] at positions [p, p + 1]; ``static_next[0]`` / ``static_logits[0]`` are the
    prediction after tokA (which accepts or rejects the draft tokB), index 1 the prediction after
    tokB (the bonus token when the draft is accepted).  Every QLinear takes the two-activation
    GEMV, the DeltaNet layers two fused steps (with a state backup for a rejected draft); attention,
    norms, rotary and the MLP product fall back to the model code for two tokens.
    ``static_pos`` (device int64 [2] = [p, p + 1]) is shared with a ``GraphDecoder`` and advanced
    by one per replay; the caller re-aligns it every round.
    Reference: pipeline/_qwen38_infer.py:732-773."""

    def __init__(self, model, cache, first_pos, hid, static_pos, n_warmup=3):
        dev = "cuda"
        self.first_pos = first_pos
        self.static_pos = static_pos
        self.static_embeds = torch.zeros(1, 2, hid, dtype=torch.float16, device=dev)
        self.static_logits = torch.zeros(2, model.lm_head.M, dtype=torch.float16, device=dev)
        self.static_next = torch.zeros(2, dtype=torch.long, device=dev)
        self._pins = [torch.empty(hid, dtype=torch.float16, pin_memory=True) for _ in range(2)]
        self._tables = {}

        def body():
            both = model(inputs_embeds=self.static_embeds, past_key_values=cache, use_cache=True,
                         cache_position=self.static_pos).logits[0, -2:, :]
            self.static_logits.copy_(both)
            self.static_next.copy_(both.argmax(dim=-1))
            self.static_pos.add_(1)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(side):
            for _ in range(n_warmup):
                body()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(self.graph):
            body()

    def _put(self, slot, tok_id, emb_w):
        dst = self.static_embeds[0, slot]
        if torch.is_tensor(emb_w) and emb_w.dtype == torch.float16:
            key = id(emb_w)
            if key not in self._tables:
                self._tables[key] = emb_w.to("cuda")
            dst.copy_(self._tables[key][tok_id])
        else:
            self._pins[slot].copy_(emb_w[tok_id])
            dst.copy_(self._pins[slot], non_blocking=True)

    def step2(self, tokA, tokB, emb_w):
        """Replay on (tokA, tokB); returns (argmax int64 [2], logits fp16 [2, V]), both device
        tensors that the next replay overwrites."""
        self._put(0, tokA, emb_w)
        self._put(1, tokB, emb_w)
        self.graph.replay()
        return self.static_next, self.static_logits

