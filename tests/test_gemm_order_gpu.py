"""W4A16 GEMMs directly behind a kernel that writes their weights and lets its successor start early.

The writer is the chunk attention of one token over 4001 keys: its CTAs allow the next kernel to start
when they begin and store their results 0.2 ms later.  Its 16384 fp16 outputs are taken as the packed
bytes of a 256 x 256 matrix (any byte is two weights)."""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu
M = K = 256
KEYS = 4001


class Writer:
    def __init__(self, lib):
        g = torch.Generator(device="cuda")
        g.manual_seed(1)
        r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
        self.lib, self.q, self.gate, self.keys = lib, r(64 * 256), r(64 * 256), r(KEYS, 256)
        self.values = [r(KEYS, 256), r(KEYS, 256)]
        self.packed = torch.zeros(M * K // 4, dtype=torch.float16, device="cuda")
        self.scales = torch.randint(118, 123, (M * K // 16,), dtype=torch.uint8, device="cuda", generator=g)

    def __call__(self, which):
        assert self.lib.launch_attn_prefill(ptr(self.q), ptr(self.keys), ptr(self.values[which]), KEYS, 1,
                                            ptr(self.gate), ptr(self.packed), KEYS, 64, 1, 1 / 16, stream()) == 0


def _check(writer, product, between, new_out):
    want = []
    for w in (0, 1):
        writer(w)
        torch.cuda.synchronize()
        want.append(new_out())
        product(want[w])
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    outs = [new_out() for _ in range(12)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        writer(i & 1)
        between()
        product(o)
    torch.cuda.synchronize()
    assert [i for i, o in enumerate(outs) if not torch.equal(o, want[i & 1])] == []


@pytest.mark.parametrize("tokens", [8, 64, 128, 136, 512])
@pytest.mark.parametrize("entry", ["token-major", "token-minor"])
def test_new_weights_are_seen(lib, tokens, entry):
    w = Writer(lib)
    x = torch.randn((tokens, K), device="cuda").half()
    if entry == "token-minor":
        x = x.t().contiguous()

    def gemm(o):
        if entry == "token-major":
            rc = lib.launch_nvfp4_gemm_w4a16_ex(ptr(w.packed), ptr(w.scales), ptr(x), K, ptr(o), M, M, tokens, K, 3,
                                                stream())
        else:
            rc = lib.launch_nvfp4_gemmtc_v5(ptr(w.packed), ptr(w.scales), ptr(x), ptr(o), M, tokens, K, stream())
        assert rc == 0

    _check(w, gemm, lambda: None, lambda: torch.empty(M * tokens, dtype=torch.float16, device="cuda"))


@pytest.mark.parametrize("tokens", [8, 136])
@pytest.mark.parametrize("entry", ["launch_nvfp4_gemv_v8", "launch_nvfp4_gemv_tc"])
def test_gemv_behind_a_gemm_sees_weights_written_in_front_of_it(lib, tokens, entry):
    # a GEMV may request weights before the kernel in front of it has finished; the GEMM in front of
    # it does not let it start before the writer in front of the GEMM has
    w = Writer(lib)
    x = torch.randn((tokens, K), device="cuda").half()
    y = torch.empty((tokens, M), dtype=torch.float16, device="cuda")
    other = torch.randint(0, 256, (M * K // 2,), dtype=torch.uint8, device="cuda")
    a = torch.randn(K, device="cuda").half()
    assert lib.nvfp4_gemv_tc_prepare() == 0

    def gemm():
        assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(other), ptr(w.scales), ptr(x), K, ptr(y), M, M, tokens, K, 3,
                                              stream()) == 0

    def gemv(o):
        assert getattr(lib, entry)(ptr(w.packed), ptr(w.scales), ptr(a), ptr(o), M, K, stream()) == 0

    _check(w, gemv, gemm, lambda: torch.empty(M, dtype=torch.float16, device="cuda"))
