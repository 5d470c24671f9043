"""Split decode attention for every number of query heads a CTA may share (1, 2, 3), against float64."""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("hq,hkv,max_len", [(24, 4, 4100), (3, 1, 600), (20, 4, 600), (32, 2, 600), (64, 1, 600), (19, 19, 300),
                                           (96, 8, 600), (320, 8, 300)])   # 32 and 160 head groups: 4 CTAs and 1 a group
def test_against_float64(lib, hq, hkv, max_len):
    g = torch.Generator(device="cuda")
    g.manual_seed(hq * 100 + hkv)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    q, gate, keys, vals = r(hq, D), r(hq, D), r(hkv, max_len, D), r(hkv, max_len, D)
    scratch = torch.zeros(lib.nvfp4_attn_split_scratch_bytes(hq), dtype=torch.uint8, device="cuda")
    rep = hq // hkv
    for L in (0, 1, 16, 17, 64, 65, 129, 257, max_len - 3, max_len):
        k, v = keys.clone(), vals.clone()
        k[:, L:], v[:, L:] = float("nan"), float("inf")          # never read
        ln = torch.tensor([L], dtype=torch.int64, device="cuda")
        out = torch.full((hq, D), 7.0, dtype=torch.float16, device="cuda")
        for _ in range(2):                                       # the counters are ready for the next launch
            assert lib.launch_attn_decode_split(ptr(q), ptr(k), ptr(v), ptr(ln), ptr(gate), ptr(out), ptr(scratch),
                                                max_len, hq, hkv, 1 / 16, stream()) == 0
        torch.cuda.synchronize()
        if L == 0:                                               # no key at all: 0 / 0, as in fp32
            assert out.isnan().all()
            continue
        kd, vd = (t[:, :L].double().repeat_interleave(rep, 0) for t in (k, v))
        s = torch.einsum("hd,hld->hl", q.double(), kd) / 16
        o = torch.einsum("hl,hld->hd", torch.softmax(s, -1), vd)
        want = o.half().double() * torch.sigmoid(gate.double()).half().double()
        # one fp16 step in the rounded sum and one in the product, and the fp32 sums
        bound = want.abs() * 2 ** -9 + vd.abs().max() * (2 ** -20 + s.abs().max() * 2 ** -21)
        assert ((out.double() - want).abs() <= bound).all(), L


@pytest.mark.parametrize("hq,hkv", [(24, 4), (32, 2)])
@pytest.mark.parametrize("gate_at,out_at", [(1, 0), (0, 1), (1, 1), (2, 3)])
def test_gate_and_output_need_no_more_than_two_byte_alignment(lib, hq, hkv, gate_at, out_at):
    g = torch.Generator(device="cuda")
    g.manual_seed(hq)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    max_len = 700
    q, gate, keys, vals = r(hq, D), r(hq * D), r(hkv, max_len, D), r(hkv, max_len, D)
    scratch = torch.zeros(lib.nvfp4_attn_split_scratch_bytes(hq), dtype=torch.uint8, device="cuda")
    gate_view = torch.empty(hq * D + 4, dtype=torch.float16, device="cuda")[gate_at:gate_at + hq * D]
    gate_view.copy_(gate)
    for L in (1, 300, 700):
        ln = torch.tensor([L], dtype=torch.int64, device="cuda")
        room = torch.full((2, hq * D + 8), 7.0, dtype=torch.float16, device="cuda")
        outs = [room[0, :hq * D], room[1, out_at:out_at + hq * D]]
        for gt, out in zip((gate, gate_view), outs):
            assert lib.launch_attn_decode_split(ptr(q), ptr(keys), ptr(vals), ptr(ln), ptr(gt), ptr(out), ptr(scratch),
                                                max_len, hq, hkv, 1 / 16, stream()) == 0
        torch.cuda.synchronize()
        # One head a CTA or several: sums in another order, each within the bound of the test above (scores
        # here stay below 8), and outputs that cancel to almost nothing differ by that and not by a step.
        a, b = outs[0].double(), outs[1].double()
        bound = a.abs() * 2 ** -9 + 2 * vals.double().abs().max() * (2 ** -20 + 8 * 2 ** -21)
        assert ((a - b).abs() <= bound).all()
        assert (room[1, :out_at] == 7).all() and (room[1, out_at + hq * D:] == 7).all()
