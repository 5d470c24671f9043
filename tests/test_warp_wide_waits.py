"""Source check: a warp that issues tensor-core instructions as a whole never parts on a wait.

MMAs and commits go through elect.sync with a full mask, tcgen05.ld / st are .aligned: all 32 lanes must
arrive.  A bounded wait gives each lane its own answer, so a wait that runs out on some lanes only must not
send them another way: no branch or loop of such a role depends on it beyond skipping further waits, and
.aligned accesses stand behind a __syncwarp."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nvfp4_v100_b200", "csrc")
WAITS = r"\b(?:mbar_wait|f4_wait|tc_wait|tc_wait_poll|few_wait|gp_wait|atc_wait)\("
ELECTED = r"\b(?:tcgen05_mma_f16|tcgen05_mma_f16_ta|tcgen05_mma_fp4_block16|tc_mma|gp_mma|tcgen05_commit|gp_commit)\("
ALIGNED = r"\b(?:tcgen05_st_32x32b_x16|tcgen05_ld_32x32b_x16|tcgen05_ld_32x32b_x32|few_ld_x8)\("


def _block(text, start):
    """The braced block that opens at or after `start`."""
    at = text.index("{", start)
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("unbalanced braces")


def _roles(name, pattern, one_thread=False):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"if \(warp (?:==|>=) \d+\)", text):
        body = _block(text, m.end())
        one = re.match(r"\{\s*if \(lane == 0", body)              # one thread's loop: nothing to agree on
        if bool(one) == one_thread and re.search(pattern, body):
            yield m.group(0), body


@pytest.mark.parametrize("name", ["gemm.cu", "gemm_few.cu", "gemm_pair.cu", "gemm_fp4.cu", "gemv_tc.cu", "attn_prefill_tc.cu"])
def test_issuing_roles_go_on_whatever_a_wait_answers(name):
    waits = 0
    for where, body in _roles(name, ELECTED):
        for m in re.finditer(WAITS, body):
            waits += 1
            start = max(body.rfind(c, 0, m.start()) for c in ";{}") + 1
            statement = " ".join(body[start:body.index(";", m.end())].split())
            assert re.match(r"(?:if \(ok(?: && \w+(?: > 0)?)?\) |bool )ok = " + WAITS, statement), (name, where, statement)
        for loop in re.findall(r"for \([^{;]*;[^{;]*;", body):
            assert not re.search(r"\bok\b|piece\(|slot\(", loop), (name, where, loop)
        for m in re.finditer(r"\bok\b", body):
            rest = body[m.end():m.end() + 40]
            assert not re.match(r"\) (?:break|return|\{)|\) scores", rest), (name, where, rest)
    assert waits, "no issuing role found: the pattern no longer fits the source"


@pytest.mark.parametrize("name", ["gemm_few.cu", "gemm_pair.cu", "attn_prefill_tc.cu"])
def test_aligned_accesses_stand_behind_a_syncwarp(name):
    seen = 0
    for where, body in _roles(name, ALIGNED):
        events = sorted((m.start(), kind) for kind, p in (("wait", WAITS), ("sync", r"__syncwarp\(\)"), ("access", ALIGNED))
                        for m in re.finditer(p, body))
        parted = False
        for at, kind in events:
            assert not (kind == "access" and parted), (name, where, body[at:at + 60])
            seen += kind == "access"
            parted = kind == "wait" or (parted and kind != "sync")
    assert seen, "no such role found: the pattern no longer fits the source"


@pytest.mark.parametrize("name,rings", [("gemm_few.cu", {"bar_full", "bar_ready"}), ("gemm_pair.cu", {"bar_full", "bar_ready"}),
                                        ("attn_prefill_tc.cu", {"bar_full", "bar_q"})])
def test_copies_are_waited_for_before_the_cta_leaves(name, rings):
    # a thread that stops copying early (its own wait ran out) has copies in flight: behind the last
    # copy, that thread (thread 0, or the first of its role) waits for every barrier that copies complete
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    kernel = _block(text, text.index("__global__"))
    roles = [b for _, b in _roles(name, r"\b(?:tma_load_\w+|request)\(", one_thread=True)]
    assert roles
    waited = set()
    for body in roles:
        last = max(m.start() for m in re.finditer(r"\b(?:tma_load_\w+|request)\(|\bbreak;", body))
        waited |= set(re.findall(r"_wait\(smem_u32\(&(\w+)", body[last:]))
    for m in re.finditer(r"if \(threadIdx\.x == 0 && s_ran_out\)", kernel):
        waited |= set(re.findall(r"_wait\(smem_u32\(&(\w+)", _block(kernel, m.end())))
    assert rings <= waited
