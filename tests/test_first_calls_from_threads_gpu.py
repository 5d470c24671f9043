"""First calls of one entry point from several threads at once, in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DELTANET = """
import threading
import torch
from nvfp4_v100_b200 import _lib
from tests.gpu_util import ptr

lib = _lib.load()
HEADS = [1, 19, 37, 56, 74, 100, 148, 2]      # the scan's padding differs from head count to head count
n = 5
start, codes = threading.Barrier(len(HEADS)), {}

def call(nv):
    C = (2 + nv) * 128
    ld = C + nv * 128 + 2 * nv
    ld += -ld % 4
    z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    x, cw, cs, al, dt, nw, out = z(n, ld), z(C, 4), z(C, 4), z(nv), z(nv), z(128), z(n, nv * 128)
    state = torch.zeros((nv, 128, 128), device="cuda")
    nbytes = lib.nvfp4_dn_prefill_work_bytes(n, 1, nv)
    work = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    start.wait()
    codes[nv] = [lib.launch_dn_prefill(ptr(x), ld, ptr(cw), ptr(cs), ptr(al), ptr(dt), ptr(nw), ptr(state), ptr(work),
                                       nbytes, ptr(out), n, 1, nv, 1e-6, side.cuda_stream) for _ in range(20)]
    side.synchronize()

threads = [threading.Thread(target=call, args=(nv,)) for nv in HEADS]
for t in threads:
    t.start()
for t in threads:
    t.join()
assert codes == {nv: [0] * 20 for nv in HEADS}, codes
"""


ATTENTION = """
import threading
import torch
from nvfp4_v100_b200 import _lib
from tests.gpu_util import ptr

lib = _lib.load()
CONTEXTS = [3000, 300, 2000, 600, 3900, 1200, 900, 2500]      # one query: scores of its keys in shared memory
start, codes = threading.Barrier(len(CONTEXTS)), {}

def call(keys):
    z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    q, gate, k, v, out = z(256), z(256), z(keys, 256), z(keys, 256), z(256)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    start.wait()
    codes[keys] = [lib.launch_attn_prefill(ptr(q), ptr(k), ptr(v), keys, 1, ptr(gate), ptr(out), keys, 1, 1, 0.0625,
                                           side.cuda_stream) for _ in range(20)]
    side.synchronize()

threads = [threading.Thread(target=call, args=(keys,)) for keys in CONTEXTS]
for t in threads:
    t.start()
for t in threads:
    t.join()
assert codes == {keys: [0] * 20 for keys in CONTEXTS}, codes
"""


GEMM = """
import threading
import torch
from nvfp4_v100_b200 import _lib
from tests.gpu_util import ptr

lib = _lib.load()
TOKENS = [1, 20, 40, 100, 130, 300, 600, 1100]      # every kernel has tensor maps made for it, by an encoder looked up once
start, codes = threading.Barrier(len(TOKENS)), {}

def call(n):
    M, K = 512, 1024
    z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    p, s = (torch.zeros(M * K // d, dtype=torch.uint8, device="cuda") for d in (2, 16))
    x, out, side = z(n, K), z(n, M), torch.cuda.Stream()
    torch.cuda.synchronize()
    start.wait()
    codes[n] = [lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(x), K, ptr(out), M, M, n, K, 3, side.cuda_stream)
                for _ in range(20)]
    side.synchronize()

threads = [threading.Thread(target=call, args=(n,)) for n in TOKENS]
for t in threads:
    t.start()
for t in threads:
    t.join()
assert codes == {n: [0] * 20 for n in TOKENS}, codes
"""


@pytest.mark.parametrize("program", [DELTANET, ATTENTION, GEMM], ids=["deltanet", "attention", "gemm"])
def test_no_call_fails(program):
    for _ in range(4):
        subprocess.run([sys.executable, "-c", program], cwd=ROOT, check=True, timeout=120)
