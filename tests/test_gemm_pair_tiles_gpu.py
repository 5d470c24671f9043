"""The W4A16 pair GEMM over all its token tiles, with one tile a pair and with several in turn, against the tile
kernel: every output is the same sum in the same order, so the bits are equal.  (tests/test_gemm_pair_gpu.py has
the comparison with float64.)"""
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def config(lib):
    yield
    lib.nvfp4_b200_gemm_config(3)


# token tile on 74 pairs: (one tile a pair) 128, 192, 224, 128 in three groups of columns; (several) 160 with the
# last pair's second tile, 224, 192 with a single column, 256 and 224 with ragged groups of columns and rows
@pytest.mark.parametrize("M,n,K", [
    (4000, 250, 512), (2300, 1500, 256), (18944, 224, 256), (300, 2600, 512),
    (18945, 257, 1280), (19000, 600, 512), (30000, 190, 768), (4096, 4400, 256), (2049, 5000, 512),
])
@pytest.mark.parametrize("flags", [0, 1, 2, 3, 6, 7])
def test_same_bits_as_the_tile_kernel(lib, M, n, K, flags):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + n)
    p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    s = torch.randint(118, 123, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
    n8 = (n + 7) // 8 * 8
    act = torch.randn((n, K) if flags & 1 else (K, n8), device="cuda", generator=g).half()
    ld = M + (M % 2) * 3 if flags & 2 else n8              # odd M: rows of a stride that is a multiple of 4, not of 8
    old = torch.randn((n if flags & 2 else M, ld), device="cuda", generator=g).half()
    outs = []
    for config in (7, 1):                                  # pairs wherever they can run; tiles only
        lib.nvfp4_b200_gemm_config(config)
        outs.append(torch.cat([old.flatten(), torch.full((64,), 7.0, dtype=torch.float16, device="cuda")]))
        assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(act), act.shape[1], ptr(outs[-1]), ld, M, n, K,
                                              flags, stream()) == 0
    torch.cuda.synchronize()
    assert lib.nvfp4_gemm_status(0) == 0
    assert torch.equal(outs[0], outs[1])
    assert (outs[0][-64:] == 7).all()
    if flags & 2 and ld > M:
        assert torch.equal(outs[0][:-64].view(n, ld)[:, M:], old[:, M:])


def test_launches_side_by_side(lib):
    # two streams share nothing but the GPU; each result as if alone, launch after launch into the same buffers
    jobs = []
    for seed, (M, n, K) in enumerate(((19000, 300, 512), (4096, 2048, 768))):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
        s = torch.randint(118, 123, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
        x = torch.randn((n, K), device="cuda", generator=g).half()
        jobs.append((M, n, K, p, s, x, [torch.zeros((n, M), dtype=torch.float16, device="cuda") for _ in range(9)]))
    lib.nvfp4_b200_gemm_config(7)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in jobs]
    for i in range(9):
        for (M, n, K, p, s, x, outs), st in zip(jobs, streams):
            with torch.cuda.stream(st):
                assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(x), K, ptr(outs[i]), M, M, n, K, 3, stream()) == 0
        if i == 0:
            torch.cuda.synchronize()                       # the first of each by itself
    torch.cuda.synchronize()
    assert lib.nvfp4_gemm_status(0) == 0
    for job in jobs:
        assert all(torch.equal(job[-1][0], o) for o in job[-1][1:])


# fused: 192, 256 (groups of columns), 160 and 224 tokens a tile, the last rows of a tile missing; in two
# launches: short K, one tile a pair, few tokens, K of 64
@pytest.mark.parametrize("M,n,K", [
    (30000, 190, 4096), (4096, 4400, 2560), (18960, 257, 5120), (2064, 4999, 5120),
    (34816, 512, 256), (2064, 300, 512), (4096, 27, 512), (4096, 300, 64),
])
@pytest.mark.parametrize("wide", [False, True])
def test_gate_up_with_the_activation(lib, M, n, K, wide):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + n)
    p = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    # wide: up to infinite and NaN outputs
    s = torch.randint(108, 134 if wide else 122, (M, K // 16), dtype=torch.uint8, device="cuda", generator=g)
    n8 = (n + 7) // 8 * 8
    x = torch.randn((n, K), device="cuda", generator=g).half()
    gu, rows, spare = (torch.zeros(d, dtype=torch.float16, device="cuda") for d in ((M, n8), (M // 2, n8), (n, M)))
    got = torch.full((n * M // 2 + 64,), 7.0, dtype=torch.float16, device="cuda")
    lib.nvfp4_b200_gemm_config(1)
    assert lib.launch_nvfp4_gemm_w4a16_ex(ptr(p), ptr(s), ptr(x), K, ptr(gu), n8, M, n, K, 1, stream()) == 0
    assert lib.launch_silu_mul_rows(ptr(gu), ptr(rows), M // 2, n8, stream()) == 0
    lib.nvfp4_b200_gemm_config(3)
    assert lib.launch_nvfp4_gemm_silu(ptr(p), ptr(s), ptr(x), K, ptr(spare), ptr(got), M, n, K, stream()) == 0
    torch.cuda.synchronize()
    assert lib.nvfp4_gemm_status(0) == 0
    assert (got[-64:] == 7).all()
    a, b = got[:-64].view(n, M // 2), rows[:, :n].t()
    assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a[~a.isnan()], b[~b.isnan()])
    fused = (n, K) in ((190, 4096), (4400, 2560), (257, 5120), (4999, 5120))
    assert (spare == 0).all().item() == fused
