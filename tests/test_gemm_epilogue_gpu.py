"""Stores of the CTA-pair GEMM: blocks that leave by TMA and blocks that are stored row by row, in every output mode."""
import os
import subprocess
import sys

import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.gemm import OUT_BF16, OUT_BF16_ACC, OUT_F32, OUT_F32_ACC

pytestmark = pytest.mark.gpu
DEV = "cuda"


# whole tiles, ragged rows and columns (clipped boxes), a pitch that is no multiple of 16 bytes, more tiles than pairs
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 328, 72), (257, 1000, 136), (1000, 333, 64), (2600, 2568, 64)])
@pytest.mark.parametrize("mode", [OUT_BF16, OUT_F32, OUT_F32_ACC, OUT_BF16_ACC])
@pytest.mark.parametrize("shift", [0, 1])
def test_every_store_of_the_pair_kernel(M, N, K, mode, shift):
    g = torch.Generator(device=DEV).manual_seed(M + N + mode)
    a, b = (torch.randn(n, K, device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16)
    dt = torch.float32 if mode in (OUT_F32, OUT_F32_ACC) else torch.bfloat16
    whole = torch.full((M + 2, N + 3 + shift), 2.0, device=DEV, dtype=dt)       # C is a window of a wider matrix
    out = whole[1:M + 1, shift:N + shift]
    ops.gemm(a, b, out=out, out_mode=mode, bias=bias, pair=True)
    ref = a.double() @ b.double().t() + bias.double() + (2.0 if mode in (OUT_F32_ACC, OUT_BF16_ACC) else 0.0)
    err = ((out.double() - ref).norm() / ref.norm()).item()
    assert err < (1e-5 if dt == torch.float32 else 2.0 ** -8)                   # fp32 sums; one rounding
    out.fill_(2.0)
    assert (whole == 2.0).all()                                                 # nothing outside the window
    packed = ops.gemm(a, b, out_mode=mode, bias=bias, pair=True) if mode in (OUT_BF16, OUT_F32) else None
    if packed is not None:
        assert ((packed.double() - ref).norm() / ref.norm()).item() < (1e-5 if dt == torch.float32 else 2.0 ** -8)
    _lib.assert_healthy()


# C as a window that a tensor map covers (its pitch, width and first column whole 16-byte groups): columns that end in a
# box of 64, in a tile and on its edge, rows that end in a block of 32 and on its edge, more tiles than pairs
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 328, 72), (257, 1000, 136), (321, 8, 64), (2600, 2568, 64)])
@pytest.mark.parametrize("left,right", [(0, 8), (8, 8), (8, 64)])
@pytest.mark.parametrize("a_mn", [False, True])
def test_tma_stores_stay_inside_their_window(M, N, K, left, right, a_mn):
    if a_mn and M % 8:
        pytest.skip("rows of an M-major operand are whole 16-byte groups")
    g = torch.Generator(device=DEV).manual_seed(M + N + left)
    a, b = (torch.randn(n, K, device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16)
    whole = torch.full((M + 34, left + N + right), 2.0, device=DEV, dtype=torch.bfloat16)
    out = whole[1:M + 1, left:left + N]
    assert out.stride(0) % 8 == 0 and N % 8 == 0 and out.data_ptr() % 16 == 0     # what the tensor map asks for
    ops.gemm(a.t().contiguous() if a_mn else a, b, out=out, a_mn=a_mn, bias=bias, pair=True)
    ref = a.double() @ b.double().t() + bias.double()
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8, atol=1e-4 * K ** 0.5)  # one rounding; fp32 sums of K products
    out.fill_(2.0)
    assert (whole == 2.0).all()
    _lib.assert_healthy()


# fp32 results and accumulating modes in a window of whole 16-byte groups: one box of 32 columns and less, columns that end
# inside a box and on a tile's edge, whole and clipped blocks of 32 rows, a bias whose last columns are not 16 bytes wide
@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (300, 36, 72), (257, 1000, 136), (352, 260, 64), (2600, 2568, 64)])
@pytest.mark.parametrize("mode", [OUT_F32, OUT_F32_ACC, OUT_BF16_ACC])
@pytest.mark.parametrize("biased", [False, True])
def test_wide_stores_stay_inside_their_window(M, N, K, mode, biased):
    g = torch.Generator(device=DEV).manual_seed(M + N + mode)
    a, b = (torch.randn(n, K, device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16) if biased else None
    dt = torch.bfloat16 if mode == OUT_BF16_ACC else torch.float32
    whole = torch.full((M + 34, 4 + N + 8), 2.0, device=DEV, dtype=dt)
    out = whole[1:M + 1, 4:4 + N]
    assert out.stride(0) % 4 == 0 and N % 4 == 0 and out.data_ptr() % 8 == 0
    ops.gemm(a, b, out=out, out_mode=mode, bias=bias, pair=True)
    ref = a.double() @ b.double().t() + (bias.double() if biased else 0.0) + (0.0 if mode == OUT_F32 else 2.0)
    # fp32 sums of K products of unit normals; one rounding to 16 bits where C is 16 bits wide
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8 if dt == torch.bfloat16 else 1e-6, atol=1e-5 * K ** 0.5)
    out.fill_(2.0)
    assert (whole == 2.0).all()
    _lib.assert_healthy()


# tiles of the last wave shared along K by the default rule: one tile and no whole wave, a ragged few with every layout's
# k-blocks uneven over the slices, a last wave behind a whole one; in a window, with a bias, every result type
@pytest.mark.parametrize("M,N,K", [(256, 256, 4096), (300, 520, 8200), (2304, 2304, 4168)])
@pytest.mark.parametrize("mode", [OUT_BF16, OUT_F32, OUT_F32_ACC])
@pytest.mark.parametrize("a_mn,b_mn,biased", [(False, False, True), (False, True, False), (True, True, False)])
def test_shared_tiles_of_the_last_wave(M, N, K, mode, a_mn, b_mn, biased):
    assert _lib.load().hg_gemm2_scratch(M, N, K) > 0 and _lib.load().hg_gemm2_scratch(M, N, 512) == 0
    g = torch.Generator(device=DEV).manual_seed(M + K + mode)
    pad = lambda r, c: torch.randn(r, (c + 7) // 8 * 8, device=DEV, generator=g).to(torch.bfloat16)[:, :c]
    a, b = pad(K, M) if a_mn else pad(M, K), pad(K, N) if b_mn else pad(N, K)
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16) if biased else None
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double() + (bias.double() if biased else 0.0)
    whole = torch.full((M + 2, N + 8), 2.0, device=DEV, dtype=torch.bfloat16 if mode == OUT_BF16 else torch.float32)
    out = whole[1:M + 1, 4:4 + N]
    run = lambda: ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, out_mode=mode, bias=bias, pair=True)
    run()
    first = out.clone()
    want = ref + (2.0 if mode == OUT_F32_ACC else 0.0)
    # K / 16 additions in the tensor core, each off by at most a unit 2^-23 of a running sum of K products of unit normals, six
    # standard deviations sqrt(K) at most; one rounding to 16 bits where C is 16 bits wide
    assert torch.allclose(first.double(), want, rtol=2.0 ** -8 if mode == OUT_BF16 else 1e-6,
                          atol=K / 16 * 2.0 ** -23 * 6 * K ** 0.5)
    graph, other = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    out.fill_(2.0)
    with torch.cuda.graph(graph):
        run()
    for _ in range(3):                                # a replayed launch finds the flags cleared
        out.fill_(2.0)
        graph.replay()
        assert torch.equal(out, first)
    results = []
    for s in (torch.cuda.current_stream(), other):    # launches of two streams do not share their parts
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            for _ in range(4):
                results.append(ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_mode=OUT_F32 if mode == OUT_F32_ACC else mode,
                                        bias=bias, pair=True))
    torch.cuda.synchronize()
    assert all(torch.equal(r, results[0]) for r in results)
    whole[1:M + 1, 4:4 + N] = 2.0
    assert (whole == 2.0).all()
    _lib.assert_healthy()


# many slices a tile, every one of which may be the last: C is added to once, whoever does it, and the same bits each time
@pytest.mark.parametrize("M,N,K", [(256, 256, 66000), (300, 300, 20000)])
def test_shared_tiles_of_many_slices(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(K)
    a, b = (torch.randn(n, K, device=DEV, generator=g).to(torch.bfloat16) for n in (M, N))
    once = torch.zeros(M, N, device=DEV)
    ops.gemm(a, b, out=once, out_mode=OUT_F32_ACC, pair=True)
    ref = a.double() @ b.double().t()
    assert torch.allclose(once.double(), ref, rtol=1e-6, atol=K / 16 * 2.0 ** -23 * 6 * K ** 0.5)   # as above
    outs, streams = [torch.zeros(M, N, device=DEV) for _ in range(6)], [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        with torch.cuda.stream(streams[i % 3]):
            for _ in range(4):
                o.zero_()
                ops.gemm(a, b, out=o, out_mode=OUT_F32_ACC, pair=True)
    torch.cuda.synchronize()
    assert all(torch.equal(o, once) for o in outs)
    _lib.assert_healthy()


# products that the plan cuts into tiles of other widths: whole columns of 64 to 224, turned ones whose rows end inside a tile, a
# block and a pair of columns, alone and shared, and results that turned tiles cannot store (an odd pitch, an odd base)
@pytest.mark.parametrize("M,N,K", [(1024, 512, 512), (1531, 4608, 712), (333, 3072, 768), (128, 1600, 6400), (258, 1602, 6400),
                                   (580, 16642, 512), (1554, 9474, 1024), (200, 3584, 8192), (312, 1600, 1600), (1600, 1600, 2997)])
@pytest.mark.parametrize("a_mn,b_mn,biased", [(False, False, True), (False, True, False), (True, True, False)])
@pytest.mark.parametrize("mode,left", [(OUT_BF16, 0), (OUT_BF16, 2), (OUT_BF16, 1), (OUT_F32, 0), (OUT_F32_ACC, 4)])
def test_tiles_of_every_width(M, N, K, a_mn, b_mn, biased, mode, left):
    g = torch.Generator(device=DEV).manual_seed(M + K + mode)
    pad = lambda r, c: torch.randn(r, (c + 7) // 8 * 8, device=DEV, generator=g).to(torch.bfloat16)[:, :c]
    a, b = pad(K, M) if a_mn else pad(M, K), pad(K, N) if b_mn else pad(N, K)
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16) if biased else None
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double() + (bias.double() if biased else 0.0)
    whole = torch.full((M + 2, N + 8), 2.0, device=DEV, dtype=torch.bfloat16 if mode == OUT_BF16 else torch.float32)
    out = whole[1:M + 1, left:left + N]
    ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, out_mode=mode, bias=bias, pair=True)
    # K / 16 additions in the tensor core, each off by at most a unit 2^-23 of a running sum of K products of unit normals, six
    # standard deviations sqrt(K) at most; one rounding to 16 bits where C is 16 bits wide
    assert torch.allclose(out.double(), ref + (2.0 if mode == OUT_F32_ACC else 0.0), rtol=2.0 ** -8 if mode == OUT_BF16 else 1e-6,
                          atol=K / 16 * 2.0 ** -23 * 6 * K ** 0.5)
    out.fill_(2.0)
    assert (whole == 2.0).all()                                                 # nothing outside the window
    _lib.assert_healthy()


# 16-bit results of shared tiles with two epilogue warps per 32 rows, which only HG_GEMM_SPLIT_TAIL=1 leads to: the blocks in which a
# warp leaves its parts are those in which it adds them
@pytest.mark.parametrize("M,N,K", [(256, 256, 1024), (343, 448, 1064), (600, 328, 1088), (512, 512, 1536)])
def test_shared_16_bit_tiles_with_two_warps(M, N, K):
    code = """
import ctypes, torch
from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
M, N, K = %r
plan = (ctypes.c_int * 5)()
_lib.load().hg_gemm2_plan(M, N, K, 0, 1, 0, 74, plan)
assert plan[0] == 64 and not plan[1] and plan[2] > 1 and plan[4] == 2, list(plan)
g = torch.Generator(device="cuda").manual_seed(K)
a, b = (torch.randn(n, K, device="cuda", generator=g).to(torch.bfloat16) for n in (M, N))
ref = a.double() @ b.double().t()
outs = [ops.gemm(a, b, pair=True) for _ in range(200)]
assert torch.allclose(outs[0].double(), ref, rtol=2.0 ** -8, atol=K / 16 * 2.0 ** -23 * 6 * K ** 0.5)     # as above
assert all(torch.equal(o, outs[0]) for o in outs)
_lib.assert_healthy()
""" % ((M, N, K),)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, HG_GEMM_SPLIT_TAIL="1"), capture_output=True, text=True,
                         timeout=300, cwd=root)
    assert run.returncode == 0, run.stderr[-2000:]
