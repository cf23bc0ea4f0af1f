"""The weight-streaming GEMM for few rows (csrc/sm100/gemm_skinny.cu) at the edges of its tiles and splits."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.gemm import OUT_F32

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel_err(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


# token counts on both sides of every tile width; widths of one column, a ragged tile and many tiles; contractions of
# less than one block, a ragged last block and enough blocks for a split over eight CTAs
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (4096, 4096), (1000, 2056), (40000, 264)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_skinny_gemm(M, N, K, b_mn):
    g = torch.Generator(device=DEV).manual_seed(M * 131 + N + K)
    x = torch.randn(M, K, device=DEV, generator=g).to(torch.bfloat16)
    w = torch.randn((K, N) if b_mn else (N, K), device=DEV, generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV, generator=g).to(torch.bfloat16)
    ref = x.double() @ (w.double() if b_mn else w.double().t()) + bias.double()
    # products of two bf16 are exact in fp32: what is left are fp32 sums (some K * 2^-24 at worst, far less at random)
    assert rel_err(ops.gemm(x, w, b_mn=b_mn, bias=bias, out_mode=OUT_F32), ref) < 1e-5
    # one rounding to bf16: at most 2^-8 of each value
    out = ops.gemm(x, w, b_mn=b_mn, bias=bias)
    assert out.dtype == torch.bfloat16 and rel_err(out, ref) < 2.0 ** -8
    assert torch.equal(out, ops.gemm(x, w, b_mn=b_mn, bias=bias))      # fixed order of the partial sums
    _lib.assert_healthy()


# contractions on both sides of the lengths from which eight CTAs (12 blocks of 64), four (24) and two (64) share a tile
@pytest.mark.parametrize("N,K", [(512, 704), (512, 768), (520, 776), (8192, 1472), (8192, 1536), (12288, 4032), (12288, 4096)])
@pytest.mark.parametrize("M", [4, 64, 128])
def test_skinny_gemm_around_its_split_lengths(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K, device=DEV, generator=g).to(torch.bfloat16)
    w = torch.randn(N, K, device=DEV, generator=g).to(torch.bfloat16)
    ref = x.double() @ w.double().t()
    for s in (0, 1):                                                  # the rule's split, and none
        out = torch.empty(M, N, device=DEV)
        _lib.check(_lib.load().hg_gemm_skinny_bf16(x.data_ptr(), w.data_ptr(), out.data_ptr(), 0, M, N, K, K, K, N, 0, OUT_F32, s,
                                                   _lib.stream()), "hg_gemm_skinny_bf16")
        assert rel_err(out, ref) < 1e-5
    _lib.assert_healthy()


def test_skinny_gemm_writes_only_its_rows_of_a_wider_output():
    M, N, K = 5, 200, 512
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(N, K, device=DEV).to(torch.bfloat16)
    whole = torch.full((M + 2, N + 7), 3.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm(x, w, out=whole[1:M + 1, 3:N + 3])
    ref = x.double() @ w.double().t()
    assert rel_err(whole[1:M + 1, 3:N + 3], ref) < 2.0 ** -8
    whole[1:M + 1, 3:N + 3] = 3.0
    assert (whole == 3.0).all()
    _lib.assert_healthy()
