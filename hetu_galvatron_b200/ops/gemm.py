"""bf16 GEMM on the tcgen05 kernel (csrc/sm100/gemm.cu) and the autograd ``linear`` built on it.

The three products of a linear layer read the tensors exactly as PyTorch stores them:

* forward  ``y = x @ w.T``      : A = x [T,K] (K-major),  B = w [N,K] (K-major)
* dgrad    ``dx = dy @ w``      : A = dy [T,N] (K-major), B = w [N,K] read N-major
* wgrad    ``dw = dy.T @ x``    : A = dy [T,N] read M-major, B = x [T,K] read N-major

so no transpose pass ever runs.  With ``w.main_grad`` (an fp32 buffer owned by the sharded-parameter
manager) the weight gradient is accumulated there by the GEMM epilogue (``C += acc``), which is what
gradient accumulation over micro-batches and the ZeRO reduce-scatter consume.

Reference call sites replaced: galvatron/core/runtime/tensor_parallel/layers.py:300 (fwd), :342
(dgrad), :414 (wgrad).
"""
from __future__ import annotations

import os

import torch

from . import _lib

OUT_BF16, OUT_F32, OUT_F32_ACC, OUT_BF16_ACC = 0, 1, 2, 3


def _rowmajor(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        raise ValueError("expected a matrix")
    if t.stride(1) != 1 or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


# CTA-pair kernel (tcgen05.mma.cta_group::2, 256x256 tiles): "auto" uses it for problems of at least one pair tile,
# "0" never, "1" always.  The one-CTA kernel is the fallback when the device cannot co-schedule a pair.
_PAIR_MODE = os.environ.get("HG_GEMM_PAIR", "auto")
_pair_ok = True


# Rows up to which every product of a decoder layer runs on the weight-streaming kernel, whatever its width
# (csrc/sm100/decoder_step.cu launches such a layer in one call).
NATIVE_STEP_ROWS = 64


def _use_skinny(M: int, N: int, K: int, a_mn: bool, out_mode: int, max_ctas: int, pair) -> bool:
    """Whether the weight-streaming kernel (csrc/sm100/gemm_skinny.cu) takes the product.  Up to 64 rows it is as fast as
    the one-CTA kernel or faster, by the microsecond that the timing resolves (4 rows, cold: 4096 x 4096 16 us against 35
    for the one-CTA kernel, 4096 x 11008 29 against 78, 152064 x 3584 176 against 208; 64 rows: 512 x 512 8.8 against 9.2,
    16384 columns x 1024 15.8 against 15.8).  From 65 to 128 rows it pays for long contractions of up to 64 of its tiles
    (128 rows: 4096 columns, K = 1024 14.9 against 14.1, 1536 14.9 against 17.0, 4096 19.5 against 32.6; 8192 columns,
    K = 2048 23.6 against 21.9, 3072 24.8 against 28.5; 16384 columns x 4096 41.5 against 39.5)."""
    if a_mn or out_mode not in (OUT_BF16, OUT_F32) or pair is not None or max_ctas != 0 or _PAIR_MODE == "1":
        return False
    if M <= NATIVE_STEP_ROWS:
        return N <= 65535 * 128                          # its grid has one y index per 128 columns
    return M <= 128 and N <= 8192 and K >= (1536 if N <= 4096 else 3072)


def _use_pair(M: int, N: int, pair) -> bool:
    if pair is not None:
        return bool(pair)
    if not _pair_ok or _PAIR_MODE == "0":
        return False
    return _PAIR_MODE == "1" or (M >= 256 and N >= 256)


def _use_grouped_pair(rows: int, N: int, K: int, G: int) -> bool:
    """Whether grouped products that cannot be turned (below) take the CTA-pair tile.  Its 256 rows are mostly padding for groups of
    one 128-row segment, and the store of a 256 x 256 tile is hidden only under a long contraction, so it pays for groups of about 512 rows
    and K from 2560 on.  Ragged groups, us, pair against one CTA: 8 x (128 rows, 28672 columns, K = 4096) 347 / 312, 512 rows
    822 / 796, 1024 rows 1351 / 1554; 64 x (512, 2048, 1408) 220 / 177, 1024 rows 384 / 312; 64 x (1024, 2816, 2048) 615 / 605;
    8 x (512, 4096, 2560) 87 / 89, 32 x (512, 4096, 3072) 323 / 333, 1024 rows 577 / 613.  (Weight gradients contract
    over the rows and gain at every size: 64 x (128, 2816, 2048) 1206 / 1634.)"""
    return _use_pair(rows, N, None) and (_PAIR_MODE == "1" or (rows >= 512 * G and K >= 2560))


def _use_grouped_turned(out: torch.Tensor, N: int, K: int) -> bool:
    """Whether grouped products take the CTA-pair kernel with tiles that are cut along a group's rows (a multiple of 64 of them;
    ``TurnedSegments`` in csrc/sm100/gemm2.cu), which it does wherever it is called and the results can be stored that way.  Ragged
    groups, us, one CTA / turned pair: 8 x (1024 rows, 28672 columns, K = 4096) 1667 / 1589, 512 rows 974 / 920, 128 rows 430 / 374,
    64 rows 350 / 340, 32 rows 344 / 325; 8 x (128, 4096, 14336) 235 / 189, 64 rows 170 / 172; 64 x (128, 2816, 2048) 185 / 176; 64 x
    (512, 2048, 1408) 230 / 221; 8 x (300, 4096, 1024) 31.1 / 30.8; 16384 rows of one group, 28672 columns, K = 4096 3927 / 2855, as the
    pair kernel without turning."""
    return (_use_pair(256, N, None) and K >= 1280 and N % 2 == 0 and out.stride(0) % 2 == 0 and out.data_ptr() % 4 == 0)


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False, out: torch.Tensor | None = None,
         out_mode: int = OUT_BF16, bias: torch.Tensor | None = None, max_ctas: int = 0, pair=None) -> torch.Tensor:
    """``C[M,N] = op(A) op(B)`` with fp32 accumulation.

    ``a`` is ``[M,K]`` (or ``[K,M]`` when ``a_mn``), ``b`` is ``[N,K]`` (or ``[K,N]`` when ``b_mn``).
    ``pair``: force (True) / forbid (False) the CTA-pair kernel; ``None`` follows ``HG_GEMM_PAIR``.
    """
    if not a.is_cuda:
        A = a.t() if a_mn else a
        Bm = b if b_mn else b.t()
        acc = A.float() @ Bm.float()
        if bias is not None:
            acc = acc + bias.float()
        if out is None:
            return acc.to(torch.float32 if out_mode in (OUT_F32, OUT_F32_ACC) else a.dtype)
        if out_mode in (OUT_F32_ACC, OUT_BF16_ACC):
            out.add_(acc.to(out.dtype))
        else:
            out.copy_(acc.to(out.dtype))
        return out
    lp = _lib.lp_dtype()
    if a.dtype != lp or b.dtype != lp:
        raise TypeError("the tcgen05 GEMM of this build takes %s operands, got %s and %s" % (lp, a.dtype, b.dtype))
    a, b = _rowmajor(a), _rowmajor(b)
    if a_mn:
        K, M = a.shape
    else:
        M, K = a.shape
    if b_mn:
        Kb, N = b.shape
    else:
        N, Kb = b.shape
    if K != Kb:
        raise ValueError("contraction mismatch: %s vs %s" % (tuple(a.shape), tuple(b.shape)))
    if out is None:
        dt = torch.float32 if out_mode in (OUT_F32, OUT_F32_ACC) else lp
        if out_mode in (OUT_F32_ACC, OUT_BF16_ACC):
            raise ValueError("accumulating output modes need `out`")
        out = torch.empty((M, N), dtype=dt, device=a.device)
    else:
        if out.shape[0] != M or out.shape[1] != N or out.stride(1) != 1:
            raise ValueError("bad output tensor")
    lib = _lib.load()
    if _use_skinny(M, N, K, a_mn, out_mode, max_ctas, pair):
        rc = lib.hg_gemm_skinny_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.ptr(bias), M, N, K, a.stride(0),
                                     b.stride(0), out.stride(0), int(b_mn), out_mode, 0, _lib.stream())
        if rc != 0:
            raise _lib.KernelError("hg_gemm_skinny_bf16 failed with code %d (M=%d N=%d K=%d b_mn=%d)" % (rc, M, N, K, b_mn))
        _lib.count_launch()
        return out
    if _use_pair(M, N, pair):
        need = lib.hg_gemm2_scratch(M, N, K) if max_ctas == 0 else 0   # parts of tiles that several CTA pairs share
        ws = torch.empty(need, dtype=torch.uint8, device=a.device) if need else None
        rc = lib.hg_gemm2_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.ptr(bias), M, N, K, a.stride(0),
                                  b.stride(0), out.stride(0), int(a_mn), int(b_mn), out_mode, max_ctas, _lib.ptr(ws), need,
                                  _lib.stream())
        if rc == 0:
            _lib.count_launch()
            return out
        if rc != -2 or pair:
            raise _lib.KernelError("hg_gemm2_bf16 failed with code %d (M=%d N=%d K=%d a_mn=%d b_mn=%d)" % (rc, M, N, K, a_mn, b_mn))
        global _pair_ok
        _pair_ok = False  # this device cannot co-schedule the pair: one-CTA kernel from now on
    rc = lib.hg_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.ptr(bias), M, N, K, a.stride(0),
                          b.stride(0), out.stride(0), int(a_mn), int(b_mn), out_mode, max_ctas, _lib.stream())
    if rc != 0:
        raise _lib.KernelError(
            "hg_gemm_bf16 failed with code %d (M=%d N=%d K=%d a_mn=%d b_mn=%d a=%s/%s b=%s/%s out=%s/%s mode=%d)" %
            (rc, M, N, K, a_mn, b_mn, tuple(a.shape), a.stride(), tuple(b.shape), b.stride(), tuple(out.shape),
             out.stride(), out_mode))
    _lib.count_launch()
    return out


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias):
        ctx.save_for_backward(x, w)
        ctx.has_bias = bias is not None
        return gemm(x, w, bias=bias)

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dy = _rowmajor(dy)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy, w, b_mn=True)
        if ctx.needs_input_grad[1]:
            mg = getattr(w, "main_grad", None)
            if mg is not None:
                fresh = getattr(w, "mg_fresh", False)
                gemm(dy, x, a_mn=True, b_mn=True, out=mg, out_mode=OUT_F32 if fresh else OUT_F32_ACC)
                w.mg_fresh = False
                dw = None
            else:
                dw = gemm(dy, x, a_mn=True, b_mn=True)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = column_sums(dy)
        return dx, dw, db


def column_sums(x: torch.Tensor) -> torch.Tensor:
    """``x.float().sum(0)`` of a matrix, rounded back to its dtype: the gradient of a bias."""
    rows, cols = x.shape
    if torch.is_grad_enabled() and x.requires_grad:      # a graph of the gradient is wanted
        return x.float().sum(0).to(x.dtype)
    if x.is_cuda and x.dtype == _lib.lp_dtype():
        x = _rowmajor(x)
    if rows == 0 or cols == 0 or not x.is_cuda or x.dtype != _lib.lp_dtype() or x.stride(0) % 8 or x.data_ptr() % 16:
        return x.float().sum(0).to(x.dtype)
    lib = _lib.load()
    out = torch.empty(cols, dtype=x.dtype, device=x.device)
    parts = lib.hg_colsum_parts(rows, cols)
    partial = torch.empty((parts, cols), dtype=torch.float32, device=x.device) if parts > 1 else None
    _lib.check(lib.hg_colsum_bf16(x.data_ptr(), x.stride(0), rows, cols, _lib.ptr(partial), parts, out.data_ptr(),
                                  _lib.stream()), "hg_colsum_bf16")
    _lib.count_launch(2 if parts > 1 else 1)
    return out


def linear(x: torch.Tensor, w: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor:
    """``x @ w.T (+ bias)`` over the last dimension; leading dimensions are flattened."""
    if not x.is_cuda:
        return torch.nn.functional.linear(x, w, bias)
    native = _lib.native()
    if native is not None:
        y = native.linear(x, w, bias)
        if y is not None:
            return y
    shp = x.shape
    y = _Linear.apply(x.reshape(-1, shp[-1]), w, bias)
    return y if len(shp) == 2 else y.view(*shp[:-1], w.shape[0])


def grouped_gemm(a: torch.Tensor, b: torch.Tensor, row_start: torch.Tensor, *, b_mn: bool = False,
                 out: torch.Tensor | None = None) -> torch.Tensor:
    """Per-group product for the MoE experts.

    ``a``: ``[rows, K]``; ``row_start``: int32 ``[G+1]`` on the device (segment boundaries, ascending);
    ``b``: ``[G, N, K]`` (or ``[G, K, N]`` when ``b_mn``).  Rows outside every segment are left untouched.
    """
    G = b.shape[0]
    if b_mn:
        K, N = b.shape[1], b.shape[2]
    else:
        N, K = b.shape[1], b.shape[2]
    fresh = out is None
    if fresh:
        # on the GPU the product covers every row of a segment: only the rows outside them are cleared (below)
        out = (torch.empty if a.is_cuda and N % 8 == 0 else torch.zeros)((a.shape[0], N), dtype=a.dtype, device=a.device)
    if not a.is_cuda:
        rs = row_start.tolist()
        for g in range(G):
            Bm = b[g] if b_mn else b[g].t()
            out[rs[g]:rs[g + 1]] = (a[rs[g]:rs[g + 1]].float() @ Bm.float()).to(out.dtype)
        return out
    if b_mn and K % 64 != 0:
        raise ValueError("grouped GEMM with an N-major B needs K % 64 == 0")
    a = _rowmajor(a)
    b2 = b.reshape(G * b.shape[1], b.shape[2])
    lib = _lib.load()
    args = (a.data_ptr(), b2.data_ptr(), out.data_ptr(), row_start.data_ptr(), G, a.shape[0], N, K, a.stride(0),
            b2.stride(0), out.stride(0), int(b_mn), OUT_BF16, _lib.stream())
    pair = _use_grouped_turned(out, N, K) or _use_grouped_pair(a.shape[0], N, K, G)
    rc = lib.hg_grouped_gemm2_bf16(*args) if pair else -2
    if rc == -2:
        rc = lib.hg_grouped_gemm_bf16(*args)
    _lib.check(rc, "hg_grouped_gemm_bf16")
    _lib.count_launch()
    if fresh and N % 8 == 0:
        _lib.check(lib.hg_zero_outside(out.data_ptr(), row_start.data_ptr(), G, out.shape[0], N, _lib.stream()),
                   "hg_zero_outside")
        _lib.count_launch()
    return out


def grouped_wgrad(dy: torch.Tensor, x: torch.Tensor, row_start: torch.Tensor, out: torch.Tensor,
                  accumulate: bool = True) -> torch.Tensor:
    """``out[g] (+)= dy[seg_g].T @ x[seg_g]``;  ``out``: fp32 ``[G, N, K]``.  Segment boundaries must be
    multiples of 64 rows (the permutation pads every expert's segment and zero-fills the padding)."""
    G = out.shape[0]
    if not dy.is_cuda:
        rs = row_start.tolist()
        for g in range(G):
            acc = dy[rs[g]:rs[g + 1]].float().t() @ x[rs[g]:rs[g + 1]].float()
            if accumulate:
                out[g] += acc.to(out.dtype)
            else:
                out[g] = acc.to(out.dtype)
        return out
    dy, x = _rowmajor(dy), _rowmajor(x)
    lib = _lib.load()
    args = (dy.data_ptr(), x.data_ptr(), out.data_ptr(), row_start.data_ptr(), G, dy.shape[0], out.shape[1],
            out.shape[2], dy.stride(0), x.stride(0), OUT_F32_ACC if accumulate else OUT_F32, 0, _lib.stream())
    rc = lib.hg_grouped_wgrad2_bf16(*args) if _use_pair(out.shape[1], out.shape[2], None) else -2
    if rc == -2:
        rc = lib.hg_grouped_wgrad_bf16(*args)
    _lib.check(rc, "hg_grouped_wgrad_bf16")
    _lib.count_launch()
    return out


