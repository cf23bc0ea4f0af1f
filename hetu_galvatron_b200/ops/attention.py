"""Flash attention (tcgen05 kernels of csrc/sm100/attention.cu) with autograd.

Two entry points:

* :func:`flash_attention_packed` -- reads Q, K, V straight out of the fused QKV projection
  ``[S*B, (nh + 2*ng) * hd]`` whose columns are grouped per kv head as ``[ng, (nh/ng + 2), hd]``
  (the layout of the reference's ``linear_qkv``, galvatron/core/runtime/transformer/attention.py:876-926)
  and writes the context as ``[S*B, nh*hd]`` ready for the output projection.  No split / transpose
  copies exist in either direction: the backward writes dQ, dK, dV into one packed gradient buffer.
* :func:`flash_attention` -- separate ``[S, B, heads, hd]`` tensors with optional global position
  offsets and LSE output; the building block of the Ulysses and ring (context-parallel) paths.

Oracle: fp32 ``softmax(Q K^T / sqrt(hd) + causal mask) V``.
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import _lib
from ._lib import AttnTensor


def _desc(t: torch.Tensor, ss: int, sb: int, slots: int, gs: int, hs: int, off: int) -> AttnTensor:
    return AttnTensor(t.data_ptr(), ss, sb, slots, gs, hs, off)


def attention_reference(q, k, v, causal=True, scale=None, q_pos0=0, k_pos0=0, dropout_p: float = 0.0):
    """q: [S,B,nh,hd], k/v: [Skv,B,ng,hd] -> (out [S,B,nh,hd], lse [B,nh,S]); fp32 math.  ``dropout_p`` drops
    attention probabilities (after the softmax, rescaled by 1 / (1 - p)) from the current random stream."""
    S, B, nh, hd = q.shape
    Skv, ng = k.shape[0], k.shape[2]
    scale = scale if scale is not None else 1.0 / math.sqrt(hd)
    qf = q.float().permute(1, 2, 0, 3)
    kf = k.float().permute(1, 2, 0, 3).repeat_interleave(nh // ng, dim=1)
    vf = v.float().permute(1, 2, 0, 3).repeat_interleave(nh // ng, dim=1)
    s = torch.einsum("bhqd,bhkd->bhqk", qf, kf) * scale
    if causal:
        qp = torch.arange(S, device=q.device) + q_pos0
        kp = torch.arange(Skv, device=q.device) + k_pos0
        s = s.masked_fill(kp[None, :] > qp[:, None], float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    p = torch.exp(s - lse[..., None])
    p = torch.nan_to_num(p, nan=0.0)
    if dropout_p > 0.0:
        p = torch.nn.functional.dropout(p, dropout_p, True)
    o = torch.einsum("bhqk,bhkd->bhqd", p, vf)
    return o.permute(2, 0, 1, 3).to(q.dtype), lse


def _backward_scratch(lib, S, Skv, B, nh, ng, hd, causal, q_pos0, k_pos0, device):
    """fp32 scratch of the backward kernels: row sums of dO * O and, where key blocks are shared between CTAs, their parts; and the
    pieces that hold dS where storing it pays, none if there is no room for them: dQ then takes longer."""
    wants = (ctypes.c_longlong * 3)()
    lib.hg_flash_bwd_wants(S, Skv, B, nh, ng, hd, int(causal), q_pos0, k_pos0, wants)
    ws = torch.empty(wants[0], dtype=torch.float32, device=device)
    if wants[1] and lib.hg_flash_bwd_has_room(device.index):
        try:
            return ws, [torch.empty(wants[2], dtype=torch.float32, device=device) for _ in range(wants[1])]
        except torch.cuda.OutOfMemoryError:
            lib.hg_flash_bwd_no_room(device.index)
    return ws, []


def _tiles_args(tiles):
    """The pieces as the kernels' entry point takes them."""
    return (ctypes.c_void_p * len(tiles))(*[t.data_ptr() for t in tiles]), len(tiles), tiles[0].numel() if tiles else 0


class _FlashPacked(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, S, B, nh, ng, hd, causal, scale):
        lib = _lib.load()
        T, P = qkv.shape
        qpg = nh // ng
        slots = nh + 2 * ng
        out = torch.empty((T, nh * hd), dtype=qkv.dtype, device=qkv.device)
        lse = torch.empty((B, nh, S), dtype=torch.float32, device=qkv.device)
        ss, sb = B * P, P
        q = _desc(qkv, ss, sb, slots, qpg + 2, 1, 0)
        k = _desc(qkv, ss, sb, slots, qpg + 2, 0, qpg)
        v = _desc(qkv, ss, sb, slots, qpg + 2, 0, qpg + 1)
        o = _desc(out, B * nh * hd, nh * hd, nh, qpg, 1, 0)
        rc = lib.hg_flash_fwd(ctypes.byref(q), ctypes.byref(k), ctypes.byref(v), ctypes.byref(o), lse.data_ptr(), S, S,
                              B, nh, ng, hd, int(causal), 0, 0, float(scale), _lib.stream())
        _lib.check(rc, "hg_flash_fwd")
        _lib.count_launch()
        ctx.save_for_backward(qkv, out, lse)
        ctx.cfg = (S, B, nh, ng, hd, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv, out, lse = ctx.saved_tensors
        S, B, nh, ng, hd, causal, scale = ctx.cfg
        lib = _lib.load()
        T, P = qkv.shape
        qpg = nh // ng
        slots = nh + 2 * ng
        dout = dout.contiguous()
        dqkv = torch.empty_like(qkv)
        ws, tiles = _backward_scratch(lib, S, S, B, nh, ng, hd, causal, 0, 0, qkv.device)
        ss, sb = B * P, P
        q = _desc(qkv, ss, sb, slots, qpg + 2, 1, 0)
        k = _desc(qkv, ss, sb, slots, qpg + 2, 0, qpg)
        v = _desc(qkv, ss, sb, slots, qpg + 2, 0, qpg + 1)
        o = _desc(out, B * nh * hd, nh * hd, nh, qpg, 1, 0)
        do = _desc(dout, B * nh * hd, nh * hd, nh, qpg, 1, 0)
        dq = _desc(dqkv, ss, sb, slots, qpg + 2, 1, 0)
        dk = _desc(dqkv, ss, sb, slots, qpg + 2, 0, qpg)
        dv = _desc(dqkv, ss, sb, slots, qpg + 2, 0, qpg + 1)
        kernels = ctypes.c_int()
        rc = lib.hg_flash_bwd_ws(ctypes.byref(q), ctypes.byref(k), ctypes.byref(v), ctypes.byref(o), ctypes.byref(do),
                                 lse.data_ptr(), ws.data_ptr(), ws.numel(), *_tiles_args(tiles), ctypes.byref(dq), ctypes.byref(dk),
                                 ctypes.byref(dv), S, S, B, nh, ng, hd, int(causal), 0, 0, float(scale),
                                 ctypes.byref(kernels), _lib.stream())
        _lib.check(rc, "hg_flash_bwd")
        _lib.count_launch(kernels.value)
        return dqkv, None, None, None, None, None, None, None


def split_packed(qkv, nh, ng, hd):
    """Views of q [T,nh,hd], k [T,ng,hd], v [T,ng,hd] inside the packed projection (reference layout)."""
    T = qkv.shape[0]
    qpg = nh // ng
    g = qkv.view(T, ng, qpg + 2, hd)
    return g[:, :, :qpg].reshape(T, nh, hd), g[:, :, qpg], g[:, :, qpg + 1]


def flash_attention_packed(qkv: torch.Tensor, S: int, B: int, nh: int, ng: int, hd: int, causal: bool = True,
                           scale: float | None = None) -> torch.Tensor:
    scale = scale if scale is not None else 1.0 / math.sqrt(hd)
    if not qkv.is_cuda:
        q, k, v = split_packed(qkv, nh, ng, hd)
        o, _ = attention_reference(q.reshape(S, B, nh, hd), k.reshape(S, B, ng, hd), v.reshape(S, B, ng, hd), causal,
                                   scale)
        return o.reshape(S * B, nh * hd)
    if hd not in (64, 128):
        raise ValueError("the sm_100a flash attention kernels support head_dim 64 and 128")
    native = _lib.native()
    if native is not None:
        out = native.flash_packed(qkv, S, B, nh, ng, hd, causal, scale)
        if out is not None:
            return out
    return _FlashPacked.apply(qkv.contiguous(), S, B, nh, ng, hd, causal, scale)


def _forward_launch(q, k, v, o, lse, S, Skv, B, nh, ng, hd, causal, q_pos0, k_pos0, scale, spread=None):
    """Forward on tensor descriptors: the kernels that split the keys over the chip when a kv head has at most eight
    query rows and that pays (csrc/sm100/flash_decode.cu; ``spread`` forces or forbids it), the tile kernels otherwise."""
    lib = _lib.load()
    args = (S, Skv, B, nh, ng, hd, int(causal), q_pos0, k_pos0)
    refs = [ctypes.byref(t) for t in (q, k, v)]
    if spread is None:
        spread = S * (nh // ng) <= 8 and lib.hg_flash_decode_pays(*args)
    need = lib.hg_flash_decode_scratch(*refs, *args) if spread else -1
    if need >= 0:
        ws = torch.empty(need, dtype=torch.float32, device=lse.device) if need else None
        rc = lib.hg_flash_decode(*refs, ctypes.byref(o), lse.data_ptr(), _lib.ptr(ws), *args, float(scale), _lib.stream())
        _lib.check(rc, "hg_flash_decode")
        _lib.count_launch(2 if need else 1)
        return
    rc = lib.hg_flash_fwd(*refs, ctypes.byref(o), lse.data_ptr(), *args, float(scale), _lib.stream())
    _lib.check(rc, "hg_flash_fwd")
    _lib.count_launch()


def _nested(dims, width: int) -> bool:
    """Whether rows of ``width`` packed elements under outer dimensions of ``(stride, size)`` are all apart: each stride
    spans everything inside it."""
    reach = width
    for stride, n in sorted(d for d in dims if d[1] > 1):
        if stride < reach:
            return False
        reach += stride * (n - 1)
    return True


def _disjoint(a: torch.Tensor, b: torch.Tensor, width: int) -> bool:
    """Whether two caches ``[seq, batch, heads, hd]`` of ``width`` packed elements per token share no memory: separate ranges,
    or equal strides and an offset that keeps every token apart from the other cache's (two halves of one buffer)."""
    lo, hi = (a, b) if a.data_ptr() <= b.data_ptr() else (b, a)
    apart = (hi.data_ptr() - lo.data_ptr()) // lo.element_size()
    if lo.stride(0) * (lo.shape[0] - 1) + lo.stride(1) * (lo.shape[1] - 1) + width <= apart:
        return True
    dims = [i for i in (0, 1) if max(lo.shape[i], hi.shape[i]) > 1]
    if any(lo.stride(i) != hi.stride(i) for i in dims):
        return False
    if not _nested([(lo.stride(i), max(lo.shape[i], hi.shape[i])) for i in dims], width):
        return False
    dims.sort(key=lo.stride, reverse=True)

    def meet(off, at):                # whether tokens of the two can lie closer than a token's width
        if at == len(dims):
            return abs(off) < width
        st, d = lo.stride(dims[at]), -off // lo.stride(dims[at])       # steps that bring them nearest from either side
        return any(1 - lo.shape[dims[at]] <= n < hi.shape[dims[at]] and meet(off + n * st, at + 1) for n in (d, d + 1))

    return not meet(apart, 0)


def caches_usable(like: torch.Tensor, kc: torch.Tensor, vc: torch.Tensor, past: int, S: int, b0: int, B: int, ng: int,
                  hd: int) -> bool:
    """Whether the kernels can write ``S`` tokens of ``B`` sequences behind ``past`` cached ones to these caches
    ``[max_seq, max_batch, ng, hd]`` and read them: ``like``'s dtype and device, room for the tokens, contiguous heads,
    whole 16-byte groups, elements that do not share memory, no gradient recorded through them, and an in-place write that
    autograd would allow (:func:`caches_written` tells it of the kernels')."""
    return ((torch.is_inference_mode_enabled() or not (kc.is_inference() or vc.is_inference())) and past >= 0 and b0 >= 0 and kc.dtype == vc.dtype == like.dtype and kc.device == vc.device == like.device
            and not (kc.requires_grad or vc.requires_grad)
            and all(c.dim() == 4 and c.shape[0] >= past + S and c.shape[1] >= b0 + B and c.shape[2:] == (ng, hd)
                    and c.stride(3) == 1 and c.stride(2) == hd and min(c.stride(0), c.stride(1)) >= ng * hd
                    and c.stride(0) % 8 == c.stride(1) % 8 == 0 and c.data_ptr() % 16 == 0
                    and _nested(((c.stride(0), c.shape[0]), (c.stride(1), c.shape[1])), ng * hd) for c in (kc, vc))
            and _disjoint(kc, vc, ng * hd))


def caches_written(kc: torch.Tensor, vc: torch.Tensor):
    """Tell autograd that the kernels have written to the caches, as an in-place operation would: a graph that has saved
    them must not go backward over other values."""
    torch.autograd.graph.increment_version((kc, vc))


def cached_attention_usable(qkv, kc, vc, past: int, S: int, b0: int, B: int, ng: int, hd: int) -> bool:
    """Whether :func:`cached_attention` takes these tensors: no gradient wanted, a 16-bit packed projection on a GPU and
    usable caches."""
    return (qkv.is_cuda and not (torch.is_grad_enabled() and qkv.requires_grad) and hd in (64, 128)
            and qkv.dtype == _lib.lp_dtype() and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0
            and caches_usable(qkv, kc, vc, past, S, b0, B, ng, hd))


def cached_attention(qkv: torch.Tensor, kc: torch.Tensor, vc: torch.Tensor, past: int, b0: int, S: int, B: int, nh: int,
                     ng: int, hd: int, cos: torch.Tensor | None = None, sin: torch.Tensor | None = None,
                     interleaved: bool = False) -> torch.Tensor:
    """One cached forward of ``S`` new tokens (no gradient): rotates the queries of the packed ``qkv [S*B, P]`` in place,
    writes the rotated keys and the values behind the ``past`` cached ones (``kc`` / ``vc`` ``[max_seq, max_batch, ng,
    hd]``, sequences ``b0 ..``) and attends causally to everything cached.  Returns ``[S, B, nh*hd]``."""
    lib = _lib.load()
    qpg, P = nh // ng, qkv.shape[1]
    kn, vn = kc[past:, b0:], vc[past:, b0:]
    rc = lib.hg_rope_append(qkv.data_ptr(), S * B, B, ng, qpg, hd, past, _lib.ptr(cos), _lib.ptr(sin),
                            2 * cos.shape[1] if cos is not None else 0, int(interleaved), kn.data_ptr(), vn.data_ptr(),
                            kc.stride(0), kc.stride(1), vc.stride(0), vc.stride(1), _lib.stream())
    _lib.check(rc, "hg_rope_append")
    _lib.count_launch()
    caches_written(kc, vc)
    out = torch.empty((S, B, nh * hd), dtype=qkv.dtype, device=qkv.device)
    lse = torch.empty((B, nh, S), dtype=torch.float32, device=qkv.device)
    k, v = kc[:, b0:], vc[:, b0:]
    _forward_launch(_desc(qkv, B * P, P, nh + 2 * ng, qpg + 2, 1, 0), _desc(k, k.stride(0), k.stride(1), ng, 1, 0, 0),
                    _desc(v, v.stride(0), v.stride(1), ng, 1, 0, 0), _desc(out, B * nh * hd, nh * hd, nh, qpg, 1, 0), lse,
                    S, past + S, B, nh, ng, hd, True, past, 0, 1.0 / math.sqrt(hd))
    return out


class _Flash(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale, q_pos0, k_pos0):
        S, B, nh, hd = q.shape
        Skv, ng = k.shape[0], k.shape[2]
        qpg = nh // ng
        out = torch.empty_like(q)
        lse = torch.empty((B, nh, S), dtype=torch.float32, device=q.device)
        qd = _desc(q, q.stride(0), q.stride(1), nh, qpg, 1, 0)
        kd = _desc(k, k.stride(0), k.stride(1), ng, 1, 0, 0)
        vd = _desc(v, v.stride(0), v.stride(1), ng, 1, 0, 0)
        od = _desc(out, out.stride(0), out.stride(1), nh, qpg, 1, 0)
        _forward_launch(qd, kd, vd, od, lse, S, Skv, B, nh, ng, hd, causal, q_pos0, k_pos0, scale)
        ctx.save_for_backward(q, k, v, out, lse)
        ctx.cfg = (causal, scale, q_pos0, k_pos0)
        ctx.mark_non_differentiable(lse)
        return out, lse

    @staticmethod
    def backward(ctx, dout, _dlse):
        q, k, v, out, lse = ctx.saved_tensors
        causal, scale, q_pos0, k_pos0 = ctx.cfg
        dq, dk, dv = flash_backward(q, k, v, out, dout.contiguous(), lse, causal, scale, q_pos0, k_pos0)
        return dq, dk, dv, None, None, None, None


def flash_backward(q, k, v, out, dout, lse, causal, scale, q_pos0=0, k_pos0=0):
    """Raw backward with an externally supplied (possibly global) LSE -- used by ring attention."""
    lib = _lib.load()
    S, B, nh, hd = q.shape
    Skv, ng = k.shape[0], k.shape[2]
    qpg = nh // ng
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    ws, tiles = _backward_scratch(lib, S, Skv, B, nh, ng, hd, causal, q_pos0, k_pos0, q.device)
    qd = _desc(q, q.stride(0), q.stride(1), nh, qpg, 1, 0)
    kd = _desc(k, k.stride(0), k.stride(1), ng, 1, 0, 0)
    vd = _desc(v, v.stride(0), v.stride(1), ng, 1, 0, 0)
    od = _desc(out, out.stride(0), out.stride(1), nh, qpg, 1, 0)
    dod = _desc(dout, dout.stride(0), dout.stride(1), nh, qpg, 1, 0)
    dqd = _desc(dq, dq.stride(0), dq.stride(1), nh, qpg, 1, 0)
    dkd = _desc(dk, dk.stride(0), dk.stride(1), ng, 1, 0, 0)
    dvd = _desc(dv, dv.stride(0), dv.stride(1), ng, 1, 0, 0)
    kernels = ctypes.c_int()
    rc = lib.hg_flash_bwd_ws(ctypes.byref(qd), ctypes.byref(kd), ctypes.byref(vd), ctypes.byref(od), ctypes.byref(dod),
                             lse.data_ptr(), ws.data_ptr(), ws.numel(), *_tiles_args(tiles), ctypes.byref(dqd), ctypes.byref(dkd),
                             ctypes.byref(dvd), S, Skv, B, nh, ng, hd, int(causal), q_pos0, k_pos0, float(scale),
                             ctypes.byref(kernels), _lib.stream())
    _lib.check(rc, "hg_flash_bwd")
    _lib.count_launch(kernels.value)
    return dq, dk, dv


def flash_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal: bool = True,
                    scale: float | None = None, q_pos0: int = 0, k_pos0: int = 0, return_lse: bool = False):
    """q ``[S,B,nh,hd]``, k/v ``[Skv,B,ng,hd]`` -> out ``[S,B,nh,hd]`` (and LSE ``[B,nh,S]``)."""
    hd = q.shape[-1]
    scale = scale if scale is not None else 1.0 / math.sqrt(hd)
    if not q.is_cuda:
        o, lse = attention_reference(q, k, v, causal, scale, q_pos0, k_pos0)
        return (o, lse) if return_lse else o

    def fix(t):
        return t if (t.stride(-1) == 1 and t.stride(-2) == hd) else t.contiguous()

    out, lse = _Flash.apply(fix(q), fix(k), fix(v), causal, scale, q_pos0, k_pos0)
    return (out, lse) if return_lse else out


def attention_merge(out_acc: torch.Tensor, lse_acc: torch.Tensor, out_new: torch.Tensor, lse_new: torch.Tensor):
    """In-place log-sum-exp merge of a partial attention result over a disjoint key set (CUDA):
    ``out_acc`` fp32 ``[S, B, h, d]`` contiguous, ``lse_acc`` fp32 ``[B, h, S]`` whose last dimension may be a slice of a
    longer sequence, ``out_new`` bf16 ``[S, B, h, d]``, ``lse_new`` fp32 ``[B, h, S]``.  Oracle:
    ``l = logaddexp(lse_acc, lse_new); out = exp(lse_acc - l) * out_acc + exp(lse_new - l) * out_new``."""
    S, B, h, d = out_acc.shape
    if not (out_acc.is_contiguous() and lse_acc.stride(2) == 1 and lse_acc.stride(0) == h * lse_acc.stride(1)):
        raise ValueError("attention_merge: unsupported layout")
    out_new, lse_new = out_new.contiguous(), lse_new.contiguous()
    lib = _lib.load()
    rc = lib.hg_attn_merge(out_acc.data_ptr(), lse_acc.data_ptr(), lse_acc.stride(1), out_new.data_ptr(),
                           lse_new.data_ptr(), S, B * h, d, _lib.stream())
    _lib.check(rc, "hg_attn_merge")
    _lib.count_launch()
