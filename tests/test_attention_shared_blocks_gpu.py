"""dK and dV of key blocks that several CTAs share, against one CTA per key block and 64-bit arithmetic."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.attention import _desc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel_err(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


# grouped heads whose early blocks are shared and late ones are not, no mask, one head of many queries, queries that start
# behind or before the keys (keys that no query sees among them), a ragged end, the
# last length that is not shared for one head and the first that is, the last grid of less than a wave and the first of more
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("Sq,Skv,B,nh,ng,causal,q0,k0", [
    (1531, 1531, 1, 7, 1, True, 0, 0), (640, 640, 1, 6, 2, False, 0, 0), (2049, 2049, 1, 1, 1, True, 0, 0),
    (1100, 1100, 2, 1, 1, True, 0, 0), (1200, 1200, 2, 1, 1, True, 0, 0),
    (512, 900, 2, 4, 2, True, 388, 0), (300, 700, 1, 8, 1, True, 0, 100), (4096, 130, 1, 2, 1, True, 0, 64),
    (257, 129, 37, 2, 2, True, 0, 0), (257, 129, 75, 1, 1, False, 0, 0)])
def test_shared_key_blocks(hd, Sq, Skv, B, nh, ng, causal, q0, k0):
    g = torch.Generator(device=DEV).manual_seed(Sq + Skv + hd)
    q, dout = (torch.randn(Sq, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "qd")
    k, v = (torch.randn(Skv, B, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv")
    scale, qpg, lib = hd ** -0.5, nh // ng, _lib.load()
    out, lse = ops.flash_attention(q, k, v, causal=causal, q_pos0=q0, k_pos0=k0, return_lse=True)
    dq, dk, dv = ops.flash_backward(q, k, v, out, dout, lse, causal, scale, q0, k0)

    one = [torch.empty_like(t) for t in (q, k, v)]                        # the entry point without scratch for parts
    heads = lambda t: _desc(t, t.stride(0), t.stride(1), nh, qpg, 1, 0)
    groups = lambda t: _desc(t, t.stride(0), t.stride(1), ng, 1, 0, 0)
    args = [heads(q), groups(k), groups(v), heads(out), heads(dout)]
    outs = [heads(one[0]), groups(one[1]), groups(one[2])]
    dsum = torch.empty(B, nh, Sq, device=DEV)
    rc = lib.hg_flash_bwd(*[ctypes.byref(t) for t in args], lse.data_ptr(), dsum.data_ptr(),
                          *[ctypes.byref(t) for t in outs], Sq, Skv, B, nh, ng, hd, int(causal), q0, k0, scale, _lib.stream())
    assert rc == 0
    # the same 16-bit probabilities and dS, summed in fp32 in another order and rounded once
    assert torch.equal(dq, one[0]) and rel_err(dk, one[1]) < 1e-3 and rel_err(dv, one[2]) < 1e-3

    if B == 1 or Sq * Skv < 1 << 18:
        qr, kr, vr = (t.double().requires_grad_() for t in (q, k, v))
        s = torch.einsum("sbhd,tbhd->bhst", qr, kr.repeat_interleave(qpg, 2)) * scale
        dead = torch.zeros(Sq, Skv, dtype=torch.bool, device=DEV)
        if causal:
            dead = (torch.arange(Skv, device=DEV) + k0)[None, :] > (torch.arange(Sq, device=DEV) + q0)[:, None]
        p = torch.softmax(s.masked_fill(dead, -1e300), -1).masked_fill(dead, 0.0)      # rows that see no key: zeros
        torch.einsum("bhst,tbhd->sbhd", p, vr.repeat_interleave(qpg, 2)).backward(dout.double())
        # two 16-bit roundings before a product, one after (see test_attention_hd64_gpu)
        assert rel_err(dk, kr.grad) < 5e-3 and rel_err(dv, vr.grad) < 5e-3
    _lib.assert_healthy()


# dS in memory: launches over some of the heads, or of the sequences, where all tiles are too many (1.5 GiB), a last one smaller than
# the others; one query block, one row more than two, an odd number of them; rows and keys that end inside a block
@pytest.mark.parametrize("Sq,Skv,B,nh,ng,hd,causal,q0,k0", [
    (8192, 8192, 1, 32, 32, 64, True, 0, 0), (4096, 4096, 3, 16, 8, 64, False, 0, 0), (8192, 8192, 2, 25, 25, 128, True, 0, 0),
    (1, 1, 1, 1, 1, 128, True, 0, 0), (128, 65, 2, 3, 1, 64, True, 0, 0), (257, 257, 1, 2, 2, 128, True, 0, 0),
    (640, 200, 2, 4, 2, 128, False, 0, 0), (385, 1000, 1, 4, 4, 64, True, 615, 0), (300, 300, 1, 2, 1, 128, True, 0, 900)])
def test_dq_from_stored_ds(Sq, Skv, B, nh, ng, hd, causal, q0, k0):
    lib = _lib.load()
    sizes = (Sq, Skv, B, nh, ng, hd, int(causal), q0, k0)
    assert lib.hg_flash_bwd_scratch(*sizes) > lib.hg_flash_bwd_scratch_of(*sizes, 0) or k0 > q0 + Sq    # pairs to store
    assert 4 * (lib.hg_flash_bwd_scratch(*sizes) - lib.hg_flash_bwd_scratch_of(*sizes, 0)) <= 3 << 29
    g = torch.Generator(device=DEV).manual_seed(Sq + Skv + hd)
    q, dout = (torch.randn(Sq, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "qd")
    k, v = (torch.randn(Skv, B, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv")
    out, lse = ops.flash_attention(q, k, v, causal=causal, q_pos0=q0, k_pos0=k0, return_lse=True)
    grads = ops.flash_backward(q, k, v, out, dout, lse, causal, hd ** -0.5, q0, k0)
    one = [torch.empty_like(t) for t in (q, k, v)]                       # without scratch S and dP are computed again for dQ
    kv = lambda t: _desc(t, t.stride(0), t.stride(1), ng, 1, 0, 0)
    heads = lambda t: _desc(t, t.stride(0), t.stride(1), nh, nh // ng, 1, 0)
    args, outs = [heads(q), kv(k), kv(v), heads(out), heads(dout)], [heads(one[0]), kv(one[1]), kv(one[2])]
    dsum = torch.empty(B, nh, Sq, device=DEV)
    assert lib.hg_flash_bwd(*[ctypes.byref(t) for t in args], lse.data_ptr(), dsum.data_ptr(), *[ctypes.byref(t) for t in outs],
                            Sq, Skv, B, nh, ng, hd, int(causal), q0, k0, hd ** -0.5, _lib.stream()) == 0
    # the same 16-bit dS, multiplied and added by the tensor core in the same order
    assert torch.equal(grads[0], one[0])
    assert all((a.double() - b.double()).norm() <= 1e-3 * b.double().norm() for a, b in zip(grads[1:], one[1:]))
    _lib.assert_healthy()


# all pieces, one piece less, pieces of one float less, one that starts at an odd place; scratch for shared key blocks, one float less, for
# the row sums alone; launches over some of the heads and of the sequences, which the callers of this package do not ask for; key blocks
# that are shared; pieces of several heads and of one
@pytest.mark.parametrize("Sq,Skv,B,nh,ng,hd,causal", [(8192, 8192, 1, 32, 32, 64, True), (4096, 4096, 3, 16, 8, 64, False),
                                                      (1531, 1531, 1, 28, 4, 128, True), (1531, 1531, 1, 7, 1, 128, True),
                                                      (640, 640, 1, 6, 2, 64, False), (4096, 4096, 1, 10, 5, 128, True)])
def test_backward_with_any_scratch(Sq, Skv, B, nh, ng, hd, causal):
    lib, sizes, each = _lib.load(), (Sq, Skv, B, nh, ng, hd, int(causal), 0, 0), ctypes.c_longlong()
    g = torch.Generator(device=DEV).manual_seed(Sq + hd)
    q, dout = (torch.randn(Sq, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "qd")
    k, v = (torch.randn(Skv, B, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv")
    out, lse = ops.flash_attention(q, k, v, causal=causal, return_lse=True)
    parts, sums = lib.hg_flash_bwd_scratch_of(*sizes, 0), B * nh * Sq
    n = lib.hg_flash_bwd_pieces(*sizes, ctypes.byref(each))
    assert n > 0
    pieces = [torch.empty(each.value + 64, device=DEV) for _ in range(n)]
    at = [t.data_ptr() for t in pieces]
    heads = lambda t: ctypes.byref(_desc(t, t.stride(0), t.stride(1), nh, nh // ng, 1, 0))
    kv = lambda t: ctypes.byref(_desc(t, t.stride(0), t.stride(1), ng, 1, 0, 0))
    results, launched = [], ctypes.c_int()
    for floats, tiles, most in ((parts, at, each.value), (parts, at[1:], each.value), (parts, at, each.value - 1),
                                (parts, [*at[:-1], at[-1] + 4], each.value), (max(parts - 1, sums), at, each.value), (sums, [], 0)):
        got, ws = [torch.full_like(t, float("nan")) for t in (q, k, v)], torch.full((floats,), float("nan"), device=DEV)
        for t in pieces:
            t.fill_(float("nan"))
        assert lib.hg_flash_bwd_ws(heads(q), kv(k), kv(v), heads(out), heads(dout), lse.data_ptr(), ws.data_ptr(), floats,
                                   (ctypes.c_void_p * len(tiles))(*tiles), len(tiles), most, heads(got[0]), kv(got[1]), kv(got[2]),
                                   *sizes[:6], int(causal), 0, 0, hd ** -0.5, ctypes.byref(launched), _lib.stream()) == 0
        stored = not all(t.isnan().all() for t in pieces)
        assert stored == (tiles is at and most == each.value)
        assert all(t[each.value:].isnan().all() for t in pieces)         # nothing behind them
        results.append(got)
    for got in results:
        assert torch.equal(got[0], results[0][0])                        # dQ: the same bits, stored dS or not
        assert rel_err(got[1], results[0][1]) < 1e-3 and rel_err(got[2], results[0][2]) < 1e-3
    for i in (1, 2):                                                     # dK and dV: as long as the same CTAs share
        assert all(torch.equal(results[0][i], r[i]) for r in results[1:4]) and torch.equal(results[4][i], results[5][i])
    _lib.assert_healthy()


# a process that may have less memory than dS takes: one failed allocation, not one a layer, and the same gradients; by the C++ nodes and
# by the function of the parallel paths
@pytest.mark.parametrize("route", ["node", "function"])
def test_backward_without_room_for_ds(route):
    code = """
import torch
from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
S, nh, hd, route = 2048, 32, 128, %r
g = torch.Generator(device="cuda").manual_seed(1)
qkv = torch.randn(S, 3 * nh * hd, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
d = torch.randn(S, nh * hd, device="cuda", generator=g).to(torch.bfloat16)
if route == "node":
    assert _lib.load() and _lib.NATIVE is not None
    out = ops.flash_attention_packed(qkv, S, 1, nh, nh, hd, causal=True)
    run = lambda: torch.autograd.grad(out, qkv, d, retain_graph=True)
else:
    q, k, v = (t.contiguous() for t in qkv.detach().view(S, 1, nh, 3, hd).unbind(3))
    out, lse = ops.flash_attention(q, k, v, causal=True, return_lse=True)
    run = lambda: ops.flash_backward(q, k, v, out, d.view(S, 1, nh, hd), lse, True, hd ** -0.5)
want = [t.cpu() for t in run()]
ooms = lambda: torch.cuda.memory_stats()["num_ooms"]
assert ooms() == 0
torch.cuda.empty_cache()
total = torch.cuda.get_device_properties(0).total_memory
torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 120e6) / total)      # dS: 142 MB
for _ in range(3):
    assert all(torch.equal(a.cpu(), b) for a, b in zip(run(), want))
assert ooms() == 1, ooms()
_lib.assert_healthy()
""" % (route,)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root)
    assert run.returncode == 0, run.stderr[-2000:]
