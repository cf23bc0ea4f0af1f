"""Attention of a few queries over long key ranges (csrc/sm100/flash_decode.cu) and the cached forward built on it."""
import math

import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.attention import _desc, _forward_launch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def reference64(q, k, v, causal, q_pos0, k_pos0):
    o, lse = [], []
    nh, ng = q.shape[2], k.shape[2]
    for h in range(nh):
        s = torch.einsum("sbd,tbd->bst", q[:, :, h].double(), k[:, :, h // (nh // ng)].double()) / math.sqrt(q.shape[3])
        if causal:
            qp = torch.arange(q.shape[0], device=DEV)[:, None] + q_pos0
            s = s.masked_fill(torch.arange(k.shape[0], device=DEV) + k_pos0 > qp, float("-inf"))
        lse.append(torch.logsumexp(s, -1))
        p = torch.nan_to_num(torch.exp(s - lse[-1][..., None]))
        o.append(torch.einsum("bst,tbd->sbd", p, v[:, :, h // (nh // ng)].double()))
    return torch.stack(o, 2), torch.stack(lse, 1)


# one to eight rows per kv head (padded row counts 1, 2, 4, 8), one key range and many, range ends in and off a range's
# last key, 64 and 128 keys per CTA, a key offset that hides every key from the first query
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("Sq,B,nh,ng,Skv,causal,q0,k0", [
    (1, 1, 4, 4, 1, True, 0, 0), (1, 3, 2, 2, 64, True, 63, 0), (1, 2, 7, 1, 65, True, 64, 0), (1, 1, 8, 2, 1000, True, 999, 0),
    (1, 40, 32, 32, 129, True, 128, 0), (3, 2, 4, 2, 300, True, 297, 0), (8, 1, 2, 2, 200, False, 0, 0),
    (2, 1, 8, 2, 777, True, 100, 101), (1, 2, 4, 4, 500, True, 200, 0)])
def test_flash_decode(hd, Sq, B, nh, ng, Skv, causal, q0, k0):
    g = torch.Generator(device=DEV).manual_seed(Skv + nh)
    q = torch.randn(Sq, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16)
    cache = torch.randn(2, Skv + 5, B + 1, ng, hd, device=DEV, generator=g).to(torch.bfloat16)
    k, v = cache[0, :Skv, 1:], cache[1, :Skv, 1:]
    out, lse = torch.empty_like(q), torch.empty(B, nh, Sq, device=DEV)
    d = [_desc(t, t.stride(0), t.stride(1), t.shape[2], n, 1, 0) for t, n in ((q, nh // ng), (k, 1), (v, 1), (out, nh // ng))]
    d[1].hs = d[2].hs = 0
    _forward_launch(*d, lse, Sq, Skv, B, nh, ng, hd, causal, q0, k0, 1.0 / math.sqrt(hd), spread=True)
    ref, ref_lse = reference64(q, k, v, causal, q0, k0)
    dead = torch.isinf(ref_lse)
    assert torch.equal(dead, torch.isinf(lse))
    assert torch.allclose(lse[~dead].double(), ref_lse[~dead], rtol=1e-5, atol=1e-5)      # fp32 scores and sums
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8, atol=1e-5)                   # one rounding to bf16
    # what the rule gives the call to must agree (16-bit probabilities on the tile kernel: 2^-9 per element)
    by_rule = ops.flash_attention(q, k, v, causal=causal, q_pos0=q0, k_pos0=k0)
    assert ((by_rule.double() - ref).norm() <= 5e-3 * ref.norm()).item()
    _lib.assert_healthy()


# a NaN in a query, in one key that the row sees, in a key that it does not see; a score of +inf; -inf scores only.  One key
# range (40 keys) and several, whose first holds the bad key
@pytest.mark.parametrize("Skv", [40, 300])
@pytest.mark.parametrize("qpg", [1, 4])
@pytest.mark.parametrize("what", ["query", "key", "unseen", "inf", "-inf"])
def test_flash_decode_passes_nan_and_inf_on(Skv, qpg, what):
    """Bad scores reach the output as on the tile kernel."""
    B, ng, hd = 2, 2, 64
    g = torch.Generator(device=DEV).manual_seed(Skv + qpg)
    q = torch.randn(1, B, ng * qpg, hd, device=DEV, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(Skv, B, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv")
    q0 = Skv - 1
    if what == "query":
        q[0, 1, 0, 3] = float("nan")
    elif what == "unseen":
        q0, k[-1, 1, 0, 3] = Skv - 2, float("nan")
    else:
        q[0, 1, :, 3] = 1.0
        k[slice(None) if what == "-inf" else 7, 1, 0, 3] = float("nan") if what == "key" else float(what)
    got = []
    for spread in (True, False):
        out, lse = torch.empty_like(q), torch.empty(B, ng * qpg, 1, device=DEV)
        d = [_desc(t, t.stride(0), t.stride(1), t.shape[2], n, 1, 0) for t, n in ((q, qpg), (k, 1), (v, 1), (out, qpg))]
        d[1].hs = d[2].hs = 0
        _forward_launch(*d, lse, 1, Skv, B, ng * qpg, ng, hd, True, q0, 0, 1.0 / math.sqrt(hd), spread=spread)
        got.append((out, lse))
    bad = {"query": 1, "key": qpg, "inf": qpg}.get(what, 0)          # query heads whose output has to be NaN
    for out, _ in got:
        assert out[0, 1, :bad].isnan().all() and out[0, 1, bad:].isfinite().all() and out[0, 0].isfinite().all()
    live = got[0][0].isfinite()
    assert torch.equal(live, got[1][0].isfinite())
    assert torch.allclose(got[0][0][live].double(), got[1][0][live].double(), rtol=2e-2, atol=2e-2)   # 16-bit probabilities there
    assert torch.equal(got[0][1].isfinite(), got[1][1].isfinite())
    _lib.assert_healthy()


@pytest.mark.parametrize("interleaved,rot", [(False, 1.0), (True, 1.0), (False, 0.5), (True, 0.25), (False, 0.0)])
@pytest.mark.parametrize("S,B,nh,ng,hd,past", [(1, 4, 4, 4, 128, 70), (5, 2, 8, 2, 64, 3), (130, 1, 4, 1, 128, 0)])
def test_cached_attention_against_rope_and_copies(S, B, nh, ng, hd, past, interleaved, rot):
    """Rotating, appending and attending in place gives what the separate operations give."""
    qpg, P = nh // ng, (nh + 2 * ng) * hd
    g = torch.Generator(device=DEV).manual_seed(S + past)
    qkv = torch.randn(S * B, P, device=DEV, generator=g).to(torch.bfloat16)
    caches = [torch.randn(past + S + 2, B + 2, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv"]
    want = [c.clone() for c in caches]
    cos, sin = ops.rope_tables(past + S + 2, int(hd * rot), 10000.0, DEV) if rot else (None, None)
    with torch.no_grad():
        ref = qkv.clone()
        if rot:
            slots = torch.tensor([i * (qpg + 2) + j for i in range(ng) for j in range(qpg + 1)], device=DEV, dtype=torch.int32)
            ref = ops.rope_packed(ref, slots, hd, cos, sin, B, None, past, interleaved)
        q, k, v = ops.attention.split_packed(ref, nh, ng, hd)
        want[0][past:past + S, 1:1 + B] = k.reshape(S, B, ng, hd)
        want[1][past:past + S, 1:1 + B] = v.reshape(S, B, ng, hd)
        o = ops.flash_attention(q.reshape(S, B, nh, hd), want[0][:past + S, 1:1 + B], want[1][:past + S, 1:1 + B],
                                causal=True, q_pos0=past)
        got = ops.attention.cached_attention(qkv, caches[0], caches[1], past, 1, S, B, nh, ng, hd, cos, sin, interleaved)
    assert torch.equal(got, o.reshape(S, B, nh * hd))
    assert torch.equal(caches[0], want[0]) and torch.equal(caches[1], want[1])
    _lib.assert_healthy()
