"""Attention of one query per head and kv head (streamed keys, clusters of CTAs) against 64 bits."""
import math

import pytest
import torch

from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.attention import _desc, _forward_launch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(q, k, v, causal, q0):
    out, lse = torch.full_like(q, 7.0), torch.full((q.shape[1], q.shape[2], 1), 7.0, device=DEV)
    d = [_desc(t, t.stride(0), t.stride(1), t.shape[2], 1, 1 if t is q or t is out else 0, 0) for t in (q, k, v, out)]
    _forward_launch(*d, lse, 1, k.shape[0], q.shape[1], q.shape[2], q.shape[2], q.shape[3], causal, q0, 0,
                    1.0 / math.sqrt(q.shape[3]))
    return out, lse[..., 0]


# keys around a step (16 and 32 of them), around the ring and a batch of steps, one to eight CTAs a head with even and uneven
# shares, two waves of heads; a last query that sees fewer keys than there are, and none
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,nh", [(1, 3), (2, 32), (5, 23), (3, 99)])
@pytest.mark.parametrize("keys,q0", [(1, 0), (15, 14), (17, 16), (33, 32), (64, 63), (129, 128), (300, 299), (1025, 1024), (700, 450),
                                     (40, -1)])
def test_streamed_keys(hd, B, nh, keys, q0):
    g = torch.Generator(device=DEV).manual_seed(keys + nh)
    q = torch.randn(1, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16)
    cache = torch.randn(2, keys + 3, B + 1, nh, hd, device=DEV, generator=g).to(torch.bfloat16)
    k, v = cache[0, :keys, 1:], cache[1, :keys, 1:]
    cache[:, keys:] = float("nan")                                    # rows past the end are not read
    out, lse = run(q, k, v, True, q0)
    seen = min(keys, q0 + 1)
    s = torch.einsum("sbhd,tbhd->bht", q.double(), k[:seen].double()) / math.sqrt(hd)
    ref = torch.einsum("bht,tbhd->bhd", s.softmax(-1), v[:seen].double()) if seen else torch.zeros(B, nh, hd, device=DEV).double()
    if seen:
        assert torch.allclose(lse.double(), torch.logsumexp(s, -1), rtol=1e-5, atol=1e-5)       # fp32 scores and sums
    else:
        assert torch.isneginf(lse).all()
    assert torch.allclose(out[0].double(), ref, rtol=2.0 ** -8, atol=1e-5)                     # one rounding to 16 bits
    again, lse2 = run(q, k, v, True, q0)
    assert torch.equal(out, again) and torch.equal(lse, lse2)
    free, _ = run(q, k, v, False, 0)
    if seen == keys:
        assert torch.equal(out, free)
    _lib.assert_healthy()


def test_scores_that_are_no_numbers():
    q, k = torch.ones(1, 1, 2, 128, device=DEV, dtype=torch.bfloat16), torch.ones(200, 1, 2, 128, device=DEV, dtype=torch.bfloat16)
    v = torch.ones_like(k)
    k[150, 0, 0, 3] = float("inf")
    k[70, 0, 1, 5] = -float("inf")
    out, lse = run(q, k, v, True, 199)
    assert torch.isnan(out[0, 0, 0]).all() and torch.isneginf(lse[0, 0])
    assert (out[0, 0, 1] == 1).all() and torch.isfinite(lse[0, 1])     # a score of -inf counts nothing
    k[150, 0, 0, 3] = float("nan")
    out, _ = run(q, k, v, True, 199)
    assert torch.isnan(out[0, 0, 0]).all() and (out[0, 0, 1] == 1).all()
    _lib.assert_healthy()
