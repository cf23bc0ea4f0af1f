"""Attention grids of many more blocks than CTAs run at once: every block's result is what the block gives in a grid of its own."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one key block per query block and fewer steps than stages, blocks of very different length, ragged ends, grouped heads,
# queries that see no key, a grid of just over the CTAs that fit, thousands of blocks
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("Sq,Skv,B,nh,ng,causal,q0,k0", [
    (100, 100, 300, 4, 4, True, 0, 0), (130, 257, 150, 4, 2, False, 0, 0), (777, 777, 24, 8, 2, True, 0, 0),
    (513, 900, 40, 4, 4, True, 387, 0), (400, 300, 64, 4, 1, True, 0, 150), (256, 256, 149, 1, 1, True, 0, 0),
    (128, 128, 1200, 4, 4, False, 0, 0)])
def test_blocks_do_not_depend_on_the_grid(hd, Sq, Skv, B, nh, ng, causal, q0, k0):
    g = torch.Generator(device=DEV).manual_seed(Sq + Skv + B)
    q, dout = (torch.randn(Sq, B, nh, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "qd")
    k, v = (torch.randn(Skv, B, ng, hd, device=DEV, generator=g).to(torch.bfloat16) for _ in "kv")

    def run(q, k, v, dout):
        out, lse = ops.flash_attention(q, k, v, causal=causal, q_pos0=q0, k_pos0=k0, return_lse=True)
        return (out, *ops.flash_backward(q, k, v, out, dout, lse, causal, hd ** -0.5, q0, k0)), lse

    whole, lse = run(q, k, v, dout)
    again, lse2 = run(q, k, v, dout)
    assert torch.equal(lse, lse2) and all(torch.equal(a, b) for a, b in zip(whole, again))
    for b in sorted({0, 1, B // 3, B // 2, B - 2, B - 1}):
        one, l1 = run(*(t[:, b:b + 1].contiguous() for t in (q, k, v, dout)))
        assert torch.equal(l1[0], lse[b])
        for i, (x, y) in enumerate(zip(one, whole)):
            y = y[:, b:b + 1]
            # the keys of a small grid may be shared by several CTAs: dK and dV in another order of the sums
            assert torch.equal(x, y) or (i >= 2 and (x.double() - y.double()).norm() <= 1e-3 * y.double().norm())
    _lib.assert_healthy()
