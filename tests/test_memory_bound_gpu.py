"""Memory-bound kernels at the edges of their thread layouts."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel_err(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("shift", [0, 1])
def test_embedding_gradient_into_any_buffer(shift):
    """Repeated tokens and learned positions into gradient buffers that are, and are not, 16-byte aligned."""
    V, H, S, B = 50, 264, 40, 3
    ids = torch.randint(0, V + 10, (S * B,), device=DEV)            # some ids belong to another shard
    W = torch.randn(V, H, device=DEV).to(torch.bfloat16).requires_grad_()
    P = torch.randn(S, H, device=DEV).to(torch.bfloat16).requires_grad_()
    for t in (W, P):
        t.main_grad = torch.full((t.numel() + shift,), 1.0, device=DEV)[shift:].view(t.shape)
    out = ops.embedding(ids, W, v0=0, pos_emb=P, batch=B)
    g = torch.randn(S * B, H, device=DEV).to(torch.bfloat16)
    out.backward(g)
    inside = ids < V
    ref = torch.ones(V, H, dtype=torch.float64, device=DEV).index_add_(0, ids[inside], g.double()[inside])
    assert rel_err(W.main_grad, ref) < 1e-6                         # fp32 sums of a few terms
    assert rel_err(P.main_grad, 1.0 + g.double().view(S, B, H).sum(1)) < 1e-6
    _lib.assert_healthy()
