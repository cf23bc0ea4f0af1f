"""Which caches the kernels of the cached forward may be handed (anything else takes the tensor-library path, which
checks shapes itself)."""
import pytest
import torch

from hetu_galvatron_b200.ops.attention import caches_usable


def cache(seq=8, batch=4, ng=2, hd=64):
    return torch.zeros(seq, batch, ng, hd, dtype=torch.bfloat16)


@pytest.mark.parametrize("make,past,S,b0,B,ok", [
    (cache, 5, 3, 1, 3, True), (cache, 6, 3, 0, 4, False), (cache, 0, 1, 2, 3, False), (cache, -1, 1, 0, 1, False),
    (cache, 0, 1, -1, 1, False), (lambda: cache(ng=1), 0, 1, 0, 1, False), (lambda: cache(hd=128), 0, 1, 0, 1, False),
    (lambda: cache().float(), 0, 1, 0, 1, False), (lambda: cache(batch=1).expand(8, 4, 2, 64), 0, 1, 0, 4, False),
    (lambda: cache(batch=2).transpose(0, 1), 0, 1, 0, 2, True), (lambda: cache(hd=72)[..., 8:], 0, 1, 0, 1, False),
    (lambda: cache().requires_grad_(), 0, 1, 0, 1, False)])
def test_caches_usable(make, past, S, b0, B, ok):
    like = torch.zeros(1, dtype=torch.bfloat16)
    c = make()
    for k, v in ((c, c), (c, cache()), (cache(), c)):
        assert caches_usable(like, k, v, past, S, b0, B, 2, 64) is ok
