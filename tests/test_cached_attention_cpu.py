"""Which caches the kernels of the cached forward may be handed (anything else takes the tensor-library path, which
checks shapes itself)."""
import pytest
import torch

from hetu_galvatron_b200.ops import _lib
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


# Measured on both sides (csrc/sm100/flash_decode.cu): calls that the kernels with spread keys lose by more than a tenth,
# and calls that they win
@pytest.mark.skipif(not _lib.available(), reason="the kernel library is not built")
@pytest.mark.parametrize("Sq,B,nh,nkv,hd,keys,spread", [
    (8, 16, 32, 32, 128, 2000, 0), (4, 6, 32, 32, 128, 2000, 0), (2, 4, 32, 32, 128, 1536, 0), (8, 6, 32, 32, 64, 512, 0),
    (1, 4, 32, 32, 128, 1536, 0), (1, 3, 32, 32, 128, 4000, 0), (1, 8, 32, 8, 128, 128, 0), (1, 8, 28, 4, 64, 256, 0),
    (1, 1, 32, 8, 128, 1000, 0), (1, 1, 32, 8, 128, 2000, 1), (1, 4, 32, 32, 64, 2000, 1), (1, 8, 32, 8, 128, 1000, 1),
    (1, 6, 32, 32, 128, 128, 1), (1, 16, 32, 32, 128, 64, 1), (1, 32, 28, 4, 128, 200, 1), (2, 10, 32, 8, 128, 2000, 1)])
def test_rule_of_the_spread_kernels(Sq, B, nh, nkv, hd, keys, spread):
    assert _lib.load().hg_flash_decode_pays(Sq, keys, B, nh, nkv, hd, 1, keys - Sq, 0) == spread
