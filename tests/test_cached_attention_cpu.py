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
    for k, v in ((make(), make()), (make(), cache()), (cache(), make())):
        assert caches_usable(like, k, v, past, S, b0, B, 2, 64) is ok


def strided(size, stride, offset=0):
    return torch.zeros(8192, dtype=torch.bfloat16).as_strided(size, stride, offset)


def pair(size, k_stride, v_stride, v_offset):
    flat = torch.zeros(65536, dtype=torch.bfloat16)
    return flat.as_strided(size, k_stride), flat.as_strided(size, v_stride, v_offset)


# keys and values written by different threads: each element has its own memory
@pytest.mark.parametrize("make,ok", [
    (lambda: (cache(), cache()), True),
    (lambda: (lambda c: (c, c))(cache()), False),                                        # one cache for both
    (lambda: (lambda c: (c[:4], c[4:]))(cache(seq=8)), True),                            # halves of one buffer
    (lambda: (lambda c: (c[:5], c[3:]))(cache(seq=8)), False),
    (lambda: (lambda c: (c[:, :2], c[:, 2:]))(cache(batch=4)), True),                    # side by side along the batch
    (lambda: (lambda c: (c[:, :3], c[:, 1:]))(cache(batch=4)), False),
    (lambda: (lambda c: (c[:, :, 0], c[:, :, 1]))(torch.zeros(8, 4, 2, 2, 64, dtype=torch.bfloat16)), True),    # [.., k | v, ..]
    (lambda: pair((4, 2, 2, 64), (512, 256, 64, 1), (512, 256, 64, 1), 128), True),
    (lambda: pair((4, 2, 2, 64), (512, 256, 64, 1), (512, 256, 64, 1), 64), False),      # second head of k = first of v
    (lambda: pair((4, 2, 2, 64), (512, 256, 64, 1), (512, 256, 64, 1), 192), False),     # v runs into the next sequence's k
    (lambda: pair((4, 2, 2, 64), (512, 256, 64, 1), (256, 1024, 64, 1), 128), False),    # other strides in one range
    (lambda: (strided((4, 4, 2, 64), (128, 128, 64, 1)), cache(seq=4)), False),          # tokens of two sequences in one place
    (lambda: (strided((4, 4, 2, 64), (256, 128, 64, 1)), cache(seq=4)), False),
    (lambda: (strided((4, 4, 2, 64), (128, 512, 64, 1)), cache(seq=4)), True)])
def test_caches_do_not_share_memory(make, ok):
    k, v = make()
    S, B = min(k.shape[0], v.shape[0]), min(k.shape[1], v.shape[1])
    like = torch.zeros(1, dtype=torch.bfloat16)
    assert caches_usable(like, k, v, 0, S, 0, B, 2, 64) is ok and caches_usable(like, v, k, 0, S, 0, B, 2, 64) is ok


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


def test_caches_do_not_share_memory_by_their_elements():
    """The same verdict as the sets of elements, over every layout of small caches that passes for one cache alone."""
    from hetu_galvatron_b200.ops.attention import _disjoint, _nested

    flat, w, seen = torch.zeros(4096), 8, set()
    for n0, n1, m0, m1 in ((1, 1, 1, 1), (3, 2, 3, 2), (2, 3, 4, 1), (1, 3, 3, 1), (4, 2, 2, 4)):
        for s0, s1 in ((8, 24), (16, 48), (24, 8), (64, 16), (40, 8), (8, 8), (16, 40)):
            if not (_nested(((s0, n0), (s1, n1)), w) and _nested(((s0, m0), (s1, m1)), w)):
                continue
            a = flat.as_strided((n0, n1, 1, w), (s0, s1, w, 1))
            mine = {s0 * i + s1 * j + e for i in range(n0) for j in range(n1) for e in range(w)}
            for off in range(0, 260, 4):
                b = flat.as_strided((m0, m1, 1, w), (s0, s1, w, 1), off)
                apart = mine.isdisjoint(off + s0 * i + s1 * j + e for i in range(m0) for j in range(m1) for e in range(w))
                got = _disjoint(a, b, w)
                assert got is _disjoint(b, a, w) and (apart or not got)
                # strides that only one of the two uses may be refused although nothing is shared
                assert got is apart or not _nested(((s0, max(n0, m0)), (s1, max(n1, m1))), w)
                seen.add(got)
    assert seen == {True, False}
