"""Which way a backward of attention goes, on both sides of each line of the rule."""
import ctypes

import pytest
import torch

from hetu_galvatron_b200.ops import _lib, attention


# dS in one launch (1.03 GiB; head dim 64, 1.34), in launches of 1024, 768 and 704 key blocks, of few, in even and uneven ones over the
# sequences (512 and 256 key blocks of 16 heads on 8), head dim 64 in several, not even one kv head, no pair that sees each other
@pytest.mark.parametrize("S,B,nh,ng,hd,causal,k0,stored", [
    (4096, 2, 32, 32, 128, 1, 0, True), (8192, 1, 20, 20, 64, 1, 0, True), (4096, 1, 28, 4, 128, 1, 0, True),
    (8192, 1, 32, 32, 128, 1, 0, True), (8192, 2, 25, 25, 128, 1, 0, True), (8192, 1, 32, 32, 128, 0, 0, False),
    (16384, 1, 32, 32, 128, 1, 0, False), (8192, 1, 28, 4, 128, 1, 0, False), (16384, 1, 32, 8, 128, 1, 0, False),
    (4096, 4, 28, 4, 128, 1, 0, False), (8192, 2, 25, 25, 64, 1, 0, False), (16384, 1, 64, 8, 128, 1, 0, False),
    (300, 1, 2, 1, 128, 1, 900, False)])
def test_rule_of_stored_ds(S, B, nh, ng, hd, causal, k0, stored):
    lib, sizes = _lib.load(), (S, S, B, nh, ng, hd, causal, 0, k0)
    wants, floats = (ctypes.c_longlong * 3)(), ctypes.c_longlong()
    lib.hg_flash_bwd_wants(*sizes, wants)
    n = lib.hg_flash_bwd_pieces(*sizes, ctypes.byref(floats))
    assert list(wants) == [lib.hg_flash_bwd_scratch_of(*sizes, 0), *((n, floats.value) if stored else (0, 0))]
    assert 4 * (lib.hg_flash_bwd_scratch(*sizes) - lib.hg_flash_bwd_scratch_of(*sizes, 0)) <= 3 << 29


# heads of 18, 69 and 45 MB, of 2.6 MB in even pieces, one query of one head, the most pieces, none
@pytest.mark.parametrize("S,B,nh,ng,hd,pieces,heads", [(4096, 2, 32, 32, 128, 32, 2), (8192, 1, 20, 20, 64, 20, 1),
                                                       (6600, 1, 32, 32, 64, 32, 1), (1531, 1, 28, 4, 128, 2, 14), (1, 1, 1, 1, 64, 1, 1),
                                                       (4992, 1, 60, 60, 128, 60, 1), (16384, 1, 64, 8, 128, 0, 0)])
def test_pieces_of_ds(S, B, nh, ng, hd, pieces, heads):
    lib, sizes, floats = _lib.load(), (S, S, B, nh, ng, hd, 1, 0, 0), ctypes.c_longlong()
    assert lib.hg_flash_bwd_pieces(*sizes, ctypes.byref(floats)) == pieces <= 64
    blocks = (S + 127) // 128
    head = blocks * (blocks + 1) // 2 * 128 * 128 // 2                   # floats of a head's tiles
    assert floats.value == heads * head and (heads <= 1 or 4 * heads * head <= 48 << 20)
    assert lib.hg_flash_bwd_scratch(*sizes) - lib.hg_flash_bwd_scratch_of(*sizes, 0) == pieces * floats.value


def test_an_allocator_without_room_is_left_alone(monkeypatch):
    """It is asked for dS once, not at every layer of every backward, and later again; the other scratch it has to have."""
    lib, sizes, device = _lib.load(), (4096, 4096, 2, 32, 32, 128, True, 0, 0), torch.device("cuda", 7)
    small, floats, asked = lib.hg_flash_bwd_scratch_of(*sizes, 0), ctypes.c_longlong(), []
    assert lib.hg_flash_bwd_pieces(*sizes, ctypes.byref(floats)) == 32

    def empty(n, dtype, device):
        asked.append(n)
        if len(asked) % 4 == 0 and n == floats.value:                    # the third piece
            raise torch.cuda.OutOfMemoryError("no room")
        return torch.zeros(1)

    monkeypatch.setattr(attention.torch, "empty", empty)
    calls = lambda n: [attention._backward_scratch(lib, *sizes, device)[1] for _ in range(n)]
    assert calls(1) == [[]] and asked == [small] + [floats.value] * 3
    assert calls(256) == [[]] * 256 and asked[4:] == [small] * 256
    assert lib.hg_flash_bwd_has_room(6)                                  # another device
    assert calls(1) == [[]] and asked[260:] == asked[:4]
