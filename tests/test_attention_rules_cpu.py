"""Which way a backward of attention goes, on both sides of each line of the rule."""
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
    assert bool(lib.hg_flash_bwd_tiles_pay(*sizes)) is stored
    assert 4 * (lib.hg_flash_bwd_scratch(*sizes) - lib.hg_flash_bwd_scratch_of(*sizes, 0)) <= 3 << 29


def test_an_allocator_without_room_is_left_alone(monkeypatch):
    """It is asked for dS once, not at every layer of every backward, and later again; a smaller scratch it has to have."""
    lib, sizes, device = _lib.load(), (4096, 4096, 2, 32, 32, 128, True, 0, 0), torch.device("cuda", 7)
    small, asked = lib.hg_flash_bwd_scratch_of(*sizes, 0), []

    def empty(n, dtype, device):
        asked.append(n)
        if n > small:
            raise torch.cuda.OutOfMemoryError("no room")
        return torch.zeros(1)

    monkeypatch.setattr(attention.torch, "empty", empty)
    calls = lambda n: [attention._backward_scratch(lib, *sizes, device) for _ in range(n)]
    calls(1)
    assert asked == [lib.hg_flash_bwd_scratch(*sizes), small]
    calls(256)
    assert asked[2:] == [small] * 256
    assert lib.hg_flash_bwd_has_room(6)                                  # another device
    calls(1)
    assert asked[258:] == asked[:2]
