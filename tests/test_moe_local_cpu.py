"""Host side of the single-GPU expert dispatch: which calls its kernels are handed."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from hetu_galvatron_b200.models.moe import SEG_ALIGN, GalvatronMoEMLP, _rows16, local_dispatch_usable, local_rows
from hetu_galvatron_b200.models.spec import LayerCtx, ModelSpec


@pytest.mark.parametrize("what,E,ok", [
    ({}, 8, True), ({}, 256, True), ({}, 257, False), ({}, 0, False), ({"probs": (4, 1)}, 8, False), ({"probs": (3, 2)}, 8, False),
    ({"probs": (8,)}, 8, True), ({"probs": (4, 3)}, 8, False), ({"idx": (3, 2)}, 8, False), ({"idx": (4, 3)}, 8, False),
    ({"idx": (8,)}, 8, False), ({"x": (4, 12)}, 8, False), ({"idx_device": "cpu"}, 8, False), ({"probs_device": "cpu"}, 8, False),
    ({"x_device": "cpu"}, 8, False), ({"dtype": torch.float32}, 8, False), ({"idx_dtype": torch.float32}, 8, False),
    ({"idx_dtype": torch.int32}, 8, True)])
def test_local_dispatch_usable(what, E, ok):
    with FakeTensorMode():                       # tensors of a GPU that need not be there
        x = torch.empty(what.get("x", (4, 16)), dtype=what.get("dtype", torch.bfloat16), device=what.get("x_device", "cuda"))
        probs = torch.empty(what.get("probs", (4, 2)), device=what.get("probs_device", "cuda"))
        idx = torch.empty(what.get("idx", (4, 2)), dtype=what.get("idx_dtype", torch.int64), device=what.get("idx_device", "cuda"))
        assert local_dispatch_usable(x, probs, idx, E, 2) is ok


def test_fewer_weights_than_pairs_are_refused():
    spec = ModelSpec(family="llama", hidden=16, layers=1, heads=2, kv_heads=2, head_dim=8, ffn=16, vocab=64, padded_vocab=64,
                     seq_len=0, experts=4, moe_ffn=16, topk=2, dtype=torch.float32)
    m = GalvatronMoEMLP(spec, LayerCtx(), "cpu", "mlp")
    m.reset_parameters()
    idx = torch.tensor([[0, 1], [2, 3], [1, 0]])
    with pytest.raises(IndexError):
        m(torch.randn(3, 16), torch.rand(3, 1), idx)
    assert m(torch.randn(3, 16), torch.rand(3, 2), idx).shape == (3, 16)


@pytest.mark.parametrize("offset,copied", [(0, False), (8, False), (1, True), (4, True)])
def test_rows_start_on_16_byte_boundaries(offset, copied):
    flat = torch.arange(64 + 24, dtype=torch.int16)
    flat = flat[(-flat.data_ptr() % 16) // 2:]
    for t in (flat[offset:offset + 64].view(4, 16), flat[offset:offset + 64].view(2, 32)[:, :16]):
        r = _rows16(t)
        assert r.data_ptr() % 16 == 0 and torch.equal(r, t) and (r.data_ptr() != t.data_ptr()) is copied


@pytest.mark.parametrize("n", [0, 1, 2, 8, 127, 128, 129, 130, 256, 385, 1000])
@pytest.mark.parametrize("E", [1, 2, 3, 8, 160, 256])
def test_buffer_rows_are_what_the_worst_routing_fills(n, E):
    def rows(counts):
        return sum(-(-c // SEG_ALIGN) for c in counts) * SEG_ALIGN

    m = min(n, E)                                # one pair for every expert, the rest for one of them
    assert local_rows(n, E) == max(rows([1] * (m - 1) + [n - m + 1]) if n else 0, SEG_ALIGN)
    g = torch.Generator().manual_seed(n + E)
    for skew in (0.0, 0.5, 2.0):
        e = torch.multinomial(torch.rand(E, generator=g) ** (1 + skew), max(n, 1), True, generator=g)[:n]
        assert rows(e.bincount(minlength=E).tolist()) <= local_rows(n, E)
