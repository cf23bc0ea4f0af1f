"""A decoder layer launched by one native call against the same layer run module by module."""
import pytest
import torch

from hetu_galvatron_b200.models.inference import StaticInferenceContext
from hetu_galvatron_b200.models.modules import GalvatronDecoderLayer
from hetu_galvatron_b200.models.spec import LayerCtx, ModelSpec
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def layer(norm, act, pos, bias, nh, ng, hd):
    spec = ModelSpec(family="llama", hidden=nh * hd, layers=1, heads=nh, kv_heads=ng, head_dim=hd, ffn=264, vocab=512,
                     padded_vocab=512, seq_len=0, norm=norm, activation=act, pos=pos, bias=bias, qkv_bias=bias)
    m = GalvatronDecoderLayer(spec, LayerCtx(), DEV, "layer")
    m.reset_parameters()
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(0.1 * torch.randn_like(p))
    return m


# one row and the most that the native call takes; grouped heads on both head dims; biases; no rotation; a cache whose
# first sequences belong to others
@pytest.mark.parametrize("norm,act,pos,bias,nh,ng,hd", [("RMSNorm", "swiglu", "rope", False, 4, 2, 128),
                                                        ("LayerNorm", "gelu", "none", True, 6, 6, 64),
                                                        ("RMSNorm", "geglu", "rope", True, 8, 1, 64)])
@pytest.mark.parametrize("S,B,past,b0", [(1, 1, 0, 0), (1, 4, 70, 2), (16, 4, 5, 0)])
def test_native_step_equals_the_modules(norm, act, pos, bias, nh, ng, hd, S, B, past, b0):
    torch.manual_seed(S + B)
    m = layer(norm, act, pos, bias, nh, ng, hd)
    x = torch.randn(S, B, nh * hd, device=DEV).to(torch.bfloat16)
    caches = torch.randn(2, past + S + 3, b0 + B + 1, ng, hd, device=DEV).to(torch.bfloat16)
    got = []
    for hooked in (False, True):                      # a hook inside the layer sends it module by module
        ic = StaticInferenceContext(b0 + B + 1, past + S + 3)
        ic.sequence_len_offset, ic.batch_size_offset = past, b0
        mine = caches.clone()
        ic.key_value_memory_dict[0] = (mine[0], mine[1])
        m.attn.attention.inference_context = ic
        h = m.ffn.mlp.register_forward_hook(lambda *_: None) if hooked else None
        with torch.no_grad():
            assert m._takes_native_step(x) is not hooked
            got.append((m(x), mine))
        if h is not None:
            h.remove()
        m.attn.attention.inference_context = None
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    _lib.assert_healthy()


def test_native_step_is_left_to_inference_without_gradient():
    m = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64)
    x = torch.randn(65, 1, 256, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        assert not m._takes_native_step(x) and m._takes_native_step(x[:64].contiguous())
    assert not m._takes_native_step(x[:1])


@pytest.mark.parametrize("S", [1, 80])                # one native call; module by module
def test_autograd_knows_of_the_writes_to_the_caches(S):
    m = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64)
    x = torch.randn(S, 1, 256, device=DEV).to(torch.bfloat16)
    ic = StaticInferenceContext(1, 2 * S)
    m.attn.attention.inference_context = ic
    with torch.no_grad():
        m(x)
        kc, vc = ic.key_value_memory_dict[0]
        before = kc._version, vc._version
        m(x)
        assert kc._version > before[0] and vc._version > before[1]
        # a graph over the cached keys notices that they have changed
        w = torch.ones(64, device=DEV, dtype=torch.bfloat16).requires_grad_()
        with torch.enable_grad():
            loss = (kc[:1] * w).sum()
        m(x)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()
    with torch.inference_mode():                      # caches of inference mode are not written outside of it
        ic.key_value_memory_dict.clear()
        m(x)
        m(x)
    with torch.no_grad(), pytest.raises(RuntimeError, match="[Ii]nference"):
        m(x)
    m.attn.attention.inference_context = None
    _lib.assert_healthy()


def test_native_step_drops_no_tangent():
    """Forward-mode differentiation is refused by the modules' functions, not answered without the tangent."""
    from torch.autograd import forward_ad

    m = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64)
    x = torch.randn(1, 1, 256, device=DEV).to(torch.bfloat16)
    m.attn.attention.inference_context = StaticInferenceContext(1, 8)
    with torch.no_grad(), forward_ad.dual_level():
        with pytest.raises(NotImplementedError):
            m(forward_ad.make_dual(x, torch.ones_like(x)))
        m(x)
    m.attn.attention.inference_context = None
    _lib.assert_healthy()


def test_native_step_is_left_to_the_layers_own_modules():
    from hetu_galvatron_b200.models.modules import MLP, GalvatronMLP

    x = torch.randn(1, 1, 256, device=DEV).to(torch.bfloat16)

    class Twice(MLP):
        def forward(self, x):
            return 2 * super().forward(x)

    class Other(GalvatronMLP):
        def forward(self, attn_out, residual):
            return attn_out

    def patched(m):
        plain = m.attn.input_layernorm.forward
        m.attn.input_layernorm.forward = lambda x, residual=None: plain(2 * x, residual)

    for change in (lambda m: setattr(m.ffn.mlp, "__class__", Twice), lambda m: setattr(m.ffn, "__class__", Other), patched):
        m = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64)
        m.attn.attention.inference_context = StaticInferenceContext(1, 8)
        with torch.no_grad():
            assert m._takes_native_step(x)
            change(m)
            assert not m._takes_native_step(x)
            want = m.ffn(m.attn(x), x)
            assert torch.equal(m(x), want)


def test_attention_of_another_kind():
    m = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64)
    m.attn = torch.nn.Identity()
    x = torch.randn(1, 1, 256, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(m(x), m.ffn(x, x))


def test_native_step_with_a_weight_that_is_computed():
    """A parametrized weight is a new tensor at every access: it has to live until the kernels that read it are launched."""
    from torch.nn.utils import parametrize

    class Scaled(torch.nn.Module):
        def forward(self, w):
            return w * 2

    m, x = layer("RMSNorm", "swiglu", "rope", False, 4, 4, 64), torch.randn(1, 1, 256, device=DEV).to(torch.bfloat16)
    got = []
    for native in (True, False):
        m.attn.attention.inference_context = StaticInferenceContext(1, 8)
        if native:
            parametrize.register_parametrization(m.attn.attention.linear_proj, "weight", Scaled())
        with torch.no_grad():
            assert m._takes_native_step(x)
            got.append(m(x) if native else m.ffn(m.attn(x), x))
    assert torch.equal(*got)
    _lib.assert_healthy()


# one key range, the tile kernel, several ranges and their merge
@pytest.mark.parametrize("B,past,launches", [(4, 3, 10), (1, 500, 10), (1, 1600, 11), (64, 100, 11), (64, 3, 10)])
def test_launches_of_the_native_step(B, past, launches):
    m, x = layer("RMSNorm", "swiglu", "rope", False, 8, 8, 64), torch.randn(1, B, 512, device=DEV).to(torch.bfloat16)
    for native in (True, False):
        ic = StaticInferenceContext(B, past + 1)
        ic.sequence_len_offset = past
        m.attn.attention.inference_context = ic
        with torch.no_grad():
            before = _lib.launches()
            m(x) if native else m.ffn(m.attn(x), x)
            assert _lib.launches() - before == launches
    _lib.assert_healthy()


def test_weights_written_just_before_a_step_are_the_ones_it_reads():
    """The step's kernels read weights before the kernel in front of them has ended, but never before the step began."""
    torch.manual_seed(7)
    m = layer("RMSNorm", "swiglu", "rope", False, 8, 8, 128)
    x = torch.randn(1, 4, 1024, device=DEV).to(torch.bfloat16)
    weights = [p for p in m.parameters() if p.dim() == 2]
    new = [torch.randn_like(p) * 0.02 for p in weights]
    got = []
    for hooked in (False, True):
        ic = StaticInferenceContext(4, 8)
        m.attn.attention.inference_context = ic
        with torch.no_grad():
            for p in weights:
                p.zero_()
            m(x)                                          # fills position 0
            ic.sequence_len_offset = 1
            h = m.ffn.mlp.register_forward_hook(lambda *_: None) if hooked else None
            torch.cuda._sleep(1000000)                    # the writes are still queued when the step is launched
            for p, w in zip(weights, new):
                p.copy_(w)
            got.append(m(x))
        if h is not None:
            h.remove()
        m.attn.attention.inference_context = None
    assert torch.equal(got[0], got[1])
    _lib.assert_healthy()


def test_norm_weights_and_biases_written_just_before_a_step():
    """As above for every vector of a layer, the first norm's weight and bias last, against the modules after a wait."""
    torch.manual_seed(8)
    m = layer("LayerNorm", "gelu", "none", True, 8, 8, 128)
    x = torch.randn(1, 4, 1024, device=DEV).to(torch.bfloat16)
    n1 = m.attn.input_layernorm
    vectors = sorted((p for p in m.parameters() if p.dim() == 1), key=lambda p: p is n1.weight or p is n1.bias)
    assert len(vectors) == 8 and vectors[-1] is n1.bias
    new = [torch.randn_like(p) for p in vectors]
    got = []
    for hooked in (False, True):
        ic = StaticInferenceContext(4, 8)
        m.attn.attention.inference_context = ic
        with torch.no_grad():
            for p in vectors:
                p.zero_()
            m(x)                                          # fills position 0
            ic.sequence_len_offset = 1
            h = m.ffn.mlp.register_forward_hook(lambda *_: None) if hooked else None
            torch.cuda._sleep(1000000)
            for p, v in zip(vectors, new):
                p.copy_(v)
            if hooked:
                torch.cuda.synchronize()
            got.append(m(x))
        if h is not None:
            h.remove()
        m.attn.attention.inference_context = None
    assert torch.equal(got[0], got[1]) and got[0].abs().sum() > 0
    _lib.assert_healthy()
