"""The C++ autograd nodes against the Python classes that they stand for: the same kernels, hence the same bits."""
import contextlib

import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.models.modules import ops_add
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV, LP = "cuda", torch.bfloat16


@contextlib.contextmanager
def python_nodes():
    native, _lib.NATIVE = _lib.native(), None
    try:
        yield
    finally:
        _lib.NATIVE = native


def both(build, inputs, params=()):
    """Outputs, input gradients and parameter gradients (autograd's and main_grad) of ``build`` on either route."""
    assert _lib.native() is not None
    res = []
    for route in (contextlib.nullcontext, python_nodes):
        _lib.reset_launches()
        with route():
            xs = [t.detach().clone().requires_grad_(t.requires_grad) for t in inputs]
            ps = []
            for p in params:
                q = torch.nn.Parameter(p.detach().clone())
                if hasattr(p, "fresh"):
                    q.main_grad, q.mg_fresh = torch.full(p.shape, 2.0, device=DEV), p.fresh
                ps.append(q)
            outs = build(*xs, *ps)
            outs = outs if isinstance(outs, tuple) else (outs,)
            g = torch.Generator(device=DEV).manual_seed(1)
            torch.autograd.backward(outs, [torch.randn(o.shape, device=DEV, generator=g).to(o.dtype) for o in outs])
        res.append(([*outs, *[t.grad for t in xs], *[p.grad for p in ps], *[getattr(p, "main_grad", None) for p in ps]],
                    [getattr(p, "mg_fresh", None) for p in ps], _lib.launches()))
    (a, fa, la), (b, fb, lb) = res
    assert fa == fb and la == lb > 0 and len(a) == len(b)
    for s, t in zip(a, b):
        assert (s is None) == (t is None) and (s is None or (s.dtype == t.dtype and torch.equal(s, t)))
    _lib.assert_healthy()


def randn(*shape, grad=True, dtype=LP):
    return torch.randn(*shape, device=DEV).to(dtype).requires_grad_(grad)


def param(*shape, fresh=None):
    p = torch.nn.Parameter(torch.randn(*shape, device=DEV).to(LP))
    if fresh is not None:
        p.fresh = fresh
    return p


# few rows, rows of more than two dimensions and in another order, pair tiles
@pytest.mark.parametrize("shape,N", [((5, 64), 48), ((3, 7, 72), 104), ((300, 264), 520)])
@pytest.mark.parametrize("biased", [False, True])
@pytest.mark.parametrize("fresh", [None, True, False])
def test_linear(shape, N, biased, fresh):
    torch.manual_seed(N)
    ps = [param(N, shape[-1], fresh=fresh)] + ([param(N)] if biased else [])
    both(lambda x, w, b=None: ops.linear(x, w, b), [randn(*shape)], ps)
    both(lambda x, w, b=None: ops.linear(x, w, b), [randn(*shape, grad=False)], ps)
    if len(shape) == 3:
        both(lambda x, w, b=None: ops.linear(x.transpose(0, 1), w, b), [randn(shape[1], shape[0], shape[2])], ps)


@pytest.mark.parametrize("rms", [True, False])
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("fresh", [None, True, False])
def test_norm(rms, residual, fresh):
    torch.manual_seed(2)
    ps = [param(136, fresh=fresh)] + ([] if rms else [param(136)])

    def run(x, *rest):
        r, rest = (rest[0], rest[1:]) if residual else (None, rest)
        y, h = ops.norm(x, rest[0], rest[1] if not rms else None, 1e-5, rms, residual=r)
        return (y, h) if residual else y

    both(run, [randn(3, 5, 136) for _ in range(1 + residual)], ps)
    if residual:
        both(lambda *a: run(*a)[0], [randn(3, 5, 136) for _ in range(2)], ps)      # the sum itself unused
        both(lambda *a: run(*a)[1], [randn(3, 5, 136) for _ in range(2)], ps)      # only the sum used


@pytest.mark.parametrize("kind,F", [("swiglu", 32), ("geglu", 48), ("gelu", 40)])
def test_activation_and_add(kind, F):
    both(lambda y: ops.activation(y, kind), [randn(2, 9, F)])
    both(lambda y: ops.activation(y.transpose(0, 1), kind), [randn(2, 9, F)])
    both(ops_add, [randn(4, 9, F), randn(4, 9, F)])


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("positions", [False, True])
@pytest.mark.parametrize("ng", [1, 2])
def test_rotation_and_attention(interleaved, positions, ng):
    S, B, nh, hd = 130, 2, 4, 64
    cos, sin = ops.rope_tables(S + 8, hd, 10000.0, DEV)
    slots = torch.tensor([g * (nh // ng + 2) + j for g in range(ng) for j in range(nh // ng + 1)], dtype=torch.int32, device=DEV)
    pos = torch.randint(0, S, (S * B,), device=DEV) if positions else None

    def run(x, w):
        qkv = ops.rope_packed(ops.linear(x, w), slots, hd, cos, sin, B, pos, 0 if positions else 5, interleaved)
        return ops.flash_attention_packed(qkv, S, B, nh, ng, hd)

    both(run, [randn(S * B, 64)], [param((nh + 2 * ng) * hd, 64)])


def test_saved_tensor_hooks_checkpoints_and_inference():
    x, w = randn(40, 64), param(64, 64)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.clone(), lambda t: t):
        ops.activation(ops.linear(x, w), "swiglu").sum().backward()
    assert len(packed) == 3
    from torch.utils.checkpoint import checkpoint

    got, want = (r(lambda t: ops.activation(ops.linear(t, w), "gelu"), x) for r in
                 (lambda f, t: checkpoint(f, t, use_reentrant=False), lambda f, t: f(t)))
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(got.sum(), (x, w)), torch.autograd.grad(want.sum(), (x, w))))
    with torch.inference_mode():
        assert torch.equal(ops.linear(x, w), ops.linear(x, w)) and not ops.linear(x, w).requires_grad
    y = ops.linear(x, w)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()
    a = ops.linear(x, w)
    b = ops.activation(a, "gelu")
    a.detach().add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        b.sum().backward()


def test_errors_are_those_of_the_python_route():
    with pytest.raises(TypeError):
        ops.linear(randn(8, 16, dtype=torch.float32), param(8, 16))
    with pytest.raises(ValueError):
        ops.linear(randn(8, 16), param(8, 24))
    with pytest.raises(_lib.KernelError):
        ops.norm(randn(8, 20), param(20), None, 1e-5, True)
    w = param(64, 64)
    w.main_grad = torch.zeros(32, 64, device=DEV)
    with pytest.raises(ValueError, match="bad output"):
        ops.linear(randn(300, 64), w).sum().backward()


# the gradients of a bias and a norm's bias written, or added, straight to their buffers; with a hook on the parameter they take the
# way through autograd that shows them to it
@pytest.mark.parametrize("rows", [1, 40, 999])
@pytest.mark.parametrize("fresh", [True, False])
@pytest.mark.parametrize("hooked", [False, True])
def test_bias_gradients_go_to_their_buffers(rows, fresh, hooked):
    g = torch.Generator(device="cuda").manual_seed(rows)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
    w, b, nw, nb = [torch.nn.Parameter(t) for t in (rand(520, 264), rand(520), rand(264), rand(264))]
    seen = []
    for p in (w, b, nw, nb):
        p.main_grad, p.mg_fresh = torch.full(p.shape, 2.0, device="cuda"), fresh
        if hooked and p.dim() == 1 and p is not nw:
            p.register_hook(lambda t: seen.append(t.shape))
    x, dy = rand(rows, 264).requires_grad_(), rand(rows, 520)
    n = ops.norm(x, nw, nb, 1e-5, rms=False)[0]
    ops.linear(n, w, b).backward(dy)
    ref = dy.double().sum(0)
    dn = (dy.double() @ w.detach().double()).sum(0)
    for p, want in ((b, ref), (nb, dn)):
        if hooked:
            assert p.mg_fresh is fresh and (p.main_grad == 2.0).all() and len(seen) == 2
        else:
            assert p.grad is None and not p.mg_fresh
            got = p.main_grad.double() - (0.0 if fresh else 2.0)
            # fp32 sums of 16-bit rows; dy of the norm was rounded to 16 bits once: rows of about 23 (520 products of unit normals)
            atol = 1e-5 * rows ** 0.5 * 10 if p is b else 2.0 ** -9 * 23 * 6 * rows ** 0.5
            assert torch.allclose(got, want, rtol=1e-5, atol=atol)


# with a buffer bound: autograd.grad and backward(inputs=...) give the gradient of a bias and leave its buffer alone, a graph of the
# gradient is one, and a bias may change between forward and backward; afterwards a plain backward writes the buffers
def test_bias_gradients_that_are_asked_for():
    rand = lambda *shape: torch.randn(*shape, device=DEV).to(LP)
    w, b, nw, nb = [torch.nn.Parameter(t) for t in (rand(520, 264), rand(520), rand(264), rand(264))]
    for p in (w, b, nw, nb):
        p.main_grad, p.mg_fresh = torch.full(p.shape, 2.0, device=DEV), True
    x, dy, dn = rand(40, 264), rand(40, 520).requires_grad_(), rand(40, 264)
    linear, norm = lambda: ops.linear(x, w, b), lambda: ops.norm(x, nw, nb, 1e-5, rms=False)[0]
    assert _lib.native() is not None
    untouched = lambda: all(p.mg_fresh and (p.main_grad == 2.0).all() for p in (b, nb))
    want = dy.detach().double().sum(0), dn.double().sum(0)
    close = lambda got, ref: torch.allclose(got.double(), ref, rtol=2.0 ** -8, atol=1e-4)      # fp32 sums of 40, one rounding
    got = torch.autograd.grad(linear(), b, dy.detach())[0], torch.autograd.grad(norm(), nb, dn)[0]
    assert all(close(g, r) for g, r in zip(got, want)) and untouched()
    torch.autograd.backward(linear(), dy.detach(), inputs=[b])
    torch.autograd.backward(norm(), dn, inputs=[nb])
    assert close(b.grad, want[0]) and close(nb.grad, want[1]) and untouched()
    b.grad = nb.grad = None
    (g,) = torch.autograd.grad(linear(), b, dy, create_graph=True)
    v = torch.randn(520, device=DEV)
    assert torch.equal(torch.autograd.grad((g * v).sum(), dy)[0], v.to(LP).expand(40, 520)) and untouched()
    y, n = linear(), norm()
    with torch.no_grad():
        b.mul_(2.0)
        nb.mul_(2.0)
    nw.mg_fresh = True                       # the norm's kernel has one switch for both sums
    y.backward(dy.detach())
    n.backward(dn)
    assert b.grad is None and nb.grad is None and not b.mg_fresh and not nb.mg_fresh
    assert torch.allclose(b.main_grad.double(), want[0], rtol=1e-5, atol=1e-4)
    assert torch.allclose(nb.main_grad.double(), want[1], rtol=1e-5, atol=1e-4)
    _lib.assert_healthy()
