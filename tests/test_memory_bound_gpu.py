"""Memory-bound kernels at the edges of their thread layouts."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib
from hetu_galvatron_b200.ops.gemm import column_sums

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


# every group size of the norm backward (32 to 512 threads per row, one to four chunks per thread), rows fewer than,
# equal to and more than the row groups of the grid
@pytest.mark.parametrize("rms", [True, False])
@pytest.mark.parametrize("rows,H", [(1, 8), (5000, 256), (37, 264), (1500, 768), (3, 1024), (700, 1600), (300, 4104),
                                    (20, 8200), (310, 16384)])
def test_norm_backward(rms, rows, H):
    g = torch.Generator(device=DEV).manual_seed(rows + H)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x = r(rows, H).to(torch.bfloat16).requires_grad_()
    w = (1 + 0.1 * r(H)).to(torch.bfloat16).requires_grad_()
    b = None if rms else (0.1 * r(H)).to(torch.bfloat16).requires_grad_()
    res = r(rows, H).to(torch.bfloat16)
    y, h = ops.norm(x, w, b, 1e-5, rms, residual=res)
    gy, gh = r(rows, H).to(torch.bfloat16), r(rows, H).to(torch.bfloat16)
    w.main_grad = torch.full((H + 1,), 2.0, device=DEV)[1:]        # accumulated into, at any alignment
    torch.autograd.backward([y, h], [gy, gh])
    hd = h.detach().double().requires_grad_()
    wd = w.detach().double().requires_grad_()
    bd = None if rms else b.detach().double().requires_grad_()
    if rms:
        yd = hd * torch.rsqrt(hd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    else:
        yd = torch.nn.functional.layer_norm(hd, (H,), wd, bd, 1e-5)
    torch.autograd.backward([yd, hd], [gy.double(), gh.double()])
    assert rel_err(x.grad, hd.grad) < 2.0 ** -8                     # fp32 arithmetic, one rounding
    assert rel_err(w.main_grad, wd.grad + 2.0) < 1e-5               # fp32 sums
    if not rms:
        assert rel_err(b.grad, bd.grad) < 2.0 ** -8
    _lib.assert_healthy()


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (64, 1000), (2997, 6400), (100000, 16), (5, 70000)])
def test_column_sums(rows, cols):
    x = torch.randn(rows, cols, device=DEV).to(torch.bfloat16)
    ref = x.double().sum(0)
    # fp32 sums of `rows` unit-variance terms, one rounding of the result
    assert torch.allclose(column_sums(x).double(), ref, rtol=2.0 ** -8, atol=1e-6 * rows)
    wide = torch.randn(rows, cols + 8, device=DEV).to(torch.bfloat16)
    assert torch.allclose(column_sums(wide[:, :cols]).double(), wide[:, :cols].double().sum(0), rtol=2.0 ** -8,
                          atol=1e-6 * rows)


def test_bias_gradient_has_a_gradient():
    """create_graph: the bias gradient is linear in the incoming gradient."""
    x, w = (torch.randn(n, 64, device=DEV).to(torch.bfloat16) for n in (24, 40))
    b = torch.zeros(40, device=DEV, dtype=torch.bfloat16).requires_grad_()
    dy = torch.randn(24, 40, device=DEV).to(torch.bfloat16).requires_grad_()
    v = torch.randn(40, device=DEV).to(torch.bfloat16)
    (gb,) = torch.autograd.grad(ops.linear(x, w, b), b, dy, create_graph=True)
    assert torch.equal(torch.autograd.grad((gb * v).sum(), dy)[0], v.expand(24, 40))
    _lib.assert_healthy()


# few tokens and small tables, which are scattered, the most that are sorted and one more, two more that are sorted (the kernels on their
# own: below); tokens of other shards, a buffer that holds something
@pytest.mark.parametrize("tokens,rows,H", [(255, 12288, 264), (256, 12288, 264), (1025, 6145, 2056), (1024, 3071, 4096),
                                           (1024, 3072, 4096), (16384, 98304, 2056), (16385, 98304, 2056), (1024, 16000, 4096),
                                           (4097, 39532, 4096)])
@pytest.mark.parametrize("fresh", [True, False])
@pytest.mark.parametrize("positions", [False, True])
def test_embedding_gradient(tokens, rows, H, fresh, positions):
    from hetu_galvatron_b200 import ops
    from hetu_galvatron_b200.ops import _lib

    g = torch.Generator(device="cuda").manual_seed(tokens + H)
    v0 = 7
    u = torch.rand(tokens, device="cuda", generator=g, dtype=torch.float64)
    ids = (torch.exp(u * float(torch.tensor(rows + 2.0).log())).long() - 1).clamp_(0, rows + 1) + v0 - 1   # some before, some behind
    W = torch.nn.Parameter(torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16))
    W.main_grad, W.mg_fresh = torch.full((rows, H), float("nan") if fresh else 2.0, device="cuda"), fresh
    pos = torch.nn.Parameter(torch.zeros(tokens // 2 + 1, H, device="cuda", dtype=torch.bfloat16)) if positions else None
    dout = torch.randn(tokens, H, device="cuda", generator=g).to(torch.bfloat16)
    ops.embedding(ids, W, v0, pos, 2).backward(dout)
    want = torch.full((rows + 2, H), 0.0 if fresh else 2.0, device="cuda", dtype=torch.float64)
    want.index_add_(0, ids - v0 + 1, dout.double())
    most = int(torch.bincount(ids - v0 + 1).max())
    # fp32 sums of at most `most` unit normals and what was there, each addition off by half a unit in the last place
    assert torch.allclose(W.main_grad.double(), want[1:-1], rtol=0, atol=most * 2.0 ** -24 * (2 + 6 * most ** 0.5))
    assert not W.mg_fresh
    if positions:
        ref = torch.zeros(pos.shape, device="cuda", dtype=torch.float64).index_add_(0, torch.arange(tokens, device="cuda") // 2, dout.double())
        assert torch.allclose(pos.grad.double(), ref, rtol=2.0 ** -8, atol=1e-6)
    _lib.assert_healthy()


# the kernels on their own, whatever the rule says: one token, counts around a block of eight, a power of two and the most there can be;
# more columns than a block takes; a shard that has none of the tokens
@pytest.mark.parametrize("tokens", [1, 7, 8, 9, 255, 256, 257, 1025, 16384])
@pytest.mark.parametrize("rows,H", [(3, 8), (300, 2056)])
@pytest.mark.parametrize("v0", [0, 7, 10 ** 6])
def test_sums_of_sorted_tokens(tokens, rows, H, v0):
    from hetu_galvatron_b200.ops import _lib

    lib, g = _lib.load(), torch.Generator(device="cuda").manual_seed(tokens + H)
    ids = torch.randint(0, rows + 12, (tokens,), device="cuda", generator=g)
    dout = torch.randn(tokens, H, device="cuda", generator=g).to(torch.bfloat16)
    dW, keys = torch.full((rows + 1, H), float("nan"), device="cuda"), torch.empty(tokens, dtype=torch.int32, device="cuda")
    assert lib.hg_embedding_bwd_runs(ids.data_ptr(), dout.data_ptr(), dW.data_ptr(), keys.data_ptr(), tokens, H, v0, rows, _lib.stream()) == 0
    want, mine = torch.zeros(rows, H, device="cuda", dtype=torch.float64), (ids >= v0) & (ids < v0 + rows)
    want.index_add_(0, ids[mine] - v0, dout[mine].double())
    most = int(torch.bincount(ids).max())
    assert torch.allclose(dW[:rows].double(), want, rtol=0, atol=most * 2.0 ** -24 * (2 + 6 * most ** 0.5))      # as above
    assert dW[rows].isnan().all()
    _lib.assert_healthy()
