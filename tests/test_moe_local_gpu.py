"""Single-GPU expert dispatch (csrc/sm100/moe_local.cu): the placement against a list-based restatement, and the row
passes against index operations in 64 bits."""
from types import SimpleNamespace

import pytest
import torch

from hetu_galvatron_b200.models.moe import SEG_ALIGN, _LocalCombine, _LocalDispatch, _LocalPlan
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def placement(idx, E):
    """(row_start, dest) of every pair, expert-major and in pair order."""
    by = [[] for _ in range(E)]
    for p, e in enumerate(idx.reshape(-1).tolist()):
        if e >= 0:
            by[e].append(p)
    starts, dest = [0], [-1] * idx.numel()
    for e in range(E):
        for i, p in enumerate(by[e]):
            dest[p] = starts[-1] + i
        starts.append(starts[-1] + (len(by[e]) + SEG_ALIGN - 1) // SEG_ALIGN * SEG_ALIGN)
    return starts, dest


# one token; all pairs on one expert; chunk edges of the placement kernel (1024 pairs); dropped pairs; 256 experts
@pytest.mark.parametrize("T,k,E,H,drop", [(1, 1, 1, 8, 0.0), (128, 2, 8, 264, 0.0), (512, 2, 8, 4096, 0.1),
                                          (513, 2, 4, 72, 1.0), (1000, 8, 160, 256, 0.3), (341, 3, 256, 2048, 0.0)])
def test_local_dispatch_and_combine(T, k, E, H, drop):
    g = torch.Generator().manual_seed(T + k + E)
    idx = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    idx[torch.rand(T, k, generator=g) < drop] = -1
    plan = _LocalPlan(idx.to(DEV), E)
    starts, dest = placement(idx, E)
    assert plan.row_start.tolist() == starts and plan.dest.tolist() == dest
    src = [-1] * plan.rows
    for p, r in enumerate(dest):
        if r >= 0:
            src[r] = p
    assert plan.src.tolist() == src

    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV).requires_grad_()
    w = torch.rand(T, k, generator=g).to(DEV).requires_grad_()
    buf = _LocalDispatch.apply(x, plan)
    tok = torch.tensor([p // k if p >= 0 else 0 for p in src], device=DEV)
    live = torch.tensor([p >= 0 for p in src], device=DEV)[:, None]
    assert torch.equal(buf, torch.where(live, x.detach()[tok], torch.zeros_like(x.detach()[tok])))
    dbuf = torch.randn(plan.rows, H, generator=g).to(torch.bfloat16).to(DEV)
    buf.backward(dbuf)
    d = torch.tensor(dest, device=DEV).view(T, k)
    rows = dbuf.double()[d.clamp(min=0)] * (d >= 0)[..., None]
    assert torch.allclose(x.grad.double(), rows.sum(1), rtol=2.0 ** -8, atol=1e-5)   # one rounding to bf16

    y = torch.randn(plan.rows, H, generator=g).to(torch.bfloat16).to(DEV).requires_grad_()
    out = _LocalCombine.apply(y, w, plan)
    rows = y.detach().double()[d.clamp(min=0)] * (d >= 0)[..., None]
    ref = (rows * w.detach().double()[..., None]).sum(1)
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8, atol=1e-5)
    dout = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    out.backward(dout)
    ref_dw = (rows * dout.double()[:, None]).sum(-1)
    assert torch.allclose(w.grad.double(), ref_dw, rtol=1e-4, atol=1e-5 * H ** 0.5)  # fp32 sums of H products
    ref_dy = torch.zeros(plan.rows, H, dtype=torch.float64, device=DEV)
    ref_dy[d[d >= 0]] = (w.detach().double()[..., None] * dout.double()[:, None])[d >= 0]
    assert torch.allclose(y.grad.double(), ref_dy, rtol=2.0 ** -8, atol=1e-7)
    _lib.assert_healthy()


# one column, every other column and a transposed matrix of expert numbers; 32-bit ones
@pytest.mark.parametrize("view", [lambda i: i[:, :1], lambda i: i[:, ::2], lambda i: i[:, :2].t().contiguous().t(),
                                  lambda i: i.to(torch.int32)[:, 1:2]])
def test_placement_of_strided_indices(view):
    E = 8
    idx = torch.randint(0, E, (300, 4), generator=torch.Generator().manual_seed(3))
    plan = _LocalPlan(view(idx.to(DEV)), E)
    starts, dest = placement(view(idx), E)
    assert plan.row_start.tolist() == starts and plan.dest.tolist() == dest
    _lib.assert_healthy()


def test_rows_between_16_byte_boundaries():
    """Tokens, expert rows and their gradients as slices of a flat buffer that start anywhere."""
    T, k, E, H = 5, 2, 4, 64
    idx = torch.randint(0, E, (T, k), device=DEV)
    plan = _LocalPlan(idx, E)

    def both(shape):
        n = shape[0] * shape[1]
        t = torch.randn(n + 3, device=DEV).to(torch.bfloat16)[3:].view(shape)
        return [v.requires_grad_() for v in (t.detach(), t.detach().clone())]

    w = torch.rand(T, k, device=DEV)
    for f, shape, out_shape in ((lambda t: _LocalDispatch.apply(t, plan), (T, H), (plan.rows, H)),
                                (lambda t: _LocalCombine.apply(t, w, plan), (plan.rows, H), (T, H))):
        xs, gs = both(shape), both(out_shape)
        outs = [f(x) for x in xs]
        for o, g in zip(outs, gs):
            o.backward(g.detach())
        assert torch.equal(outs[0], outs[1]) and torch.equal(xs[0].grad, xs[1].grad)
    lib = _lib.load()
    odd = torch.zeros(E * 256 * H + 1, device=DEV, dtype=torch.bfloat16)[1:]
    assert lib.hg_moe_scatter(odd.data_ptr(), H, plan.src.data_ptr(), 0, plan.rows, k, H, xs[1].data_ptr(), 0) == -1
    assert lib.hg_moe_gather(odd.data_ptr(), plan.dest.data_ptr(), 0, T, k, H, xs[1].data_ptr(), 0) == -1
    assert lib.hg_moe_dot(xs[1].data_ptr(), odd.data_ptr(), H, plan.dest.data_ptr(), T * k, k, H, w.data_ptr(), 0) == -1
    _lib.assert_healthy()


def test_allgather_dispatcher_buffers_only_the_local_pairs():
    """One of four ranks' view of the gathered pairs: the expert buffer follows what is routed to its two experts."""
    from hetu_galvatron_b200.models.moe import GalvatronMoEMLP
    from hetu_galvatron_b200.models.spec import LayerCtx, ModelSpec

    T, k, E, H = 1024, 2, 8, 128
    spec = ModelSpec(family="llama", hidden=H, layers=1, heads=1, kv_heads=1, head_dim=128, ffn=128, vocab=512,
                     padded_vocab=512, seq_len=0, experts=E, moe_ffn=128, topk=k, dispatcher="allgather")
    m = GalvatronMoEMLP(spec, LayerCtx(ep=SimpleNamespace(size=4, rank=1)), DEV, "mlp")
    m.reset_parameters()
    g = torch.Generator().manual_seed(5)
    idx = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    local = torch.where((idx >= 2) & (idx < 4), idx - 2, -1)
    x, p = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV), torch.rand(T, k, generator=g).to(DEV)
    rows = []
    hook = m.experts.register_forward_pre_hook(lambda _, a: rows.append(a[0].shape[0]))
    with torch.no_grad():
        out = m._routed(x, p, local.to(DEV), local_only=True)
    hook.remove()
    assert rows == [placement(local, 2)[0][-1]]
    w1, w2 = (q.double() for q in (m.experts.linear_fc1.weight, m.experts.linear_fc2.weight))
    ref = torch.zeros(T, H, dtype=torch.float64, device=DEV)
    for e in range(2):
        a, b = (x.double() @ w1[e].t()).chunk(2, -1)
        ref += (torch.nn.functional.silu(a) * b) @ w2[e].t() * (p * (local.to(DEV) == e)).sum(1, keepdim=True)
    assert ((out.double() - ref).norm() / ref.norm()).item() < 1e-2      # four roundings to bf16
    _lib.assert_healthy()


@pytest.mark.parametrize("wrt", ["gradient", "weights", "rows"])
def test_gradients_of_the_gradients(wrt):
    """Second derivatives of dispatch and combine, against the same sums in 64 bits (the rows themselves are 16-bit)."""
    T, k, E, H = 40, 2, 4, 32
    g = torch.Generator().manual_seed(11)
    idx = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    idx[5, 1] = -1
    plan = _LocalPlan(idx.to(DEV), E)
    d, live = plan.dest.long().view(T, k).clamp(min=0), (plan.dest >= 0).view(T, k, 1)
    y, x, dout, dbuf = (torch.randn(n, H, generator=g).to(torch.bfloat16).to(DEV) for n in (plan.rows, T, T, plan.rows))
    w, vw, vx = torch.rand(T, k, generator=g).to(DEV), torch.randn(T, k, generator=g).to(DEV), torch.randn(T, H, generator=g).to(DEV)
    vy = torch.randn(plan.rows, H, generator=g).to(DEV)

    def combined(y, w, dout):                      # out and a functional of its gradients
        out = _LocalCombine.apply(y, w, plan) if y.dtype == torch.bfloat16 else ((y[d] * live) * w[..., None]).sum(1)
        gy, gw = torch.autograd.grad(out, (y, w), dout, create_graph=True)
        return (gy * vy.to(gy.dtype)).sum() + (gw * vw.to(gw.dtype)).sum()

    got, want = ([t.to(dt).requires_grad_() for t, dt in ((y, a), (w, b), (dout, a))]
                 for a, b in ((torch.bfloat16, torch.float32), (torch.float64, torch.float64)))
    at = {"rows": 0, "weights": 1, "gradient": 2}[wrt]
    res, ref = (torch.autograd.grad(combined(*t), t[at])[0] for t in (got, want))
    assert ((res.double() - ref).norm() / ref.norm()).item() < 2e-2            # vy and gy are rounded to 16 bits
    if wrt == "gradient":
        xs, gs = x.clone().requires_grad_(), dbuf.clone().requires_grad_()
        (gx,) = torch.autograd.grad(_LocalDispatch.apply(xs, plan), xs, gs, create_graph=True)
        (res,) = torch.autograd.grad((gx.float() * vx).sum(), gs)
        ref = torch.zeros(plan.rows, H, device=DEV)
        ref[d[live[..., 0]]] = vx[:, None].expand(T, k, H)[live[..., 0]]
        assert ((res.float() - ref).norm() / ref.norm()).item() < 1e-2
    _lib.assert_healthy()


def test_experts_that_do_not_exist_are_not_passed_over():
    T, k, E, H = 300, 2, 4, 64
    idx = torch.randint(0, E, (T, k), generator=torch.Generator().manual_seed(9))
    idx[7, 1], idx[250, 0], idx[3, 0] = E, 1 << 40, -1
    plan = _LocalPlan(idx.to(DEV), E)
    assert _lib.read_status(clear=True) == 6                            # bad argument
    out = _LocalCombine.apply(torch.ones(plan.rows, H, device=DEV, dtype=torch.bfloat16), torch.ones(T, k, device=DEV), plan)
    bad = torch.zeros(T, dtype=torch.bool, device=DEV)
    bad[[7, 250]] = True
    assert out[bad].isnan().all() and out[~bad].isfinite().all()
    _lib.assert_healthy()


def test_grouped_gemm_clears_the_rows_outside_its_segments():
    from hetu_galvatron_b200 import ops

    a = torch.randn(640, 64, device=DEV).to(torch.bfloat16)
    b = torch.randn(2, 72, 64, device=DEV).to(torch.bfloat16)
    junk = torch.full((640, 72), float("nan"), device=DEV, dtype=torch.bfloat16)
    del junk                                                            # the allocator hands these bytes out again
    out = ops.grouped_gemm(a, b, torch.tensor([128, 256, 512], device=DEV, dtype=torch.int32))
    assert (out[:128] == 0).all() and (out[512:] == 0).all()
    ref = torch.cat([a[128:256].double() @ b[0].double().t(), a[256:512].double() @ b[1].double().t()])
    assert ((out[128:512].double() - ref).norm() / ref.norm()).item() < 2.0 ** -8
    _lib.assert_healthy()


# segments that end inside a block of 32 rows, an empty one, one row, more than a pair tile; ragged columns (a block of C
# clipped at N) and a width that is no multiple of 16 bytes (no tensor map of C)
@pytest.mark.parametrize("seg", [[77, 0, 301, 150], [1, 255, 257, 31], [300]])
@pytest.mark.parametrize("N,K", [(264, 64), (512, 192), (260, 128)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("pair", ["0", "1"])
def test_grouped_gemm_of_ragged_segments(monkeypatch, seg, N, K, b_mn, pair):
    import importlib

    from hetu_galvatron_b200 import ops

    if b_mn and N % 8:
        pytest.skip("rows of an N-major operand are whole 16-byte groups")
    monkeypatch.setattr(importlib.import_module("hetu_galvatron_b200.ops.gemm"), "_PAIR_MODE", pair)
    g = torch.Generator(device=DEV).manual_seed(N + K + len(seg))
    first, rows = 5, 5 + sum(seg) + 40                          # rows before and after the segments belong to nobody
    starts = [first + sum(seg[:i]) for i in range(len(seg) + 1)]
    a = torch.randn(rows, K, device=DEV, generator=g).to(torch.bfloat16)
    b = torch.randn(len(seg), *((K, N) if b_mn else (N, K)), device=DEV, generator=g).to(torch.bfloat16)
    whole = torch.full((rows + 2, N), 3.0, device=DEV, dtype=torch.bfloat16)
    out = whole[1:rows + 1]
    row_start = torch.tensor(starts, device=DEV, dtype=torch.int32)
    ops.grouped_gemm(a, b, row_start, b_mn=b_mn, out=out)
    for i, n in enumerate(seg):
        ref = a[starts[i]:starts[i + 1]].double() @ (b[i].double() if b_mn else b[i].double().t())
        got = out[starts[i]:starts[i + 1]].double()
        assert torch.allclose(got, ref, rtol=2.0 ** -8, atol=1e-4 * K ** 0.5)   # one rounding; fp32 sums of K products
    junk = torch.full((rows, N), float("nan"), device=DEV, dtype=torch.bfloat16)
    del junk                                                    # the allocator hands these bytes out again
    fresh = ops.grouped_gemm(a, b, row_start, b_mn=b_mn)
    assert torch.equal(fresh[first:starts[-1]], out[first:starts[-1]])
    assert (fresh[:first] == 0).all() and (fresh[starts[-1]:] == 0).all()
    out[first:starts[-1]] = 3.0
    assert (whole == 3.0).all()
    _lib.assert_healthy()


# tiles along a group's rows: one of 64 rows and one row more, five tiles of unequal need, segments that start anywhere, columns that
# end inside a tile, a block and (odd: not turned) a pair, K that ends inside a block, by the rule and not by force
@pytest.mark.parametrize("seg", [[64, 65, 1, 0, 1100], [256, 257, 511]])
@pytest.mark.parametrize("N,K,b_mn", [(768, 1344, False), (1032, 1344, True), (330, 1288, False), (261, 1280, False)])
def test_grouped_gemm_along_the_rows(seg, N, K, b_mn):
    from hetu_galvatron_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(N + K + len(seg))
    first, rows = 3, 3 + sum(seg) + 9
    starts = [first + sum(seg[:i]) for i in range(len(seg) + 1)]
    a = torch.randn(rows, K, device=DEV, generator=g).to(torch.bfloat16)
    b = torch.randn(len(seg), *((K, N) if b_mn else (N, K)), device=DEV, generator=g).to(torch.bfloat16)
    whole = torch.full((rows, N + 3 + N % 2), 3.0, device=DEV, dtype=torch.bfloat16)
    out = whole[:, 2:N + 2]
    ops.grouped_gemm(a, b, torch.tensor(starts, device=DEV, dtype=torch.int32), b_mn=b_mn, out=out)
    for i in range(len(seg)):
        ref = a[starts[i]:starts[i + 1]].double() @ (b[i].double() if b_mn else b[i].double().t())
        assert torch.allclose(out[starts[i]:starts[i + 1]].double(), ref, rtol=2.0 ** -8, atol=1e-4 * K ** 0.5)
    out[first:starts[-1]] = 3.0
    assert (whole == 3.0).all()
    _lib.assert_healthy()


# more tiles along a group's rows than are walked together: one more, two groups of them and a last one of three; columns that end
# inside a tile, so that tiles whose order was wrong would be missing or done twice
@pytest.mark.parametrize("seg", [[2049, 70], [64, 4864, 0, 300]])
@pytest.mark.parametrize("N,K,b_mn", [(520, 1280, False), (768, 1344, True)])
def test_grouped_gemm_of_many_tiles_along_the_rows(seg, N, K, b_mn):
    from hetu_galvatron_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(N + sum(seg))
    starts = [sum(seg[:i]) for i in range(len(seg) + 1)]
    a = torch.randn(starts[-1], K, device=DEV, generator=g).to(torch.bfloat16)
    b = torch.randn(len(seg), *((K, N) if b_mn else (N, K)), device=DEV, generator=g).to(torch.bfloat16)
    out = torch.full((starts[-1], N), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.grouped_gemm(a, b, torch.tensor(starts, device=DEV, dtype=torch.int32), b_mn=b_mn, out=out)
    for i in range(len(seg)):
        ref = a[starts[i]:starts[i + 1]].double() @ (b[i].double() if b_mn else b[i].double().t())
        assert torch.allclose(out[starts[i]:starts[i + 1]].double(), ref, rtol=2.0 ** -8, atol=1e-4 * K ** 0.5)   # as above
    _lib.assert_healthy()
