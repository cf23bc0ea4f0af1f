"""AdamW and the squared norm over a list of buffers against the one-buffer kernels and 64-bit sums."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one buffer, a tiny one beside a large one, lengths that are no multiple of four, more buffers than one launch takes
@pytest.mark.parametrize("sizes", [[1], [3, 1_000_003], [64, 4096, 5, 70_000], [4 * i + i % 4 + 1 for i in range(100)]])
def test_list_step_equals_single_steps(sizes):
    g = torch.Generator(device=DEV).manual_seed(len(sizes))
    hp = dict(lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3)
    coef = torch.full((1,), 0.7, device=DEV)
    rows = []
    for n in sizes:
        p, gr, m = (torch.randn(n, device=DEV, generator=g) for _ in range(3))
        rows.append((p, gr, m, torch.rand(n, device=DEV, generator=g), p.to(torch.bfloat16)))
    want = [tuple(t.clone() for t in r) for r in rows]
    for r in want:
        ops.adamw_step(*r, gscale=coef * 0.5, **hp)
    ops.adamw_step_list(rows, gscale=coef, scale=0.5, **hp)
    # the same arithmetic; the last n mod 4 elements run through another kernel's code in the one-buffer form, where the
    # compiler may contract the three chained operations differently (a few units of 2^-24 of the operands, which are
    # below 8), and the 16-bit copy may then round the other way (2^-8)
    for r, w in zip(rows, want):
        for a, b in zip(r, w):
            low = a.dtype == torch.bfloat16
            assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -7 if low else 1e-6, atol=2e-6)
            n4 = a.numel() // 4 * 4
            assert torch.equal(a[:n4], b[:n4])

    out = torch.full((1,), 5.0, device=DEV)
    terms = [(r[1], 1.0 + i) for i, r in enumerate(rows)]
    ref = sum(c * x.double().pow(2).sum().item() for x, c in terms)
    ops.sumsq_list(terms, out)
    assert abs(out.item() - 5.0 - ref) < 1e-5 * (ref + 5.0)        # fp32 sums in a fixed order
    ops.sumsq_list(terms, out, accumulate=False)
    assert abs(out.item() - ref) < 1e-5 * ref
    shifted = torch.randn(1001, device=DEV, generator=g)[1:]      # not 16-byte aligned
    ops.sumsq_list([(shifted, 1.0)], out, accumulate=False)
    assert abs(out.item() - shifted.double().pow(2).sum().item()) < 1e-2
    _lib.assert_healthy()


def test_squared_norm_over_buffers_of_both_memories():
    """A term in host memory is summed there, as by the one-buffer function."""
    out = torch.full((1,), 5.0, device=DEV)
    a, b = torch.randn(1000), torch.randn(777)
    ops.sumsq_list([(a.to(DEV), 1.0), (b, 0.5)], out, accumulate=False)
    assert abs(out.item() / (a.double().square().sum() + 0.5 * b.double().square().sum()).item() - 1) < 1e-5
    _lib.assert_healthy()


class _TwiceTheNorm:
    """Replaced methods of a unit: a norm that counts twice, a step that only counts its calls."""

    steps = 0

    def grad_sumsq(self, out):
        for x, scale in self.norm_terms():
            ops.sumsq(x, out, accumulate=True, scale=2.0 * scale)

    def optimizer_step(self, *args, **kwargs):
        self.steps += 1


@pytest.mark.parametrize("device", ["cpu", DEV])
@pytest.mark.parametrize("by", ["class", "instance"])
def test_replaced_methods_of_a_unit_are_called(device, by):
    from hetu_galvatron_b200.parallel.zero import ShardedUnit
    from hetu_galvatron_b200.runtime.optimizer import ShardedAdamW

    units = []
    for own in (False, True):
        lin = torch.nn.Linear(64, 32, bias=False, device=device, dtype=torch.bfloat16)
        cls = type("Own", (_TwiceTheNorm, ShardedUnit), {}) if own and by == "class" else ShardedUnit
        u = cls(lin, "unit", None, 1)
        if own and by == "instance":
            u.steps = 0
            u.grad_sumsq = _TwiceTheNorm.grad_sumsq.__get__(u)
            u.optimizer_step = _TwiceTheNorm.optimizer_step.__get__(u)
        u.reload_master()
        u.main_grad.fill_(0.5)
        for p in u.params:
            p.mg_fresh = False
        units.append(u)
    before = [u.master.clone() for u in units]
    opt = ShardedAdamW(units, lr=1e-2, clip_grad=1.0)
    opt.step()
    assert abs(opt._norm.item() - (64 * 32 * 0.25 * 3) ** 0.5) < 1e-3
    assert not torch.equal(units[0].master, before[0]) and torch.equal(units[1].master, before[1]) and units[1].steps == 1
