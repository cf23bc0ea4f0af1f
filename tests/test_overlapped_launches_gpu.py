"""Kernels that may start before the one in front of them has ended: the same bits as with a wait after every operation."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.models.modules import ops_add
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV, LP = "cuda", torch.bfloat16


@pytest.mark.parametrize("rows,H,F", [(300, 256, 512), (2049, 1600, 6400)])
@pytest.mark.parametrize("rms", [True, False])
def test_operations_back_to_back(rows, H, F, rms):
    torch.manual_seed(rows)
    x, new = (torch.randn(rows, H, device=DEV).to(LP) for _ in range(2))
    ps = [torch.nn.Parameter(torch.randn(*s, device=DEV).to(LP) * 0.1) for s in ((H,), (H,), (F, H), (F,), (H, F), (H,))]

    def step(wait):
        pause = torch.cuda.synchronize if wait else (lambda: None)
        for p in ps:
            p.main_grad, p.mg_fresh, p.grad = torch.full(p.shape, 2.0, device=DEV), False, None
        a = torch.zeros_like(x)
        torch.cuda.synchronize()
        if not wait:
            torch.cuda._sleep(2000000)                # everything is queued before the first kernel runs
        a.copy_(new)                                  # written by the kernel in front
        a.requires_grad_()
        y, _ = ops.norm(a, ps[0], None if rms else ps[1], 1e-5, rms)
        pause()
        h = ops.linear(y, ps[2], ps[3])
        pause()
        h = ops.activation(h, "gelu")
        pause()
        out = ops.linear(h, ps[4], ps[5])
        pause()
        loss = ops.cross_entropy(out, torch.arange(rows, device=DEV) % H)
        loss.sum().backward()
        pause()
        return [out.detach().clone(), a.grad, *[p.main_grad for p in ps], *[p.grad for p in ps if p.grad is not None]]

    want = step(True)
    for _ in range(3):
        for s, t in zip(step(False), want, strict=True):
            assert torch.equal(s, t)
    _lib.assert_healthy()


# the norm's weight and bias are the results of a kernel that lets the next one start before it has written anything
@pytest.mark.parametrize("rows,H", [(1, 4096), (300, 256), (2049, 1600), (148, 16384)])
@pytest.mark.parametrize("rms", [True, False])
def test_norm_weights_written_by_the_kernel_in_front(rows, H, rms):
    torch.manual_seed(rows)
    x, (w1, w2) = torch.randn(rows, H, device=DEV).to(LP), torch.randn(2, H, device=DEV).to(LP)
    w = ops_add(w1, w2)
    want, _ = ops.norm(x, w, None if rms else w, 1e-5, rms)
    for _ in range(5):
        del w
        torch.zeros(H, device=DEV, dtype=LP)                               # the memory that the next result takes
        torch.cuda.synchronize()
        torch.cuda._sleep(500000)                                          # everything is queued before the first kernel runs
        w = ops_add(w1, w2)
        y, _ = ops.norm(x, w, None if rms else w, 1e-5, rms)
        assert torch.equal(y, want)
    _lib.assert_healthy()


# the tables are copied right in front of the kernels that rotate by them: inside the packed projection, and into a cache
@pytest.mark.parametrize("interleaved", [False, True])
def test_rotation_tables_written_in_front(interleaved):
    S, B, nh, ng, hd = 40, 2, 8, 2, 128
    torch.manual_seed(1)
    qkv = torch.randn(S * B, (nh + 2 * ng) * hd, device=DEV).to(LP)
    new = torch.randn(2, S, hd // 2, device=DEV)
    slots = torch.arange(ng * (nh // ng + 2), device=DEV, dtype=torch.int32)

    def run(wait):
        tables, caches = torch.zeros_like(new), torch.zeros(2, S, B, ng, hd, device=DEV, dtype=LP)
        mine, other = qkv.clone(), qkv.clone()
        torch.cuda.synchronize()
        if not wait:
            torch.cuda._sleep(500000)
        tables.copy_(new)
        if wait:
            torch.cuda.synchronize()
        out = ops.attention.cached_attention(mine, *caches, 0, 0, S, B, nh, ng, hd, *tables, interleaved)
        if not wait:
            torch.cuda._sleep(500000)
        tables.copy_(-new)
        if wait:
            torch.cuda.synchronize()
        ops.rope_packed(other, slots, hd, *tables, B, interleaved=interleaved)
        return out, caches, other

    for s, t in zip(run(False), run(True), strict=True):
        assert torch.equal(s, t)
    _lib.assert_healthy()


def test_a_refused_launch_leaves_no_error_behind():
    """More sequences than a grid has layers: the host refuses the launch, and the next call knows nothing of it."""
    q = torch.zeros(2, 65536, 1, 64, device=DEV, dtype=LP)
    x, y = torch.ones(64, device=DEV), torch.empty(64, device=DEV, dtype=LP)
    with pytest.raises(_lib.KernelError):
        ops.flash_attention(q, q, q, causal=False)
    assert _lib.load().hg_cast_f32_bf16(x.data_ptr(), y.data_ptr(), 64, _lib.stream()) == 0
    with pytest.raises(_lib.KernelError):
        ops.flash_attention(q, q, q, causal=False)
    assert torch.equal(x + 1, torch.full_like(x, 2.0)) and torch.equal(y.float(), x)
    _lib.assert_healthy()


# a product's weight, and then its bias, are the results of such a kernel: the CTA-pair and the few-row kernel
@pytest.mark.parametrize("rows,K,N", [(300, 512, 1000), (2049, 1600, 6400), (4, 4096, 4096)])
def test_weights_and_biases_written_by_the_kernel_in_front(rows, K, N):
    torch.manual_seed(rows)
    x, (w1, w2), (b1, b2) = (torch.randn(*s, device=DEV).to(LP) for s in ((rows, K), (2, N, K), (2, N)))
    w, b = ops_add(w1, w2), ops_add(b1, b2)
    want = ops.linear(x, w, b)
    for first in ("weight", "bias"):
        for _ in range(3):
            del w, b
            torch.zeros(N, K, device=DEV, dtype=LP), torch.zeros(N, device=DEV, dtype=LP)      # the memory of the next results
            torch.cuda.synchronize()
            torch.cuda._sleep(500000)
            if first == "weight":
                w, b = ops_add(w1, w2), ops_add(b1, b2)
            else:
                b, w = ops_add(b1, b2), ops_add(w1, w2)
            assert torch.equal(ops.linear(x, w, b), want)
    _lib.assert_healthy()
