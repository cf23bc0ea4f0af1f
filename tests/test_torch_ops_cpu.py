"""The C++ autograd nodes (csrc/host/torch_ops.cpp) as far as they run without a GPU: routes, refusals, callbacks."""
import importlib
import itertools

import pytest
import torch

from hetu_galvatron_b200.csrc import build
from hetu_galvatron_b200.ops.gemm import OUT_BF16, OUT_F32, OUT_F32_ACC


@pytest.fixture(scope="module")
def native():
    build.build_torch_ops()
    from hetu_galvatron_b200._lib import hg_torch_ops

    return hg_torch_ops


def test_products_take_the_route_of_the_python_rules(native):
    g = importlib.import_module("hetu_galvatron_b200.ops.gemm")
    sizes = [1, 64, 65, 128, 129, 255, 256, 4096, 4097, 8192, 8193, 65535 * 128, 65535 * 128 + 1]
    for mode, a_mn, M, N, K in itertools.product((OUT_BF16, OUT_F32, OUT_F32_ACC), (False, True), sizes[:8], sizes,
                                                 (64, 1535, 1536, 3071, 3072)):
        how = 2 if g._use_skinny(M, N, K, a_mn, mode, 0, None) else int(g._use_pair(M, N, None))
        assert native.gemm_route(M, N, K, a_mn, mode, -1, True) == how
    assert native.gemm_route(512, 512, 64, False, OUT_BF16, 0, True) == 0
    assert native.gemm_route(512, 512, 64, False, OUT_BF16, -1, False) == 0
    assert native.gemm_route(8, 8, 64, False, OUT_BF16, 1, True) == 1


def test_what_is_not_on_a_gpu_is_left_to_python(native):
    x, w = torch.randn(4, 8, dtype=torch.bfloat16), torch.randn(16, 8, dtype=torch.bfloat16)
    assert native.linear(x, w, None) is None and native.linear(x, None, None) is None
    assert native.norm(x, None, w[0], None, 1e-5, True) is None
    assert native.activation(x, 2) is None and native.add(x, x) is None


def test_callback_at_the_edge_of_a_unit(native):
    calls = []
    x = torch.randn(3, 4, requires_grad=True)
    y = native.boundary(x, lambda: calls.append(1))
    assert torch.equal(y, x) and not calls
    (y * 2).sum().backward()
    assert calls == [1] and torch.equal(x.grad, torch.full((3, 4), 2.0))

    def fails():
        raise KeyError("what the callback raises")

    with pytest.raises(KeyError):
        native.boundary(x, fails).sum().backward()
    with torch.no_grad():
        assert native.boundary(x, fails) is None
    assert native.boundary(x, 3) is None


def test_tracing_and_dispatch_modes_see_the_python_classes(native):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Nothing(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    x = torch.randn(2, requires_grad=True)
    with Nothing():
        assert native.boundary(x, lambda: None) is None
    seen = []
    torch.jit.trace(lambda t: (seen.append(native.boundary(t, lambda: None)), t * 2)[1], (torch.randn(2),), check_trace=False)
    assert seen == [None]
    torch.func.grad(lambda t: (seen.append(native.boundary(t, lambda: None)), t.sum())[1])(torch.randn(2))
    assert seen == [None, None]
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(torch.randn(2), torch.randn(2))
        assert native.boundary(d, lambda: None) is None
