"""The backward entry with fewer paths than SMs: no slower than the reverse pass of
a fused call."""
import importlib

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_tuner import fastest_ms  # noqa: E402


@pytest.mark.parametrize("W,D,B", [(6, 5, 8), (4, 6, 8), (5, 5, 100)])
def test_few_paths_backward(W, D, B):
    L, basis, st = 64, pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float64)
    x = torch.randn(B * L, W, dtype=torch.float64, device="cuda") * 0.1
    sig = torch.empty(B, basis.size(), dtype=torch.float64, device="cuda")
    seed, grad, fused = torch.rand_like(sig) * 2 - 1, torch.empty_like(x), torch.empty_like(x)

    def whole(schedule, **more):
        assert pkg.signature(st, None, x, basis, B, length=L, out=sig, schedule=schedule, **more)

    def backward():
        assert pkg.signature_backward(st, None, x, basis, B, sig, seed, grad, length=L)

    both = min(fastest_ms(lambda: whole(s, seed=seed, grad=fused), 5, 5) for s in (256, 512))
    forward = min(fastest_ms(lambda: whole(s), 5, 5) for s in (256, 512))
    alone = fastest_ms(backward, 5, 5)
    assert torch.allclose(grad, fused, rtol=1e-10, atol=1e-10)
    assert alone <= 1.05 * (both - forward), (alone, both, forward)
