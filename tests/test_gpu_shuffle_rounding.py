"""Rounding of the shuffle adjoints by letters (csrc/shuffle_letters.cu): no more
than that of the subset sums (csrc/shuffle.cu), which serve the same rows in a call
of less than one tensor an SM."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_shuffle_letters import adjoint  # noqa: E402

FEW = 48


def run(op, dtype, x, y, W, D):
    x, y = (torch.from_numpy(v).to("cuda", dtype) for v in (x, y))
    out, basis = torch.zeros_like(x), pkg.TensorBasis(W, D)
    tail = (basis, len(x)) if op == "st_adj_mul" else (basis, len(x), 1.0)
    views = (pkg.make_tensor_batch(t, t.shape[1], 0, D) for t in (out, x, y))
    assert getattr(pkg, op)(pkg.GB300Strategy(dtype), None, *views, *tail)
    return out[:FEW].cpu().numpy()


@pytest.mark.parametrize("op", ["st_adj_mul", "left_hs_adj_lmul", "left_hs_adj_rmul"])
@pytest.mark.parametrize("dtype,W,D", [(torch.float32, 4, 5), (torch.float32, 5, 4), (torch.float32, 6, 4),
                                       (torch.float32, 3, 6), (torch.float64, 3, 6)])
def test_many_tensors_round_no_more_than_few(op, dtype, W, D):
    rng = np.random.default_rng(10 * W + D)
    n = sum(W ** k for k in range(D + 1))
    x, y = (rng.uniform(-1, 1, (4096, n)).astype(np.float32) for _ in range(2))  # (exact in either precision)
    many, few = run(op, dtype, x, y, W, D), run(op, dtype, x[:FEW], y[:FEW], W, D)
    wide = np.float64 if dtype is torch.float32 else np.longdouble
    a, b = x[:FEW].astype(wide), y[:FEW].astype(wide)
    want = {"st_adj_mul": lambda: adjoint(a, b, W, D), "left_hs_adj_lmul": lambda: adjoint(a, b, W, D, True),
            "left_hs_adj_rmul": lambda: adjoint(b, a, W, D, True, True)}[op]()

    def rms(v):
        return float(np.sqrt(((v.astype(wide) - want) ** 2).mean()))

    # (35 000 coefficients and more: the ratio is known to about 1 %)
    assert rms(many) <= 1.05 * rms(few), (rms(many), rms(few))
