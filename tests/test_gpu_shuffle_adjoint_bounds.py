"""The shuffle and half-shuffle adjoints coefficient by coefficient: each within
(its additions) x (unit roundoff) of the subset sums in FP64, over the same sum
of moduli -- a bound that stays far below the coefficients themselves."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_column import EPS, Rows, restrict, starts  # noqa: E402
from test_gpu_shuffle_letters import adjoint  # noqa: E402

# (depths from 6 on deal letters in both precisions, the others in FP32)
SHAPES = [(2, 4, 9), (2, 7, 5), (2, 10, 2), (3, 3, 40), (3, 6, 3), (4, 3, 30), (4, 4, 5), (4, 5, 2), (5, 4, 3),
          (6, 3, 7), (7, 3, 5), (8, 3, 5)]


@pytest.mark.parametrize("W,D,B", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_every_coefficient_within_its_own_bound(W, D, B, dtype):
    rng = np.random.default_rng(7 * W + D)
    st, basis, db = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D), starts(W, D)
    # a coefficient has at most dim terms, each a sum of interleavings formed in at
    # most D (D + 1) / 2 additions and multiplied twice; the reference's own
    # rounding, in FP64, is allowed for as much again
    additions = 2 * (int(db[-1]) + D * (D + 1) // 2 + 4)
    for ro, rx, ry in (((0, D), (0, D), (0, D)), ((0, D - 1), (1, D), (1, D - 1)), ((1, D), (0, 1), (0, D))):
        x, y = (Rows(rng, dtype, W, D, B, 3, 1) for _ in range(2))
        hx, hy = restrict(x.host(), W, D, rx), restrict(y.host(), W, D, ry)
        cases = [(lambda o: pkg.st_adj_mul(st, None, o, x.view(*rx), y.view(*ry), basis, B), 1.0, (False, False)),
                 (lambda o: pkg.left_hs_adj_lmul(st, None, o, x.view(*rx), y.view(*ry), basis, B, -0.5), -0.5,
                  (True, False)),
                 (lambda o: pkg.left_hs_adj_rmul(st, None, o, x.view(*rx), y.view(*ry), basis, B, -0.5), -0.5,
                  (True, True))]
        for call, beta, (half, first) in cases:
            a, b = (hy, hx) if first else (hx, hy)
            want = beta * adjoint(a, b, W, D, half, first)
            bound = abs(beta) * additions * EPS[dtype] * adjoint(abs(a), abs(b), W, D, half, first)
            out = Rows(rng, dtype, W, D, B, 3, 1)
            assert call(out.view(*ro))
            got = out.host()
            for m in range(ro[0], ro[1] + 1):
                at = slice(db[m], db[m + 1])
                assert (abs(got - want)[:, at] <= bound[:, at]).all(), (half, first, m)
                # zeros, or the wrong terms, could not pass
                assert bound[:, at].max() <= 0.1 * np.sqrt((want[:, at] ** 2).mean()), (half, first, m)
