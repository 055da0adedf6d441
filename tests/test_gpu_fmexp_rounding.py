"""Rounding of ft_fmexp in FP32 (csrc/ft_horner.cu): no more than the general
kernel's recursion (csrc/ft_device.cuh), restated in numpy, on the same inputs."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_column import product, starts  # noqa: E402


def fma(a, b, c):
    return (a.astype(np.float64) * b + c).astype(np.float32)  # (the product is exact in FP64)


def general(x, m, W, D):
    """o = M; then d = D .. 1: o = c_d M + o (x) X, c_d = D! / (d-1)!; then o / D!."""
    db, o, c = starts(W, D), m.copy(), np.float32(1)
    for d in range(D, 0, -1):
        c *= np.float32(d)
        new = np.empty_like(o)
        for n in range(D + 1):
            acc = np.zeros((len(o), W ** n), np.float32)
            for k in range(1, min(n, D - d + 1) + 1):
                left, right = o[:, db[n - k]:db[n - k + 1], None], x[:, None, db[k]:db[k + 1]]
                acc = fma(left, right, acc.reshape(len(o), W ** (n - k), W ** k)).reshape(len(o), -1)
            new[:, db[n]:db[n + 1]] = fma(c, m[:, db[n]:db[n + 1]], acc)
        o = new
    return o * (np.float32(1) / c)


@pytest.mark.parametrize("W,D", [(2, 7), (2, 8), (3, 6), (4, 5), (5, 4)])
def test_fp32_rounds_no_more_than_the_general_recursion(W, D):
    rng = np.random.default_rng(W * 10 + D)
    B, n = 1500, int(starts(W, D)[-1])
    x, m = rng.uniform(-0.3, 0.3, (B, n)).astype(np.float32), rng.uniform(-1, 1, (B, n)).astype(np.float32)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float32)
    out, mult, arg = (torch.from_numpy(v).cuda() for v in (np.zeros_like(m), m, x))
    assert pkg.ft_fmexp(st, None, *(pkg.make_tensor_batch(t, n, 0, D) for t in (out, mult, arg)), basis, B)
    few = 40
    x64, m64 = x[:few].astype(np.float64), m[:few].astype(np.float64)
    x64[:, 0] = 0
    want = m64.copy()
    for d in range(D, 0, -1):
        want = m64 + product(want, x64, W, D) / d

    def rms(v):
        return np.sqrt(((v.astype(np.float64) - want) ** 2).mean())

    ours, theirs = rms(out.cpu().numpy()[:few]), rms(general(x[:few], m[:few], W, D))
    # (10 000 coefficients and more: the ratio is known to about 1 %)
    assert ours <= 1.05 * theirs, (ours, theirs)
