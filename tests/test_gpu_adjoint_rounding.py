"""Rounding of the adjoint multiplies (csrc/ft_adjoint.cu): per degree, no
more than a coefficient's terms dealt to the 256 threads of the general kernel
(csrc/ft_ops.cu) and summed pairwise, on the same inputs."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_column import starts  # noqa: E402

SHAPES = [(2, 5), (2, 9), (2, 11), (3, 4), (3, 6), (4, 3), (4, 5), (5, 3), (5, 5), (6, 4), (7, 3), (7, 4), (8, 3), (8, 4)]


def terms(op, arg, W, D, m, left):
    """The factors of every coefficient of degree m: [batch, coefficient, term]."""
    db, j = starts(W, D), np.arange(W ** m)[:, None]
    places = [db[m + p] + (np.arange(W ** p) * W ** m + j if left else j * W ** p + np.arange(W ** p))
              for p in range(D - m + 1)]
    return op[:, None, :db[D - m + 1]], arg[:, np.concatenate(places, 1)]


def dealt(x, y, W, D, m):
    """FP32: the terms dealt to as many threads as a coefficient gets of up to 256,
    each a chain of multiply-adds, and their sums added pairwise."""
    nt, threads = 32, 1
    while nt < 256 and nt < W ** D:
        nt *= 2
    while 2 * threads * W ** m <= nt:
        threads *= 2
    sums = []
    for r in range(threads):
        acc = np.zeros(y.shape[:2], np.float32)
        for k in range(r, y.shape[2], threads):  # (a product of two FP32 numbers is exact in FP64)
            acc = (x[..., k].astype(np.float64) * y[..., k] + acc).astype(np.float32)
        sums.append(acc)
    while len(sums) > 1:
        sums = [a + b for a, b in zip(sums[::2], sums[1::2])]
    return sums[0]


@pytest.mark.parametrize("W,D", SHAPES)
@pytest.mark.parametrize("left", [True, False])
def test_fp32_sums_round_no_more_than_the_dealt_ones(W, D, left):
    rng = np.random.default_rng(W * 10 + D)
    db = starts(W, D)
    B = 1000  # at least 1 000 sums a degree: their rms error is known to 1 / sqrt(2 000), 2.2 %
    op, arg = (rng.uniform(-1, 1, (B, db[-1])).astype(np.float32) for _ in range(2))
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float32)
    out = torch.empty(B, int(db[-1]), dtype=torch.float32, device="cuda")
    batch = lambda t: pkg.make_tensor_batch(t, basis.size(), 0, D)  # noqa: E731
    multiply = pkg.ft_adj_lmul if left else pkg.ft_adj_rmul
    assert multiply(st, None, batch(out), *(batch(torch.from_numpy(v).cuda()) for v in (op, arg)), basis, B)
    got = out.double().cpu().numpy()
    for m in range(D + 1):
        few = max(16, min(B, 2_000_000 // int(db[-1])), 1000 // W ** m)
        x, y = terms(op[:few], arg[:few], W, D, m, left)
        want = (x.astype(np.float64) * y).sum(-1)

        def rms(v):
            return np.sqrt(((v.astype(np.float64) - want) ** 2).mean())

        # the two orders' errors differ by up to 10 % by design, and four deviations
        # of the ratio of two measured values are 13 %
        ours, theirs = rms(got[:few, db[m]:db[m + 1]]), rms(dealt(x, y, W, D, m))
        assert ours <= 1.25 * theirs, (m, ours, theirs)


def dealt_fp64(x, y, W, D, m):
    """dealt() in FP64: each multiply-add formed in the wider type and rounded once."""
    nt, threads = 32, 1
    while nt < 256 and nt < W ** D:
        nt *= 2
    while 2 * threads * W ** m <= nt:
        threads *= 2
    sums = []
    for r in range(threads):
        acc = np.zeros(y.shape[:2])
        for k in range(r, y.shape[2], threads):
            acc = (x[..., k].astype(np.longdouble) * y[..., k] + acc).astype(np.float64)
        sums.append(acc)
    while len(sums) > 1:
        sums = [a + b for a, b in zip(sums[::2], sums[1::2])]
    return sums[0]


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 106, reason="needs products of FP64 numbers exactly")
@pytest.mark.parametrize("W,D", [(2, 5), (2, 8), (3, 5), (4, 5), (5, 4), (5, 5), (6, 4), (7, 3), (8, 3)])
@pytest.mark.parametrize("left", [True, False])
def test_fp64_sums_round_no_more_than_the_dealt_ones(W, D, left):
    rng = np.random.default_rng(W * 10 + D)
    db = starts(W, D)
    B = 1000
    op, arg = (rng.uniform(-1, 1, (B, db[-1])) for _ in range(2))
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float64)
    out = torch.empty(B, int(db[-1]), dtype=torch.float64, device="cuda")
    batch = lambda t: pkg.make_tensor_batch(t, basis.size(), 0, D)  # noqa: E731
    multiply = pkg.ft_adj_lmul if left else pkg.ft_adj_rmul
    assert multiply(st, None, batch(out), *(batch(torch.from_numpy(v).cuda()) for v in (op, arg)), basis, B)
    got = out.cpu().numpy()
    for m in range(D + 1):
        few = max(8, min(B, 100_000 // int(db[-1])), 1000 // W ** m)
        x, y = terms(op[:few], arg[:few], W, D, m, left)
        want = (x.astype(np.longdouble) * y).sum(-1)

        def rms(v):
            return float(np.sqrt(((v.astype(np.longdouble) - want) ** 2).mean()))

        # (the orders differ by up to 18 % by design, where a lane sums what 16 threads
        # or more did; four deviations of the ratio of two measured values are 13 %)
        ours, theirs = rms(got[:few, db[m]:db[m + 1]]), rms(dealt_fp64(x, y, W, D, m))
        assert ours <= 1.33 * theirs, (m, ours, theirs)
