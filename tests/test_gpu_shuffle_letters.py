"""The shuffle and half-shuffle products and their adjoints a letter at a time
(csrc/shuffle_letters.cu) against the subset sums in numpy, FP64: strided and
unaligned rows, degree ranges, the in-place and fused forms, and outputs that
alias an operand (which take the general kernel)."""
import importlib
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_column import EPS, Rows, check, restrict, starts  # noqa: E402

SHAPES = [(2, 3, 5), (2, 6, 40), (2, 7, 3), (2, 10, 2), (3, 4, 40), (3, 5, 3), (4, 3, 600), (4, 4, 5), (5, 3, 33), (5, 4, 3), (6, 3, 7),
          (3, 6, 3), (7, 3, 3), (8, 3, 5)]


def splits(n, k, half=False):
    """Axis orders that gather a word's letters at k places (`half`: the first
    among them) in front, the others behind."""
    for places in itertools.combinations(range(n), k):
        if not half or 0 in places:
            yield list(places) + [i for i in range(n) if i not in places]


def shuffle(x, y, W, D, half=False):
    db, out = starts(W, D), np.zeros_like(x)
    for n in range(1 if half else 0, D + 1):
        for k in range(n + 1):
            both = (x[:, db[k]:db[k + 1], None] * y[:, None, db[n - k]:db[n - k + 1]]).reshape([len(x)] + [W] * n)
            for order in splits(n, k, half):
                back = np.argsort(order)
                out[:, db[n]:db[n + 1]] += both.transpose([0] + [i + 1 for i in back]).reshape(len(x), -1)
    return out


def adjoint(op, arg, W, D, half=False, first=False):
    """The gradient of <arg, op sh y> in y, or with `first` of <arg, x sh op> in x."""
    db, out = starts(W, D), np.zeros_like(arg)
    for n in range(1 if half else 0, D + 1):
        g = arg[:, db[n]:db[n + 1]].reshape([len(arg)] + [W] * n)
        for k in range(n + 1):
            for order in splits(n, k, half):
                m = g.transpose([0] + [i + 1 for i in order]).reshape(len(arg), W ** k, W ** (n - k))
                if first:
                    out[:, db[k]:db[k + 1]] += (m @ op[:, db[n - k]:db[n - k + 1], None])[:, :, 0]
                else:
                    out[:, db[n - k]:db[n - k + 1]] += (op[:, None, db[k]:db[k + 1]] @ m)[:, 0]
    return out


@pytest.mark.parametrize("W,D,B", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_products_and_adjoint_by_letters(W, D, B, dtype):
    rng = np.random.default_rng(31 * W + D)
    st, basis = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D)
    n = int(starts(W, D)[-1])
    # products: 2^D terms of modulus at most 1, summed in D (D + 1) / 2 levels of
    # additions; adjoint: sums of up to (2 W)^D terms in as many levels and n more
    tol = 4 * (D * (D + 1) // 2 + 4) * 2.0 ** D * EPS[dtype]
    tol_adjoint = tol * 4 * np.sqrt(n) * np.sqrt(n)
    for pad, off in ((0, 0), (3, 1)):
        x, y, a = (Rows(rng, dtype, W, D, B, pad, off) for _ in range(3))
        for ro, rx, ry in (((0, D), (0, D), (0, D)), ((0, D - 1), (1, D), (1, D - 1)), ((2, D), (0, 1), (0, D)),
                           ((D, D), (0, 0), (0, D)), ((0, D), (D, D), (1, D))):
            hx, hy, ha = restrict(x.host(), W, D, rx), restrict(y.host(), W, D, ry), a.host()
            out = Rows(rng, dtype, W, D, B, pad, off)
            before = out.host()
            want = shuffle(hx, hy, W, D)
            assert pkg.st_mul(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B)
            check(out.host(), before, want, W, D, ro, tol)
            assert pkg.st_fma(st, None, out.view(*ro), a.view(*rx), x.view(*rx), y.view(*ry), basis, B, 0.5, -0.75)
            check(out.host(), before, 0.5 * restrict(ha, W, D, rx) - 0.75 * want, W, D, ro, tol)
            out = Rows(rng, dtype, W, D, B, pad, off)
            before = out.host()
            assert pkg.st_inplace_fma(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B, 0.5, -0.75)
            check(out.host(), before, 0.5 * before - 0.75 * want, W, D, ro, tol)
            out = Rows(rng, dtype, W, D, B, pad, off)
            before = out.host()
            assert pkg.st_adj_mul(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B)
            check(out.host(), before, adjoint(hx, hy, W, D), W, D, ro, tol_adjoint)
            before = out.host()
            assert pkg.left_hs_mul(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B, -0.5)
            check(out.host(), before, -0.5 * shuffle(hx, hy, W, D, True), W, D, ro, tol)
            before = out.host()
            assert pkg.left_hs_adj_lmul(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B, -0.5)
            check(out.host(), before, -0.5 * adjoint(hx, hy, W, D, True), W, D, ro, tol_adjoint)
            before = out.host()
            assert pkg.left_hs_adj_rmul(st, None, out.view(*ro), x.view(*rx), y.view(*ry), basis, B, -0.5)
            check(out.host(), before, -0.5 * adjoint(hy, hx, W, D, True, True), W, D, ro, tol_adjoint)
        # the result over an operand
        want = shuffle(x.host(), y.host(), W, D)
        assert pkg.st_mul(st, None, x.view(), x.view(), y.view(), basis, B)
        check(x.host(), x.host(), want, W, D, (0, D), tol)
