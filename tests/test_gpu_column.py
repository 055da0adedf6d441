"""The compile-time-width per-operation kernels against plain numpy in FP64:
products a column of coefficients at a time (csrc/ft_column.cu) and the
degree-one exponential step (csrc/ft_chen.cu), at the edges of their tasks --
levels shorter than a column's first letters, partial last groups of tensors,
strided and unaligned rows, degree ranges, every in-place form."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")

EPS = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24}
SHAPES = [(2, 2, 9), (2, 3, 613), (2, 7, 40), (3, 1, 5), (3, 2, 613), (3, 5, 40), (4, 3, 1300), (4, 4, 613),
          (5, 2, 700), (5, 4, 33), (6, 3, 613), (7, 2, 33), (7, 4, 7), (8, 3, 330), (8, 1, 40), (6, 5, 3), (2, 12, 3)]


def starts(W, D):
    return np.concatenate([[0], np.cumsum([W ** n for n in range(D + 1)])])


def restrict(x, W, D, r):
    db, y = starts(W, D), np.zeros_like(x)
    if r[0] <= min(r[1], D):
        y[:, db[r[0]]:db[min(r[1], D) + 1]] = x[:, db[r[0]]:db[min(r[1], D) + 1]]
    return y


def product(x, y, W, D):
    db, out = starts(W, D), np.zeros_like(x)
    for n in range(D + 1):
        for k in range(n + 1):
            a, b = x[:, db[n - k]:db[n - k + 1]], y[:, db[k]:db[k + 1]]
            out[:, db[n]:db[n + 1]] += (a[:, :, None] * b[:, None, :]).reshape(len(x), -1)
    return out


class Rows:
    """A batch of tensors in a padded, offset buffer of sentinels."""

    def __init__(self, rng, dtype, W, D, B, pad, offset, scale=1.0):
        self.n, self.W, self.D, self.B = int(starts(W, D)[-1]), W, D, B
        self.stride, self.offset = self.n + pad, offset
        self.buf = torch.full((offset + B * self.stride,), 7.0, dtype=dtype, device="cuda")
        self.rows = self.buf[offset:].view(B, self.stride)[:, :self.n]
        self.rows.copy_(torch.from_numpy(rng.uniform(-scale, scale, (B, self.n))))

    def host(self):
        return self.rows.double().cpu().numpy()

    def view(self, lo=0, hi=None):
        return pkg.make_tensor_batch(self.buf, self.stride, lo, self.D if hi is None else hi, self.offset)


def check(got, before, want, W, D, r, tol):
    """`want` on the degrees r of the output, the old values elsewhere."""
    db = starts(W, D)
    lo, hi = db[r[0]], db[min(r[1], D) + 1]
    assert np.array_equal(got[:, :lo], before[:, :lo]) and np.array_equal(got[:, hi:], before[:, hi:])
    err = np.max(np.abs(got - want)[:, lo:hi])
    assert err <= tol, f"{err:.3e} > {tol:.3e}"


@pytest.mark.parametrize("W,D,B", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_products_in_columns(W, D, B, dtype):
    # D + 2 terms of at most 1 in modulus: D + 3 roundings of partial sums of
    # at most D + 2, and one of the result in the reference's rounding
    tol = 2 * (D + 4) * (D + 2) * EPS[dtype]
    rng = np.random.default_rng(100 * W + D)
    st, basis = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D)
    for pad, off in ((0, 0), (1, 1), (3, 2)):
        for ro, rl, rr, ra in (((0, D), (0, D), (0, D), (0, D)), ((0, D - 1), (1, D), (0, D), (1, D - 1)),
                               ((1, D), (0, D - 1), (1, 1), (0, 0)), ((D, D), (0, D), (D, D), (D, D))):
            if min(ro[1], rl[1], rr[1], ra[1]) < 0 or ro[0] > ro[1]:
                continue
            out, a, b, c = (Rows(rng, dtype, W, D, B, pad, off) for _ in range(4))
            ho, ha, hb, hc = (v.host() for v in (out, a, b, c))
            prod = product(restrict(hb, W, D, rl), restrict(hc, W, D, rr), W, D)
            assert pkg.ft_mul(st, None, out.view(*ro), b.view(*rl), c.view(*rr), basis, B)
            check(out.host(), ho, prod, W, D, ro, tol)
            before = out.host()
            assert pkg.ft_fma(st, None, out.view(*ro), a.view(*ra), b.view(*rl), c.view(*rr), basis, B, 0.5, -0.75)
            check(out.host(), before, 0.5 * restrict(ha, W, D, ra) - 0.75 * prod, W, D, ro, tol)
            # in place: a = alpha c + beta a (x) b, b (x) a, and a = alpha a + beta b (x) c
            for kind, rhs_first in ((1, False), (2, True), (0, None)):
                x = Rows(rng, dtype, W, D, B, pad, off)
                hx = x.host()
                rx, ry = restrict(hx, W, D, ro), restrict(hb, W, D, rl)
                if rhs_first is None:
                    want = 0.5 * hx - 0.75 * prod
                    third = c.view(*rr)
                else:
                    pr = product(ry, rx, W, D) if rhs_first else product(rx, ry, W, D)
                    want = 0.5 * restrict(hc, W, D, ra) - 0.75 * pr
                    third = c.view(*ra)
                assert pkg.ft_inplace_fma(kind, st, None, x.view(*ro), b.view(*rl), third, basis, B, 0.5, -0.75)
                check(x.host(), hx, want, W, D, ro, tol)
            assert torch.all(out.buf[:off] == 7) and torch.all(out.buf[off:].view(B, -1)[:, out.n:] == 7)


@pytest.mark.parametrize("W,D,B", SHAPES + [(6, 6, 2)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_degree_one_exponential_step(W, D, B, dtype):
    # M (x) exp(x) with |M| <= 1, |x_a| <= 1/2: every chain's partial values are
    # below e, formed by at most D multiply-adds of D rounded letters each
    tol = 3 * (2 * D + 4) * EPS[dtype]
    rng = np.random.default_rng(10 * W + D)
    st, basis, db = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D), starts(W, D)
    xs = torch.from_numpy(rng.uniform(-0.5, 0.5, (B, W + 3))).to("cuda", dtype)
    xb = pkg.make_tensor_batch(xs, W + 3, 1, 1, 1)  # letters in columns 2 .. W + 1
    hx = np.zeros((B, db[-1]))
    hx[:, 1:W + 1] = xs[:, 2:W + 2].double().cpu().numpy()
    e = np.zeros_like(hx)
    e[:, 0] = 1
    power = e.copy()
    for k in range(1, D + 1):
        power = product(power, hx, W, D) / k
        e += power
    for pad, off in ((0, 0), (1, 1), (3, 2)):
        for ro, rm in (((0, D), (0, D)), ((0, D), (1, D - 1)), ((1, D), (0, D)), ((0, D - 1), (0, D)), ((D, D), (0, D))):
            if ro[1] < 1:
                continue
            out, m = (Rows(rng, dtype, W, D, B, pad, off) for _ in range(2))
            ho = out.host()
            want = product(restrict(restrict(m.host(), W, D, rm), W, D, ro), e, W, D)
            assert pkg.ft_fmexp(st, None, out.view(*ro), m.view(*rm), xb, basis, B)
            check(out.host(), ho, want, W, D, ro, tol)
            before = out.host()
            assert pkg.ft_exp(st, None, out.view(*ro), xb, basis, B)
            check(out.host(), before, e if ro[0] == 0 else np.zeros_like(e), W, D, ro, tol)


def power_series(x, W, D, coefficient):
    """sum over k of coefficient(k) x^k, x without its degree 0."""
    u = x.copy()
    u[:, 0] = 0
    total, power = np.zeros_like(x), np.zeros_like(x)
    power[:, 0] = 1
    for k in range(D + 1):
        total += coefficient(k) * power
        power = product(power, u, W, D)
    return total


@pytest.mark.parametrize("W,D,B", SHAPES + [(2, 13, 2)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_horner_in_columns(W, D, B, dtype):
    # |x_w| <= 1/4: coefficients of exp and log sum the compositions of a word
    # of n letters, at most 2^(n-1) products, each below 4^-parts: below 2 in
    # sum; every round of D sums at most D + 1 terms
    tol = 4 * (D + 1) * (D + 2) * EPS[dtype]
    rng = np.random.default_rng(1000 * W + D)
    st, basis = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D)
    log_term = lambda k: 0.0 if k == 0 else (-1.0) ** (k + 1) / k  # noqa: E731
    exp_term = lambda k: 1.0 / float(np.prod(np.arange(1, k + 1, dtype=np.float64)))  # noqa: E731
    for pad, off in ((0, 0), (3, 1)):
        x, m = Rows(rng, dtype, W, D, B, pad, off, 0.25), Rows(rng, dtype, W, D, B, pad, off)
        for ro, rx, rm in (((0, D), (0, D), (0, D)), ((0, D - 1), (1, D), (1, D)), ((1, D), (2, D), (0, D - 1)),
                           ((0, 0), (0, D), (0, 0)), ((D, D), (0, D), (1, D))):
            if min(ro[1], rm[1]) < 0 or ro[0] > ro[1] or rx[0] > rx[1]:
                continue
            hx = restrict(x.host(), W, D, rx)
            exp, log = power_series(hx, W, D, exp_term), power_series(hx, W, D, log_term)
            zero = np.zeros_like(hx)
            want = {"ft_exp": exp if ro[0] == 0 else zero, "ft_log": log if ro[0] == 0 else zero}
            for name, value in want.items():
                out = Rows(rng, dtype, W, D, B, pad, off)
                before = out.host()
                assert getattr(pkg, name)(st, None, out.view(*ro), x.view(*rx), basis, B)
                check(out.host(), before, value, W, D, ro, tol)
            out = Rows(rng, dtype, W, D, B, pad, off)
            before = out.host()
            held = restrict(restrict(m.host(), W, D, rm), W, D, ro)
            assert pkg.ft_fmexp(st, None, out.view(*ro), m.view(*rm), x.view(*rx), basis, B)
            check(out.host(), before, product(held, exp, W, D), W, D, ro, tol * (D + 1))


@pytest.mark.parametrize("W,D", [(2, 5), (5, 3)])
@pytest.mark.parametrize("rx", [(2, 3), (0, 0)])
def test_exponent_without_degree_one_leaves_infinities_alone(W, D, rx):
    # degrees of the exponential without terms take no part: M (x) exp(X) keeps
    # M's degree 1 (and all of M where X has no terms), whatever its degree 0 holds
    rng = np.random.default_rng(W)
    st, basis, db = pkg.GB300Strategy(torch.float64), pkg.TensorBasis(W, D), starts(W, D)
    out, x, m = (Rows(rng, torch.float64, W, D, 2, 0, 0, 0.25) for _ in range(3))
    m.buf.view(2, -1)[:, 0] = float("inf")
    assert pkg.ft_fmexp(st, None, out.view(0, D), m.view(0, D), x.view(*rx), basis, 2)
    kept = int(db[2]) if rx[0] == 2 else int(db[-1])
    # (scaled by D! and back: a rounding a round)
    assert np.allclose(out.host()[:, :kept], m.host()[:, :kept], rtol=4 * D * EPS[torch.float64], atol=0)


def adjoint(p, a, W, D, left):
    """out[m] = sum over p of the op's degree p against the argument's degree m + p."""
    db, out = starts(W, D), np.zeros_like(a)
    for m in range(D + 1):
        for k in range(D - m + 1):
            op, arg = p[:, db[k]:db[k + 1]], a[:, db[m + k]:db[m + k + 1]]
            if left:
                part = (op[:, None, :] @ arg.reshape(len(a), W ** k, W ** m))[:, 0]
            else:
                part = (arg.reshape(len(a), W ** m, W ** k) @ op[:, :, None])[:, :, 0]
            out[:, db[m]:db[m + 1]] += part
    return out


@pytest.mark.parametrize("W,D,B", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_adjoints_in_columns(W, D, B, dtype):
    rng = np.random.default_rng(7 * W + D)
    st, basis = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D)
    n = int(starts(W, D)[-1])
    # sums of up to n terms of modulus at most 1, in any order: n roundings of
    # partial sums that grow as the square root of their number (times 4), or
    # linearly at worst for the few terms of small tensors
    tol = 4 * np.sqrt(n) * min(n, 4 * np.sqrt(n) + 16) * EPS[dtype]
    for pad, off in ((0, 0), (3, 1)):
        op, arg = (Rows(rng, dtype, W, D, B, pad, off) for _ in range(2))
        for ro, rp, ra in (((0, D), (0, D), (0, D)), ((0, D - 1), (1, D), (1, D - 1)), ((1, D), (0, 1), (0, D)),
                           ((0, D), (D, D), (1, D)), ((D, D), (0, 0), (0, D))):
            if min(ro[1], rp[1], ra[1]) < 0 or ro[0] > ro[1] or ra[0] > ra[1]:
                continue
            hp, ha = restrict(op.host(), W, D, rp), restrict(arg.host(), W, D, ra)
            for name, left in (("ft_adj_lmul", True), ("ft_adj_rmul", False)):
                out = Rows(rng, dtype, W, D, B, pad, off)
                before = out.host()
                assert getattr(pkg, name)(st, None, out.view(*ro), op.view(*rp), arg.view(*ra), basis, B)
                check(out.host(), before, adjoint(hp, ha, W, D, left), W, D, ro, tol)
