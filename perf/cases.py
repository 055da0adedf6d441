"""What the framework is timed on: the calls a user's program makes, through the
package's public entry points, over the sizes in which they are used.

Every case is one pass of one kind of work:

* ``mul``       ft_mul: products of batches of tensors (concatenating paths).
* ``mul_grad``  ft_mul with the gradients of both factors (ft_adj_lmul,
                ft_adj_rmul): one training step through a tensor product.
* ``stream``    ft_fmexp with degree-one exponents: the running signatures of a
                batch of streams take one new increment each.
* ``sig``       signatures of whole paths (inference), equal or uneven lengths.
* ``sig_grad``  signatures and the gradient of a linear loss (a training step).
* ``logsig``    log-signatures: the signature, then tensor_log_to_lie.
* ``lie_step``  lie_to_tensor_exp with a multiplier: one log-ODE step.
* ``shuffle``   st_mul and st_adj_mul: the shuffle product and its gradient.
* ``half``      left_hs_mul and both its adjoints (iterated integrals).

Signature calls run as a program that has not tuned them calls them.
"""
import functools
import importlib
import itertools
import math

import numpy as np
import torch

pkg = importlib.import_module("rough-path-primitives_gb300")

DTYPES = {"f64": torch.float64, "f32": torch.float32}


def listed():
    return [
        # one small batch of products: the least that a program sends in one call
        dict(name="mul_w4d4_b1024_f64", kind="mul", w=4, d=4, b=1024, t="f64"),
        # a product layer in training, in the precision that training uses
        dict(name="mul_grad_w5d5_b4096_f32", kind="mul_grad", w=5, d=5, b=4096, t="f32"),
        # an online feature store: many streams, one tick each
        dict(name="stream_w3d6_b3000_f32", kind="stream", w=3, d=6, b=3000, t="f32"),
        # a training step at the size that the project's headline figure is quoted on
        dict(name="sig_grad_w5d5_l256_b4096_f64", kind="sig_grad", w=5, d=5, l=256, b=4096, t="f64"),
        # a training step of an ordinary model: six channels, a hundred ticks, FP32
        dict(name="sig_grad_w6d5_l100_b1000_f32", kind="sig_grad", w=6, d=5, l=100, b=1000, t="f32"),
        # feature extraction from recordings of very uneven length
        dict(name="sig_uneven_w8d4_l2048_b10000_f32", kind="sig", w=8, d=4, l=2048, b=10000, uneven=True, t="f32"),
        # a handful of long recordings: few paths, many increments
        dict(name="sig_grad_w3d5_l1000_b4_f64", kind="sig_grad", w=3, d=5, l=1000, b=4, t="f64"),
        # log-signature features of a data set
        dict(name="logsig_w5d5_l256_b4096_f64", kind="logsig", w=5, d=5, l=256, b=4096, t="f64"),
        # two channels taken deep
        dict(name="sig_grad_w2d12_l64_b2048_f64", kind="sig_grad", w=2, d=12, l=64, b=2048, t="f64"),
        # the largest state: a tensor that does not fit one SM
        dict(name="sig_grad_w6d6_l128_b512_f64", kind="sig_grad", w=6, d=6, l=128, b=512, t="f64"),
        # one log-ODE step of a batch of solutions
        dict(name="lie_step_w5d5_b4096_f64", kind="lie_step", w=5, d=5, b=4096, t="f64"),
        # products of linear functionals, and their gradient
        dict(name="shuffle_w5d5_b4096_f64", kind="shuffle", w=5, d=5, b=4096, t="f64"),
    ]


# the work that no drawn case exceeds (that of the headline training step)
MAX_FLOPS, MAX_BYTES = 39e9, 3e8


def draw(rng):
    kind = rng.choice(["mul", "mul_grad", "stream", "sig", "sig", "sig_grad", "sig_grad", "sig_grad", "logsig",
                       "lie_step", "shuffle", "half"])
    t = rng.choice(["f64", "f32"])
    w = rng.choice([2, 3, 4, 5, 6, 7, 8])
    # the deepest tensors that a width is used with: at most about 10^4
    # coefficients (5000 where the cost grows with 2^depth or with the Lie basis)
    limit = 5000 if kind in ("shuffle", "half", "logsig", "lie_step") else 10000
    deepest = max(d for d in range(2, 13) if dim(w, d) <= limit)
    d = rng.randint(2, deepest)
    c = dict(kind=kind, w=w, d=d, t=t)

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind in ("sig", "sig_grad", "logsig"):
        c["l"] = spread(16, 2048 if d <= 6 else 256)
        c["b"] = spread(1, 10000)
        if kind == "sig":
            c["uneven"] = rng.random() < 0.5
    else:
        c["b"] = spread(16, 10000)
    while work(c)["flops"] > MAX_FLOPS or work(c)["bytes"] > MAX_BYTES:
        c["b"] = max(1, int(c["b"] * 0.7))
    return c


# ---------------------------------------------------------------------------
# Sizes and work.
# ---------------------------------------------------------------------------

def dim(w, d):
    return sum(w ** n for n in range(d + 1))


def uneven_lengths(l, b):
    """Lengths spread evenly over [16, l] (the seed decides which path has which)."""
    return np.linspace(min(16, l), l, b).round().astype(np.int64)


@functools.lru_cache(maxsize=None)
def lie_count(w, d):
    return sum(sum(mobius(n // k) * w ** k for k in range(1, n + 1) if n % k == 0) // n for n in range(1, d + 1))


def mobius(n):
    r, p = 1, 2
    while n > 1:
        if n % p == 0:
            n //= p
            if n % p == 0:
                return 0
            r = -r
        p += 1
    return r


@functools.lru_cache(maxsize=None)
def conversion_entries(w, d):
    """Non-zeros of the Lie-to-tensor matrix."""
    return sum(int((h != 0).sum()) for level in hall_tensors(w, d)[1:] for h in level)


def work(case):
    """Bytes: each input read once, each output written once.  Flops: two per
    multiply-add of the truncated products (Horner's chains where the exponent
    is of degree one)."""
    w, d, b, kind = case["w"], case["d"], case["b"], case["kind"]
    size = 8 if case["t"] == "f64" else 4
    n_tensor, n_lie = dim(w, d), lie_count(w, d)
    product = sum((n + 1) * w ** n for n in range(d + 1))
    step = sum((d - i + 1) * w ** i for i in range(1, d + 1))  # one degree-one exponential
    if kind in ("sig", "sig_grad", "logsig"):
        ticks = int(uneven_lengths(case["l"], b).sum()) if case.get("uneven") else case["l"] * b
        if kind == "sig_grad":  # the chains forward, and transposed
            return {"bytes": size * (2 * ticks * w + 2 * b * n_tensor), "flops": 8.0 * ticks * step}
        out = b * n_tensor
        flops = 2.0 * ticks * step
        if kind == "logsig":
            out += b * n_lie
            flops += 2.0 * b * (log_terms(w, d) + conversion_entries(w, d))
        return {"bytes": size * (ticks * w + out), "flops": flops}
    if kind == "mul":
        return {"bytes": size * 3 * b * n_tensor, "flops": 2.0 * b * product}
    if kind == "mul_grad":
        return {"bytes": size * 6 * b * n_tensor, "flops": 6.0 * b * product}
    if kind == "stream":
        return {"bytes": size * b * (2 * n_tensor + w), "flops": 2.0 * b * step}
    if kind == "lie_step":
        return {"bytes": size * b * (2 * n_tensor + n_lie),
                "flops": 2.0 * b * (log_terms(w, d) + conversion_entries(w, d))}
    terms = sum((2 * w) ** n for n in range(d + 1))
    if kind == "shuffle":
        return {"bytes": size * 5 * b * n_tensor, "flops": 4.0 * b * terms}
    return {"bytes": size * 6 * b * n_tensor, "flops": 3.0 * b * terms}


def log_terms(w, d):
    """Multiply-adds of a logarithm or exponential by Horner's rule."""
    return sum(sum(k * w ** k for k in range(1, m + 1)) for m in range(1, d + 1))


# ---------------------------------------------------------------------------
# Inputs, and one pass.
# ---------------------------------------------------------------------------

class Inputs:
    """Random inputs on the GPU, from the seed alone."""

    def __init__(self, case, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.t = DTYPES[case["t"]]
        self.case, self.seed = case, seed

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.gen, device="cuda", dtype=self.t) * 2 - 1

    def normal(self, *shape):
        return torch.randn(shape, generator=self.gen, device="cuda", dtype=self.t)

    def paths(self):
        """(increments, offsets or None): each path's increments have variance 1 / length."""
        c = self.case
        if not c.get("uneven"):
            return self.normal(c["b"] * c["l"], c["w"]) / math.sqrt(c["l"]), None
        lengths = np.random.default_rng(self.seed).permutation(uneven_lengths(c["l"], c["b"]))
        offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)])).cuda()
        scale = torch.from_numpy(lengths).cuda().to(self.t).rsqrt()
        scale = torch.repeat_interleave(scale, torch.from_numpy(lengths).cuda())
        return self.normal(int(offsets[-1]), c["w"]) * scale[:, None], offsets

    def signatures(self):
        """Signatures of paths of three increments (a tensor such as programs hold)."""
        c = self.case
        s = unit(c["w"], c["d"], c["b"])
        for x in self.normal(3, c["b"], c["w"]).double() / math.sqrt(3):
            s = chen_step(s, x)
        return torch.cat(s, 1).to(self.t)


@functools.lru_cache(maxsize=None)
def tools(w, d):
    """The basis, Lie basis and conversion matrices that a program makes once."""
    lie = pkg.LieBasis(w, d)
    return pkg.TensorBasis(w, d), lie, pkg.make_t2l_matrix(lie), pkg.make_l2t_matrix(lie)


def prepare(case, seed):
    w, d, b, kind = case["w"], case["d"], case["b"], case["kind"]
    make = Inputs(case, seed)
    n = dim(w, d)

    def empty(*shape):
        return torch.empty(*shape, dtype=make.t, device="cuda")

    def tensors(data, lo=0, hi=d, stride=n, offset=0):
        return pkg.make_tensor_batch(data, stride, lo, hi, offset)

    s = dict(kind=kind, b=b, strategy=pkg.GB300Strategy(make.t, 0))
    if kind in ("logsig", "lie_step"):
        s["basis"], s["lie_basis"], s["t2l"], s["l2t"] = tools(w, d)
    else:
        s["basis"] = tensor_basis(w, d)
    if kind in ("sig", "sig_grad", "logsig"):
        s["increments"], offsets = make.paths()
        s["where"] = {"length": case["l"]} if offsets is None else {"offsets": offsets}
        s["sig"] = empty(b, n)
        if kind == "sig_grad":
            s["seed"], s["grad"] = make.uniform(b, n), torch.empty_like(s["increments"])
        if kind == "logsig":
            slots = 1 + lie_count(w, d)  # slot 0 of a Lie vector is unused
            s["lie"] = empty(b, slots).zero_()
            s["sig_view"] = tensors(s["sig"])
            s["lie_view"] = pkg.make_lie_batch(s["lie"], slots, 1, d)
        return s
    s["out"] = empty(b, n)
    if kind == "stream":
        s["inputs"] = (make.signatures(), make.normal(b, w) / 16)
        s["views"] = (tensors(s["out"]), tensors(s["inputs"][0]), tensors(s["inputs"][1], 1, 1, w, -1))
        return s
    if kind == "lie_step":
        slots = 1 + lie_count(w, d)
        s["inputs"] = (make.signatures(), make.normal(b, slots) / 16)
        s["views"] = (tensors(s["out"]), tensors(s["inputs"][0]), pkg.make_lie_batch(s["inputs"][1], slots, 1, d))
        return s
    s["inputs"] = (make.uniform(b, n), make.uniform(b, n))
    s["outputs"] = [s["out"]]
    if kind in ("mul_grad", "half"):
        s["inputs"] += (make.uniform(b, n),)
        s["outputs"] += [empty(b, n), empty(b, n)]
    elif kind == "shuffle":
        s["inputs"] += (make.uniform(b, n),)
        s["outputs"] += [empty(b, n)]
    s["views"] = [tensors(x) for x in s["outputs"]] + [tensors(x) for x in s["inputs"]]
    return s


@functools.lru_cache(maxsize=None)
def tensor_basis(w, d):
    return pkg.TensorBasis(w, d)


def run(s):
    kind, st, basis, b = s["kind"], s["strategy"], s["basis"], s["b"]
    if kind == "mul":
        out, x, y = s["views"]
        pkg.ft_mul(st, None, out, x, y, basis, b).raise_if_failed()
        return s["out"]
    if kind == "mul_grad":
        out, gx, gy, x, y, g = s["views"]
        pkg.ft_mul(st, None, out, x, y, basis, b).raise_if_failed()
        pkg.ft_adj_rmul(st, None, gx, y, g, basis, b).raise_if_failed()
        pkg.ft_adj_lmul(st, None, gy, x, g, basis, b).raise_if_failed()
        return s["outputs"]
    if kind == "stream":
        out, m, x = s["views"]
        pkg.ft_fmexp(st, None, out, m, x, basis, b).raise_if_failed()
        return s["out"]
    if kind == "sig":
        pkg.signature(st, None, s["increments"], basis, b, out=s["sig"], **s["where"]).raise_if_failed()
        return s["sig"]
    if kind == "sig_grad":
        pkg.signature(st, None, s["increments"], basis, b, out=s["sig"], seed=s["seed"], grad=s["grad"],
                      **s["where"]).raise_if_failed()
        return s["sig"], s["grad"]
    if kind == "logsig":
        pkg.signature(st, None, s["increments"], basis, b, out=s["sig"], **s["where"]).raise_if_failed()
        pkg.tensor_log_to_lie(st, None, s["lie_view"], s["sig_view"], s["lie_basis"], basis, b,
                              s["t2l"]).raise_if_failed()
        return s["sig"], s["lie"]
    if kind == "lie_step":
        out, m, x = s["views"]
        pkg.lie_to_tensor_exp(st, None, out, m, x, basis, s["lie_basis"], b, s["l2t"]).raise_if_failed()
        return s["out"]
    if kind == "shuffle":
        out, gy, x, y, g = s["views"]
        pkg.st_mul(st, None, out, x, y, basis, b).raise_if_failed()
        pkg.st_adj_mul(st, None, gy, x, g, basis, b).raise_if_failed()
        return s["outputs"]
    out, gy, gx, x, y, g = s["views"]
    pkg.left_hs_mul(st, None, out, x, y, basis, b).raise_if_failed()
    pkg.left_hs_adj_lmul(st, None, gy, x, g, basis, b).raise_if_failed()
    pkg.left_hs_adj_rmul(st, None, gx, g, y, basis, b).raise_if_failed()
    return s["outputs"]


# ---------------------------------------------------------------------------
# The same results in plain torch, FP64: a tensor is the list of its levels,
# level n of shape [batch, w^n].
# ---------------------------------------------------------------------------

def unit(w, d, b):
    return [torch.ones(b, 1, dtype=torch.float64, device="cuda")] + [
        torch.zeros(b, w ** n, dtype=torch.float64, device="cuda") for n in range(1, d + 1)]


def levels(x, w, d):
    return list(torch.split(x.double(), [w ** n for n in range(d + 1)], 1))


def outer(x, y):
    return (x[:, :, None] * y[:, None, :]).reshape(len(x), -1)


def product(x, y):
    return [sum(outer(x[n - k], y[k]) for k in range(n + 1)) for n in range(len(x))]


def chen_step(s, x):
    """s (x) exp(x) for a degree-one x."""
    out = [s[0]]
    for n in range(1, len(s)):
        t = s[0]
        for j in range(1, n + 1):
            t = s[j] + outer(t, x / (n - j + 1))
        out.append(t)
    return out


def signatures(incr, w, d):
    """incr [paths, length, w]"""
    s = unit(w, d, len(incr))
    for k in range(incr.shape[1]):
        s = chen_step(s, incr[:, k])
    return s


def logarithm(x):
    """log(1 + u), u the part of degree >= 1: sum of (-1)^{k+1} u^k / k."""
    d = len(x) - 1
    u = [torch.zeros_like(x[0])] + list(x[1:])
    power, total = u, u
    for k in range(2, d + 1):
        power = product(power, u)
        total = [a + b * ((-1) ** (k + 1) / k) for a, b in zip(total, power)]
    return total


def exponential(u):
    d = len(u) - 1
    power = [torch.ones_like(u[0])] + [torch.zeros_like(v) for v in u[1:]]
    total = power
    for k in range(1, d + 1):
        power = [v / k for v in product(power, u)]
        total = [a + b for a, b in zip(total, power)]
    return total


@functools.lru_cache(maxsize=None)
def hall_tensors(w, d):
    """Per degree, the Hall basis elements as tensors (integer arrays of length
    w^degree): letters, then commutators [p, q] with p < q and q's left
    factor at most p, by degree of p, then p, then q."""
    found, parents = [[], [np.eye(w, dtype=np.int64)[i] for i in range(w)]], [None] + [(0, i + 1) for i in range(w)]
    degree, tensor = [0] + [1] * w, [None] + found[1][:]
    for n in range(2, d + 1):
        level = []
        for m in range(1, n // 2 + 1):
            for p in range(1, len(degree)):
                if degree[p] != m:
                    continue
                for q in range(p + 1, len(degree)):
                    if degree[q] != n - m or parents[q][0] > p:
                        continue
                    level.append(((p, q), np.outer(tensor[p], tensor[q]).ravel()
                                  - np.outer(tensor[q], tensor[p]).ravel()))
        for pair, x in level:
            parents.append(pair)
            degree.append(n)
            tensor.append(x)
        found.append([x for _, x in level])
    return found


def lie_coefficients(x, w, d):
    """Hall coefficients of the Lie element x, degree by degree."""
    out = [torch.zeros_like(x[0])]  # the unused slot
    for n in range(1, d + 1):
        basis = torch.from_numpy(np.stack(hall_tensors(w, d)[n]).astype(np.float64)).cuda()  # [elements, w^n]
        # coefficients c with c @ basis = x
        out.append(torch.linalg.solve(basis @ basis.T, basis @ x[n].T).T)
    return torch.cat(out, 1)


def shuffles(n, k, fixed=0):
    """Where the first factor's k letters sit among n: `fixed` of them in front."""
    for rest in itertools.combinations(range(fixed, n), k - fixed):
        yield tuple(range(fixed)) + rest


def axes(n, places):
    """Permutation that takes (first factor's letters, second's) to their places in a word of n letters."""
    order = list(places) + [i for i in range(n) if i not in places]
    inverse = [0] * n
    for i, p in enumerate(order):
        inverse[p] = i
    return [0] + [i + 1 for i in inverse], [0] + [p + 1 for p in order]


def shuffle_product(x, y, w, half):
    """x sh y, or with `half` the part whose first letter comes from x."""
    b, out = len(x[0]), []
    for n in range(len(x)):
        total = torch.zeros(b, w ** n, dtype=torch.float64, device="cuda")
        for k in range(1 if half else 0, n + 1):
            both = outer(x[k], y[n - k]).reshape([b] + [w] * n)
            for places in shuffles(n, k, 1 if half else 0):
                total = total + both.permute(axes(n, places)[0]).reshape(b, -1)
        out.append(total)
    return out


def shuffle_adjoint(fixed, g, w, half, first):
    """The gradient of <g, x sh y> in y (x = `fixed`), or with `first` in x (y = `fixed`)."""
    b, d = len(g[0]), len(g) - 1
    out = [torch.zeros(b, w ** n, dtype=torch.float64, device="cuda") for n in range(d + 1)]
    for n in range(d + 1):
        gn = g[n].reshape([b] + [w] * n)
        for k in range(1 if half else 0, n + 1):
            both = torch.zeros(b, w ** k, w ** (n - k), dtype=torch.float64, device="cuda")
            for places in shuffles(n, k, 1 if half else 0):
                both = both + gn.permute(axes(n, places)[1]).reshape(b, w ** k, w ** (n - k))
            if first:
                out[k] = out[k] + (both @ fixed[n - k][:, :, None])[:, :, 0]
            else:
                out[n - k] = out[n - k] + (fixed[k][:, None, :] @ both)[:, 0]
    return out


def by_chunks(f, limit, *arrays):
    """f over slices of at most `limit` batch entries, outputs joined."""
    got = [f(*(a[i:i + limit] for a in arrays)) for i in range(0, len(arrays[0]), limit)]
    return [torch.cat(v) for v in zip(*got)]


def exact(case, seed):
    w, d, b, kind = case["w"], case["d"], case["b"], case["kind"]
    make = Inputs(case, seed)
    n = dim(w, d)
    if kind in ("sig", "sig_grad", "logsig"):
        return exact_paths(case, make)
    if kind in ("stream", "lie_step"):
        m = make.signatures()
        if kind == "stream":
            x = make.normal(b, w) / 16
            return torch.cat(chen_step(levels(m, w, d), x.double()), 1)
        lie = make.normal(b, 1 + lie_count(w, d)) / 16

        def step(m, lie):
            x, at = [torch.zeros(len(m), 1, dtype=torch.float64, device="cuda")], 1
            for k in range(1, d + 1):
                basis = torch.from_numpy(np.stack(hall_tensors(w, d)[k]).astype(np.float64)).cuda()
                x.append(lie[:, at:at + len(basis)].double() @ basis)
                at += len(basis)
            return [torch.cat(product(levels(m, w, d), exponential(x)), 1)]

        return by_chunks(step, 1024, m, lie)[0]
    x, y = make.uniform(b, n), make.uniform(b, n)
    if kind == "mul":
        return torch.cat(product(levels(x, w, d), levels(y, w, d)), 1)
    g = make.uniform(b, n)

    def product_and_gradients(x, y, g):
        lx, ly, lg = (levels(v, w, d) for v in (x, y, g))
        gx, gy = ([torch.zeros_like(v) for v in lx] for _ in range(2))
        for i in range(d + 1):
            for k in range(i + 1):  # level i of the product: x[i - k], y[k]
                m = lg[i].reshape(len(x), w ** (i - k), w ** k)
                gx[i - k] += (m @ ly[k][:, :, None])[:, :, 0]
                gy[k] += (lx[i - k][:, None, :] @ m)[:, 0]
        return [torch.cat(v, 1) for v in (product(lx, ly), gx, gy)]

    def shuffles_and_gradient(x, y, g):
        lx, ly, lg = (levels(v, w, d) for v in (x, y, g))
        return [torch.cat(v, 1) for v in (shuffle_product(lx, ly, w, False),
                                          shuffle_adjoint(lx, lg, w, False, False))]

    def halves_and_gradients(x, y, g):
        lx, ly, lg = (levels(v, w, d) for v in (x, y, g))
        return [torch.cat(v, 1) for v in (shuffle_product(lx, ly, w, True),
                                          shuffle_adjoint(lx, lg, w, True, False),
                                          shuffle_adjoint(ly, lg, w, True, True))]

    f = {"mul_grad": product_and_gradients, "shuffle": shuffles_and_gradient, "half": halves_and_gradients}[kind]
    return by_chunks(f, 1024, x, y, g)


def exact_paths(case, make):
    w, d, b, l = case["w"], case["d"], case["b"], case["l"]
    incr, offsets = make.paths()
    if offsets is not None:
        return uneven_signatures(incr.double(), offsets, w, d)
    incr = incr.double().reshape(b, l, w)
    if case["kind"] == "sig":
        return torch.cat(signatures(incr, w, d), 1)
    if case["kind"] == "logsig":
        s = signatures(incr, w, d)
        lie = by_chunks(lambda *v: [lie_coefficients(logarithm(list(v)), w, d)], 1024, *s)[0]
        return torch.cat(s, 1), lie
    # the gradient: the steps backward, each prefix from the one after it
    s = signatures(incr, w, d)
    whole = torch.cat(s, 1)
    g = levels(make.uniform(b, dim(w, d)), w, d)
    grad = torch.empty_like(incr)
    for k in range(l - 1, -1, -1):
        s = [v.detach().requires_grad_() for v in chen_step(s, -incr[:, k])]
        x = incr[:, k].detach().requires_grad_()
        got = torch.autograd.grad(chen_step(s, x), s + [x], g)
        g, grad[:, k] = list(got[:-1]), got[-1]
        s = [v.detach() for v in s]
    return whole, grad.reshape(b * l, w)


def uneven_signatures(incr, offsets, w, d):
    lengths = offsets[1:] - offsets[:-1]
    order = torch.argsort(lengths, descending=True)
    start, length = offsets[:-1][order], lengths[order].cpu().numpy()
    s = unit(w, d, len(order))
    for k in range(int(length[0])):
        alive = int(np.searchsorted(-length, -k, side="left"))  # paths with an increment k
        new = chen_step([v[:alive] for v in s], incr[start[:alive] + k])
        for v, x in zip(s[1:], new[1:]):
            v[:alive] = x
    out = torch.empty(len(order), dim(w, d), dtype=torch.float64, device="cuda")
    out[order] = torch.cat(s, 1)
    return out
