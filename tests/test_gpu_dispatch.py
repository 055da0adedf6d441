"""Calls whose kernel depends on how many tensors there are: the same rows in a
large batch and a few at a time, on both sides of the lines (csrc/ft_column.cuh's
Worth, csrc/ft_adjoint.cu, csrc/shuffle_letters.cu), agree; and few tensors take
no longer than the general kernel takes for them, where a call can ask for it."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")
from test_gpu_column import EPS, Rows  # noqa: E402

SHAPES = [(2, 2), (2, 5), (2, 8), (3, 3), (3, 4), (4, 3), (4, 5), (5, 2), (5, 3), (6, 4), (7, 2), (7, 3), (8, 3)]
MANY, FEW = 2100, 3


def operations(st, basis, lie, t2l, l2t, D):
    """name -> (call(out, x, y, a, n), degrees of the output); `a` a Lie batch or a tensor."""
    full = (0, D)

    def on(op, *more, lo=0):
        return lambda o, x, y, a, n: op(st, None, o.view(lo), *(v.view() for v in (x, y)), basis, n, *more)

    ops = {"ft_mul": (on(pkg.ft_mul, -0.5), full), "ft_adj_lmul": (on(pkg.ft_adj_lmul), full),
           "ft_adj_rmul": (on(pkg.ft_adj_rmul), full), "ft_fmexp": (on(pkg.ft_fmexp), full),
           "ft_fma": (lambda o, x, y, a, n: pkg.ft_fma(st, None, o.view(), a.view(), x.view(), y.view(), basis, n, 2.0,
                                                       -0.5), full),
           "ft_inplace_fma": (lambda o, x, y, a, n: pkg.ft_inplace_fma(
               pkg.FTInplaceFMAType(0), st, None, o.view(), x.view(), y.view(), basis, n, 2.0, -0.5), full),
           "ft_exp": (lambda o, x, y, a, n: pkg.ft_exp(st, None, o.view(), x.view(), basis, n), full),
           "ft_log": (lambda o, x, y, a, n: pkg.ft_log(st, None, o.view(), x.view(), basis, n), full),
           "lie_exp": (lambda o, x, y, a, n: pkg.lie_to_tensor_exp(st, None, o.view(), None, a.lie, basis, lie, n, l2t),
                       full),
           "lie_fmexp": (lambda o, x, y, a, n: pkg.lie_to_tensor_exp(st, None, o.view(), y.view(), a.lie, basis, lie, n,
                                                                     l2t), full)}
    if D >= 3:
        for name in ("st_mul", "st_adj_mul", "left_hs_mul", "left_hs_adj_lmul", "left_hs_adj_rmul"):
            ops[name] = (on(getattr(pkg, name)), full)
    return ops


@pytest.mark.parametrize("W,D", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_rows_of_a_large_batch_and_a_few_at_a_time(W, D, dtype):
    rng = np.random.default_rng(W * 10 + D)
    st, basis, lie = pkg.GB300Strategy(dtype), pkg.TensorBasis(W, D), pkg.LieBasis(W, D)
    t2l, l2t, size = pkg.make_t2l_matrix(lie), pkg.make_l2t_matrix(lie), lie.true_size()
    x, y, a = (Rows(rng, dtype, W, D, MANY, 3, 1, 0.4) for _ in range(3))
    vectors = torch.from_numpy(rng.uniform(-0.3, 0.3, (MANY, size))).to("cuda", dtype)
    a.lie = pkg.make_lie_batch(vectors, size, 1, D)
    start = Rows(rng, dtype, W, D, MANY, 3, 1, 0.4)
    # two results of a sum of at most dim terms, each in its own order; 16: the rounds
    # of exp and log, each a sum again
    tol = 16 * basis.size() * EPS[dtype]
    for name, (call, _) in operations(st, basis, lie, t2l, l2t, D).items():
        outs = []
        for n in (MANY, FEW):
            out = Rows(np.random.default_rng(1), dtype, W, D, MANY, 3, 1)
            out.rows.copy_(start.rows)
            err = call(out, x, y, a, n)
            assert err, (name, err.message)
            outs.append(out.host())
        many, few = outs
        scale = max(1.0, abs(many).max())
        assert abs(many[:FEW] - few[:FEW]).max() <= tol * scale, name
        assert np.array_equal(few[FEW:], start.host()[FEW:]), name
    logs = []
    for n in (MANY, FEW):
        out = torch.zeros(MANY, size, dtype=dtype, device="cuda")
        assert pkg.tensor_log_to_lie(st, None, pkg.make_lie_batch(out, size, 1, D), x.view(), lie, basis, n, t2l)
        logs.append(out.double().cpu().numpy())
    assert abs(logs[0][:FEW] - logs[1][:FEW]).max() <= tol * max(1.0, abs(logs[0]).max())


def graph_ms(call, calls=20, runs=9):
    """The best time of a call in a replayed graph of some."""
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    call()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(calls):
            call()
    best = float("inf")
    for _ in range(runs):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        begin.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        best = min(best, begin.elapsed_time(end) / calls)
    return best


@pytest.mark.parametrize("name,W,D,dtype", [("st_adj_mul", 7, 3, torch.float32), ("st_adj_mul", 3, 6, torch.float64),
                                            ("left_hs_adj_lmul", 5, 4, torch.float32),
                                            ("left_hs_adj_rmul", 8, 4, torch.float32), ("st_mul", 4, 5, torch.float64),
                                            ("st_mul", 2, 5, torch.float32), ("left_hs_mul", 2, 7, torch.float64)])
def test_few_shuffles_take_the_subset_sums_time(name, W, D, dtype):
    B, basis, st = 64, pkg.TensorBasis(W, D), pkg.GB300Strategy(dtype)
    tensors = [torch.rand(B, basis.size(), dtype=dtype, device="cuda") * 0.01 for _ in range(3)]
    out, x, y = (pkg.make_tensor_batch(t, basis.size(), 0, D) for t in tensors)
    op = getattr(pkg, name)
    apart = graph_ms(lambda: op(st, None, out, x, y, basis, B))
    over = graph_ms(lambda: op(st, None, x, x, y, basis, B))  # over an operand: the subset sums
    assert apart <= 1.25 * over, (apart, over)  # (letters took 1.5 to 3 times as long)
