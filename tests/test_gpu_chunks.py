"""Few long paths cut in time (csrc/signature_chunks.cu): signatures and
gradients against the oracle and against the same paths run whole, for the
staged and the in-place joins, pieces that do not divide the path, and every
kind of output; a batch computed in parts gives the bits of the whole one."""
import importlib

import numpy as np
import pytest

from _helpers import TOL_F32, TOL_F64, assert_close, scaled_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")

# (W, D, paths, increments): sizes that the rule cuts with a reverse pass --
# columns of one, two and three first letters, widths without columns (the
# joins read global memory), a state too large for shared memory (W6 D6)
SHAPES = [(2, 5, 1, 97), (2, 10, 3, 64), (3, 3, 5, 301), (3, 5, 4, 200), (5, 4, 2, 131), (8, 3, 7, 100), (9, 3, 2, 120),
          (1, 5, 2, 150), (16, 3, 1, 90), (6, 6, 1, 24), (4, 2, 3, 513)]


def call(W, D, B, L, incr, ell, dtype, want_sig=True, schedule=None):
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(dtype)
    x = torch.from_numpy(incr).to("cuda", dtype)
    sig = torch.full((B, basis.size()), float("nan"), dtype=dtype, device="cuda") if want_sig else None
    seed = None if ell is None else torch.from_numpy(ell).to("cuda", dtype)
    grad = None if ell is None else torch.full_like(x, float("nan"))
    err = pkg.signature(st, None, x, basis, B, length=L, out=sig, seed=seed, grad=grad, schedule=schedule)
    assert err, err.message
    return tuple(None if t is None else t.double().cpu().numpy() for t in (sig, grad))


@pytest.mark.parametrize("W,D,B,L", SHAPES)
@pytest.mark.parametrize("dtype,tol", [(torch.float64, TOL_F64), (torch.float32, TOL_F32)])
def test_pieces_match_oracle(orc, W, D, B, L, dtype, tol):
    rng = np.random.default_rng(W * 100 + D)
    incr = rng.normal(0, 1 / np.sqrt(L), (B * L, W))
    ell = rng.uniform(-1, 1, (B, pkg.TensorBasis(W, D).size()))
    if dtype == torch.float32:
        incr, ell = (v.astype(np.float32).astype(np.float64) for v in (incr, ell))
    want_sig, want_grad = orc.signature(W, D, incr, np.arange(B + 1) * L, ell=ell)
    sig, grad = call(W, D, B, L, incr, ell, dtype)
    assert_close(sig, want_sig, tol, "signature")
    assert scaled_err(grad, want_grad) <= tol
    only, _ = call(W, D, B, L, incr, None, dtype)
    assert_close(only, want_sig, tol, "forward only")
    _, alone = call(W, D, B, L, incr, ell, dtype, want_sig=False)
    assert np.array_equal(alone, grad), "gradient only"
    if dtype == torch.float64 and W * D <= 64 and W < 16:
        whole, whole_grad = call(W, D, B, L, incr, ell, dtype, schedule=256)
        assert_close(sig, whole, tol, "in pieces against whole")
        assert scaled_err(grad, whole_grad) <= tol


@pytest.mark.parametrize("chunk", [1, 2, 5])
def test_parts_of_a_batch_are_cut_as_the_whole(chunk):
    W, D, B, L = 3, 4, 5, 400
    rng = np.random.default_rng(7)
    incr, ell = rng.normal(0, 1 / np.sqrt(L), (B * L, W)), rng.uniform(-1, 1, (B, pkg.TensorBasis(W, D).size()))
    sig, grad = call(W, D, B, L, incr, ell, torch.float64)
    host = [torch.from_numpy(v) for v in (incr, ell)]
    hsig, hgrad = torch.empty(sig.shape, dtype=torch.float64), torch.empty(grad.shape, dtype=torch.float64)
    assert pkg.signature_host(pkg.GB300Strategy(torch.float64), None, host[0], pkg.TensorBasis(W, D), B, length=L,
                              out=hsig, seed=host[1], grad=hgrad, chunk=chunk)
    torch.cuda.synchronize()
    assert np.array_equal(hsig.numpy(), sig) and np.array_equal(hgrad.numpy(), grad)


def test_pieces_in_a_graph_replay_the_eager_results():
    W, D, B, L = 4, 4, 2, 300
    rng = np.random.default_rng(8)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float64)
    x = torch.from_numpy(rng.normal(0, 1 / np.sqrt(L), (B * L, W))).cuda()
    seed = torch.from_numpy(rng.uniform(-1, 1, (B, basis.size()))).cuda()
    sig, grad = torch.empty_like(seed), torch.empty_like(x)

    def run():
        assert pkg.signature(st, None, x, basis, B, length=L, out=sig, seed=seed, grad=grad)

    run()
    torch.cuda.synchronize()
    want = sig.clone(), grad.clone()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        run()
    for _ in range(2):
        sig.zero_(), grad.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(sig, want[0]) and torch.equal(grad, want[1])
