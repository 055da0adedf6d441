"""Calls without a schedule: the forms that the default rule picks as the batch
grows (one fused launch, two launches, top level in the rows, cotangents in the
workspace, a state split over a cluster) against the oracle, with gradient-only,
forward-only and backward-entry calls, equal and uneven lengths, and parts of a
batch against the whole of it."""
import importlib

import numpy as np
import pytest

from _helpers import TOL_F32, TOL_F64, assert_close, scaled_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")

# (W, D, paths): one warp per path; 4 paths an SM; two launches; cotangents in the workspace; a cluster
SHAPES = [(3, 4, 5000), (4, 4, 600), (7, 3, 2000), (5, 4, 3000), (9, 3, 1500), (2, 10, 1600), (6, 5, 700), (2, 12, 320),
          (6, 6, 160), (1, 6, 700), (16, 3, 1000), (3, 1, 900), (5, 2, 5000)]


@pytest.mark.parametrize("W,D,B", SHAPES)
@pytest.mark.parametrize("ragged", [False, True])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, TOL_F64), (torch.float32, TOL_F32)])
def test_default_schedule_matches_oracle(orc, W, D, B, ragged, dtype, tol):
    rng = np.random.default_rng(W * 100 + D)
    lengths = rng.integers(0, 8, B) if ragged else np.full(B, 4)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(dtype)
    x = torch.from_numpy(rng.normal(0, 0.4, (int(offsets[-1]), W))).to("cuda", dtype)
    seed = torch.from_numpy(rng.uniform(-1, 1, (B, basis.size()))).to("cuda", dtype)
    where = {"offsets": torch.from_numpy(offsets).cuda()} if ragged else {"length": 4}

    def empty(like):
        return torch.full_like(like, float("nan"))

    sig, grad, forward, alone, back = empty(seed), empty(x), empty(seed), empty(x), empty(x)
    assert pkg.signature(st, None, x, basis, B, out=sig, seed=seed, grad=grad, **where)
    assert pkg.signature(st, None, x, basis, B, out=forward, **where)
    assert pkg.signature(st, None, x, basis, B, seed=seed, grad=alone, **where)
    assert pkg.signature_backward(st, None, x, basis, B, sig, seed, back, **where)
    # every 40th path (and the longest) against the oracle
    pick = np.unique(np.concatenate([np.arange(0, B, max(1, B // 40)), [int(np.argmax(lengths))]]))
    rows = np.concatenate([np.arange(offsets[b], offsets[b + 1]) for b in pick]).astype(np.int64)
    own = np.concatenate([[0], np.cumsum(lengths[pick])]).astype(np.int64)
    want_sig, want_grad = orc.signature(W, D, x[rows].double().cpu().numpy(), own,
                                        ell=seed[pick].double().cpu().numpy())
    for s in (sig, forward):
        assert_close(s[pick].double().cpu().numpy(), want_sig, tol, "signature")
    for g in (grad, alone, back):
        assert scaled_err(g[rows].double().cpu().numpy(), want_grad) <= tol
        assert torch.isfinite(g).all()
    assert torch.isfinite(sig).all() and torch.isfinite(forward).all()


def test_parts_take_the_schedule_of_the_whole_batch():
    W, D, B, L = 4, 4, 700, 5
    rng = np.random.default_rng(5)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float64)
    x, seed = rng.normal(0, 0.4, (B * L, W)), rng.uniform(-1, 1, (B, basis.size()))
    sig, grad = torch.empty(seed.shape, dtype=torch.float64, device="cuda"), torch.empty(x.shape, dtype=torch.float64,
                                                                                         device="cuda")
    assert pkg.signature(st, None, torch.from_numpy(x).cuda(), basis, B, length=L, out=sig,
                         seed=torch.from_numpy(seed).cuda(), grad=grad)
    for chunk in (0, 64):
        hsig, hgrad = torch.empty(seed.shape, dtype=torch.float64), torch.empty(x.shape, dtype=torch.float64)
        assert pkg.signature_host(st, None, torch.from_numpy(x), basis, B, length=L, out=hsig,
                                  seed=torch.from_numpy(seed), grad=hgrad, chunk=chunk)
        torch.cuda.synchronize()
        assert torch.equal(hsig, sig.cpu()) and torch.equal(hgrad, grad.cpu())
