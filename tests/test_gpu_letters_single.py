"""The warp-per-letter FP32 kernels of the shapes that only single calls take
(csrc/signature_fp32_narrow.cu, signature_fp32_wide.cu): against the FP64
oracle, with ragged batches of empty and unit paths, and the forward kernel
against the shared-memory kernel bit for bit."""
import importlib

import numpy as np
import pytest

from _helpers import TOL_F32, assert_close, scaled_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")

SHAPES = [(2, 2), (2, 3), (2, 4), (2, 5), (2, 6), (2, 7), (3, 2), (3, 3), (3, 4), (4, 2), (4, 3), (4, 6), (6, 2),
          (6, 3), (6, 5), (7, 2), (7, 3), (7, 4)]


@pytest.mark.parametrize("W,D", SHAPES)
@pytest.mark.parametrize("ragged", [False, True])
def test_shapes_of_single_calls(orc, W, D, ragged):
    rng = np.random.default_rng(W * 10 + D)
    lengths = np.array([0, 1, 2, 17, 5, 0, 9, 31, 1, 4, 12, 3, 8]) if ragged else np.full(13, 9)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    B, basis, st = len(lengths), pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float32)
    incr = rng.normal(0, 1 / 3, (int(offsets[-1]), W)).astype(np.float32).astype(np.float64)
    ell = rng.uniform(-1, 1, (B, basis.size())).astype(np.float32).astype(np.float64)
    want_sig, want_grad = orc.signature(W, D, incr, offsets, ell=ell)
    x, seed = (torch.from_numpy(v).to("cuda", torch.float32) for v in (incr, ell))
    where = {"offsets": torch.from_numpy(offsets).cuda()} if ragged else {"length": 9}

    def empty(like):
        return torch.full_like(like, float("nan"))

    sig, grad, forward, whole, alone = empty(seed), empty(x), empty(seed), empty(seed), empty(x)
    assert pkg.signature(st, None, x, basis, B, out=sig, seed=seed, grad=grad, **where)
    assert pkg.signature(st, None, x, basis, B, out=forward, **where)
    assert pkg.signature(st, None, x, basis, B, out=whole, schedule=128, **where)
    assert pkg.signature(st, None, x, basis, B, seed=seed, grad=alone, **where)
    back = empty(x)
    assert pkg.signature_backward(st, None, x, basis, B, sig, seed, back, **where)
    assert_close(sig.double().cpu().numpy(), want_sig, TOL_F32, "signature")
    assert torch.equal(forward, whole), "the forward kernel forms the shared-memory kernel's multiply-adds"
    for g in (grad, alone, back):
        assert scaled_err(g.double().cpu().numpy(), want_grad) <= TOL_F32
    # as before, a schedule cannot ask for these shapes' kernels
    assert not pkg.signature(st, None, x, basis, B, out=sig, schedule=32 | (1 << 16), **where)


def test_tuned_and_grouped_calls_of_such_a_shape(orc):
    W, D, B, L = 6, 3, 700, 12
    rng = np.random.default_rng(3)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float32)
    x = torch.from_numpy(rng.normal(0, 0.3, (B * L, W))).to("cuda", torch.float32)
    seed = torch.from_numpy(rng.uniform(-1, 1, (B, basis.size()))).to("cuda", torch.float32)
    sig, grad = torch.empty_like(seed), torch.empty_like(x)
    err, _, _ = pkg.signature_tune(st, None, x, basis, B, length=L, out=sig, seed=seed, grad=grad)
    assert err, err.message
    gsig, ggrad = torch.empty_like(sig), torch.empty_like(grad)
    job = pkg.SignatureJob(st, x, basis, B, length=L, out=gsig, seed=seed, grad=ggrad)
    err = pkg.signature_group(None, [job])
    assert err, err.message
    want_sig, want_grad = orc.signature(W, D, x.double().cpu().numpy(), np.arange(B + 1) * L,
                                        ell=seed.double().cpu().numpy())
    for s, g in ((sig, grad), (gsig, ggrad)):
        assert_close(s.double().cpu().numpy(), want_sig, TOL_F32, "signature")
        assert scaled_err(g.double().cpu().numpy(), want_grad) <= TOL_F32
