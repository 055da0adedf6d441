"""rpp_gb_signature_tune against calls that were not tuned: tuning leaves no call
slower, and what it reports is what later calls take."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

pkg = importlib.import_module("rough-path-primitives_gb300")


def fastest_ms(call, calls=20, runs=7):
    """The best mean time of a call among several runs of some."""
    best = float("inf")
    for _ in range(runs):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        begin.record()
        for _ in range(calls):
            call()
        end.record()
        torch.cuda.synchronize()
        best = min(best, begin.elapsed_time(end) / calls)
    return best


# (shapes and outputs that no other test tunes: what is recorded holds for the process)
@pytest.mark.parametrize("W,D,B,L,reverse", [(4, 4, 4096, 16, False), (3, 5, 4096, 16, True), (4, 3, 3, 1000, True)])
def test_tuned_calls_are_no_slower_than_untuned_ones(W, D, B, L, reverse):
    rng = np.random.default_rng(W * 10 + D)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float64)
    x = torch.from_numpy(rng.normal(0, 1 / np.sqrt(L), (B * L, W))).cuda()
    sig = torch.empty(B, basis.size(), dtype=torch.float64, device="cuda")
    more = {"seed": torch.rand_like(sig) * 2 - 1, "grad": torch.empty_like(x)} if reverse else {}

    def call():
        assert pkg.signature(st, None, x, basis, B, length=L, out=sig, **more)

    call()
    want = [t.clone() for t in (sig, *([more["grad"]] if reverse else []))]
    untuned = fastest_ms(call)
    err, _, ms = pkg.signature_tune(st, None, x, basis, B, length=L, out=sig, **more)
    assert err, err.message
    for got, ref in zip((sig, *([more["grad"]] if reverse else [])), want):
        assert torch.allclose(got, ref, rtol=1e-10, atol=1e-10)
    tuned = fastest_ms(call)
    # (an eighth: more than the clocks move between two runs of one call)
    assert tuned <= 1.125 * untuned, (tuned, untuned)
    assert 0.5 * tuned <= ms <= 2.0 * tuned, (ms, tuned)


# shapes with warp-per-letter kernels that only single calls take, and one that the grouped launch takes too
@pytest.mark.parametrize("W,D", [(2, 5), (4, 3), (6, 2), (6, 5), (7, 3), (5, 3)])
@pytest.mark.parametrize("reverse", [False, True])
def test_a_schedule_that_the_tuner_returns_can_be_pinned(W, D, reverse):
    B, L = 300, 12
    rng = np.random.default_rng(W * 10 + D)
    basis, st = pkg.TensorBasis(W, D), pkg.GB300Strategy(torch.float32)
    x = torch.from_numpy(rng.normal(0, 1 / np.sqrt(L), (B * L, W))).to("cuda", torch.float32)
    offsets = torch.arange(0, (B + 1) * L, L, device="cuda")  # (as an uneven batch, which is never cut in time)
    sig = torch.empty(B, basis.size(), dtype=torch.float32, device="cuda")
    more = {"seed": torch.rand_like(sig) * 2 - 1, "grad": torch.empty_like(x)} if reverse else {}
    outputs = [sig] + ([more["grad"]] if reverse else [])

    def check(want):
        torch.cuda.synchronize()
        for got, ref in zip(outputs, want):
            assert torch.allclose(got, ref, rtol=1e-4, atol=1e-4)
            got.fill_(float("nan"))

    err = pkg.signature(st, None, x, basis, B, offsets=offsets, out=sig, **more)
    assert err, err.message
    want = [t.clone() for t in outputs]
    err, word, _ = pkg.signature_tune(st, None, x, basis, B, offsets=offsets, out=sig, **more)
    assert err, err.message
    check(want)
    for schedule in (word, None, 128 | (1 << 15) | (1 << 16), *([128 | (1 << 16)] if reverse else [])):
        err = pkg.signature(st, None, x, basis, B, offsets=offsets, out=sig, schedule=schedule, **more)
        assert err, (schedule, err.message)
        check(want)
    if (reverse or (W, D) == (5, 3)) and D > 2:
        assert pkg.signature(st, None, x, basis, B, offsets=offsets, out=sig, schedule=32 | (1 << 16), **more)
        check(want)
