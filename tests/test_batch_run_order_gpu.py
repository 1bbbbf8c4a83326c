"""Consecutive runs of one batch on a side stream, queued without waiting
(GPU): long runs go through row-padded states, runs of under 8 steps in place,
and each kind has arguments, maps and a graph of its own, so a run that is
queued behind a long one changes nothing that the long one still reads. Traces
and final states equal those of the solves run alone, bit for bit; a new work
layout between two queued runs too."""
import numpy as np
import pytest

from helpers import make_small

pytestmark = pytest.mark.gpu

CUTS = {"long_then_short": [(0, 300), (300, 305), (305, 320)],
        "alternating": [(0, 200), (200, 203), (203, 213), (213, 220), (220, 320)],
        "short_first": [(0, 5), (5, 205), (205, 210), (210, 320)]}


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("cuts", sorted(CUTS))
def test_queued_runs_of_both_kinds(persistent, cuts):
    from pefdtd import batch, fdtd
    probs = [make_small(nt=320, shape=s, n_grains=5, sponge=3, seed=60 + i)
             for i, s in enumerate([(20, 40, 61), (18, 36, 64), (24, 33, 50)])]
    specs = [batch.spec_from_problem(p) for p in probs]
    want = []
    for sp in specs:
        kw = {k: v for k, v in sp.items() if k != "wavelet"}
        d = fdtd.DeviceSolve(**kw)
        d.set_wavelet(sp["wavelet"])
        d.run(0, 320)
        want.append((d.traces_numpy(320), d.state.clone()))
        d.close()
    b = batch.BatchSolver(specs, chunk_steps=100)
    assert b.set_persistent(persistent) == persistent
    torch = b.torch
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    for again in range(2):
        with torch.cuda.stream(stream):
            b.reset()
            for i, (n0, n1) in enumerate(CUTS[cuts]):
                b.run(n0, n1)
                if again and i == 0:
                    b.schedule(9, 100)
        stream.synchronize()
        for got, st, (tr, state) in zip(b.traces_numpy(320), b.states, want):
            assert np.array_equal(got, tr)
            assert torch.equal(st, state)
    b.close()
