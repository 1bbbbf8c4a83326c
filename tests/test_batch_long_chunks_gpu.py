"""Batches whose graphs cover more steps than a solver's own chunk of 200 (GPU;
the autotuner tries 400): the receivers' sample buffer holds every step of the
chunk, for a schedule set later and for solves that were made with shorter
chunks than the batch's."""
import numpy as np
import pytest

from helpers import make_small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("chunks,schedule", [((0, 0), 400), ((0, 0), 900), ((450, 7), 0), ((450, 7), 600)])
def test_chunks_longer_than_the_solvers(monkeypatch, dtype, persistent, chunks, schedule):
    from pefdtd import batch, fdtd
    if persistent and dtype == "float64":
        pytest.skip("the persistent kernel is FP32")
    nt = 900
    probs = [make_small(nt=nt, shape=s, n_grains=4, sponge=2, seed=90 + i) for i, s in enumerate([(16, 20, 24), (18, 22, 21)])]
    specs = [batch.spec_from_problem(p) for p in probs]
    want = []
    for sp in specs:
        d = fdtd.DeviceSolve(**{k: v for k, v in sp.items() if k != "wavelet"}, dtype=dtype, chunk_steps=40)
        d.set_wavelet(sp["wavelet"])
        d.run(0, nt)
        want.append(d.traces_numpy(nt))
        d.close()
    structs, todo = batch.c_solve_structs, list(chunks)
    monkeypatch.setattr(batch, "c_solve_structs", lambda *a, **kw: structs(*a, **dict(kw, chunk_steps=todo.pop(0))))
    b = batch.BatchSolver(specs, dtype=dtype)
    if schedule:
        b.schedule(0, schedule)
    assert b.set_persistent(persistent) == persistent
    b.run(0, nt)
    for got, ref in zip(b.traces_numpy(nt), want):
        assert np.array_equal(got, ref)
    b.close()
