"""Batches whose launches have fewer blocks than the GPU holds, and batches in
which only some solves ask for a march length of their own through the C
interface (GPU): the traces of every solve alone, bit for bit, per step and
persistent, with more stress than velocity marches and fewer."""
import numpy as np
import pytest

from helpers import make_small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z_chunks", [(0, 0, 0), (0, 5, 0), (3, 0, 30), (1, 1, 1)])
@pytest.mark.parametrize("shapes", [[(20, 24, 32), (44, 30, 29), (16, 20, 64)], [(50, 90, 96), (24, 24, 24), (45, 31, 33)]])
def test_partly_chunked_batches(monkeypatch, z_chunks, shapes):
    from pefdtd import batch, fdtd
    probs = [make_small(nt=40, shape=s, n_grains=5, sponge=3, seed=80 + i) for i, s in enumerate(shapes)]
    specs = [batch.spec_from_problem(p) for p in probs]
    want = []
    for sp in specs:
        d = fdtd.DeviceSolve(**{k: v for k, v in sp.items() if k != "wavelet"})
        d.set_wavelet(sp["wavelet"])
        d.run(0, 40)
        want.append(d.traces_numpy(40))
        d.close()
    structs, todo = batch.c_solve_structs, list(z_chunks)
    monkeypatch.setattr(batch, "c_solve_structs", lambda *a, **kw: structs(*a, **dict(kw, z_chunk=todo.pop(0))))
    b = batch.BatchSolver(specs, chunk_steps=15)
    for persistent in (False, True):
        assert b.set_persistent(persistent) == persistent
        b.reset()
        b.run(0, 40)
        for got, ref in zip(b.traces_numpy(40), want):
            assert np.abs(ref).max() > 0
            assert np.array_equal(got, ref)
    b.close()
