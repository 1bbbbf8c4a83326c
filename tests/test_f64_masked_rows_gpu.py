"""FP64 solves with a damping volume on rows that are 16-byte units of doubles
but not of floats (nx = 2 mod 4, GPU): the TMA kernels' damping boxes come from
a row-padded copy. Traces against the oracle bit for bit, alone (a second run
on the same buffers too) and in a batch; the gradient against the untiled
kernels, to the order of its float64 atomic sums; the memory plan counts the copy."""
import numpy as np
import pytest

from helpers import make_small, oracle_prob
from oracle import oracle as O


def _masked(shape, nt=60):
    p = dict(make_small(nt=nt, shape=shape, n_grains=5, sponge=3, seed=13))
    p["damp_volume"] = np.random.default_rng(4).uniform(0.9, 1.0, shape).astype(np.float32)
    return p


def _oracle(p, **kw):
    return O.run_oracle(oracle_prob(p, record=p["record"], damped_record=True, dtype=np.float64,
                                    damp_mask=p["damp_volume"], **kw), dtype=np.float64, fma_mode=1)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(12, 20, 22), (14, 37, 30), (13, 24, 74), (12, 18, 338)])
def test_f64_masked_rows_equal_oracle(shape):
    from pefdtd import batch, fdtd
    p = _masked(shape)
    ref = _oracle(p)
    assert np.abs(ref).max() > 0
    spec = batch.spec_from_problem(p)
    wav = spec.pop("wavelet")
    d = fdtd.DeviceSolve(**spec, dtype="float64", chunk_steps=25)
    d.set_wavelet(wav)
    for _ in range(2):
        d.reset()
        d.run(0, p["nt"])
        assert np.array_equal(d.traces_numpy(p["nt"]), ref)
        d.traces.zero_()
    d.close()
    q = _masked((12, 20, 24))
    b = batch.BatchSolver([batch.spec_from_problem(x) for x in (p, q, p)], dtype="float64", chunk_steps=25)
    b.run(0, p["nt"])
    for got, want in zip(b.traces_numpy(p["nt"]), (ref, _oracle(q), ref)):
        assert np.array_equal(got, want)
    b.close()


@pytest.mark.gpu
def test_f64_masked_gradient_equals_untiled():
    from pefdtd import adjoint, batch, fdtd
    p = _masked((14, 24, 34), nt=40)
    spec = batch.spec_from_problem(p)
    wav = spec.pop("wavelet")
    got = []
    for variant in ("tiled", "simple"):
        d = fdtd.DeviceSolve(**spec, dtype="float64", variant=variant)
        d.set_wavelet(wav)
        a = adjoint.AdjointSolve(d, 15)
        tr = a.forward()
        got.append((tr.cpu().numpy(), a.backward(tr)))
        d.close()
    assert np.array_equal(got[0][0], got[1][0])
    # the same terms; their atomic sums in any order
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-12 * np.abs(got[1][1]).max()


def test_memory_plan_counts_the_padded_damping_volume():
    from pefdtd import adjoint
    shape = (40, 50, 62)
    plain = adjoint.adjoint_bytes(shape, 100, esize=8)
    assert adjoint.adjoint_bytes(shape, 100, esize=8, damp_volume=True) == plain + 4 * 40 * 50 * (62 + 64)
    assert adjoint.adjoint_bytes((40, 50, 64), 100, esize=8, damp_volume=True) == \
        adjoint.adjoint_bytes((40, 50, 64), 100, esize=8) + 4 * 40 * 50 * 64
