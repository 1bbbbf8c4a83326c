"""A longer wavelet set between runs that keep their state and trace buffers
(GPU, as a caller of the C interface may): the captured graphs and the batch's
uploaded arguments follow the wavelet to its new buffer."""
import ctypes as C

import numpy as np
import pytest

from helpers import make_small

pytestmark = pytest.mark.gpu
SHORT, LONG = 60, 400


def _problem(shape, seed):
    from pefdtd import batch
    spec = batch.spec_from_problem(make_small(nt=SHORT, shape=shape, n_grains=5, sponge=3, seed=seed))
    w = np.sin(0.21 * np.arange(LONG) + seed) * np.hanning(LONG)
    return spec, w


def _alone(spec, w):
    from pefdtd import fdtd
    d = fdtd.DeviceSolve(**{k: v for k, v in spec.items() if k != "wavelet"}, chunk_steps=20)
    d.set_wavelet(w)
    d.run(0, LONG)
    out = d.traces_numpy(LONG)
    d.close()
    return out


@pytest.mark.parametrize("shape", [(16, 24, 40), (16, 24, 37)])
def test_solver_follows_a_new_wavelet(shape):
    from pefdtd import _capi, fdtd
    spec, w = _problem(shape, 1)
    want = _alone(spec, w)
    d = fdtd.DeviceSolve(**{k: v for k, v in spec.items() if k != "wavelet"}, chunk_steps=20)
    d.set_wavelet(w[:SHORT] * 0.5)
    d.traces = d.torch.zeros((LONG, 1), device="cuda")   # one trace buffer for all runs
    for _ in range(2):
        d.reset()
        d.run(0, SHORT)
    w32 = np.ascontiguousarray(w.astype(np.float32))
    _capi.check(d._L.pe_solver_set_wavelet(d._h, _capi.ptr(w32), LONG))
    d.reset()
    d.run(0, LONG)
    assert np.array_equal(d.traces_numpy(LONG), want)
    d.close()


@pytest.mark.parametrize("persistent", [False, True])
def test_batch_follows_a_new_wavelet(persistent):
    from pefdtd import _capi, batch
    probs = [_problem((16, 24, 40), 2), _problem((18, 22, 35), 3)]
    want = [_alone(*q) for q in probs]
    b = batch.BatchSolver([dict(s, wavelet=w[:SHORT] * 0.5) for s, w in probs], chunk_steps=20)
    assert b.set_persistent(persistent) == persistent
    for i in range(2):
        b.traces[i] = b.torch.zeros((LONG, 1), device="cuda")
        b._tr[i] = b.traces[i].data_ptr()
    for _ in range(2):
        b.reset()
        b.run(0, SHORT)
    for i, (_, w) in enumerate(probs):
        w32 = np.ascontiguousarray(w.astype(np.float32))
        _capi.check(b._L.pe_batch_set_wavelet(b._h, i, _capi.ptr(w32), C.c_int64(LONG)))
    b.reset()
    b.run(0, LONG)
    for got, ref in zip(b.traces_numpy(LONG), want):
        assert np.array_equal(got, ref)
    b.close()
