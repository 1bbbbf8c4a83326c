"""Couplant warps of a solve that diverges while it runs (GPU): strains pass the
couplant path's limit plane by plane, in some tiles before others, and the
warps of a block change to the full product in the middle of a march. The same
bits as the same medium with its table rows in another order (no couplant
path), up to fields that are all NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(mats, Ct, rho, field, steps):
    from pefdtd import fdtd
    from pefdtd.coeffs import taylor_coeffs
    n = int(np.prod(mats.shape))
    cells = np.array([n // 2, n // 3], np.int64)
    # ten times the stable step: growth of some orders of magnitude a step
    d = fdtd.DeviceSolve(mats, Ct, rho, 1e-4, 3e-7, taylor_coeffs(8), cells, np.ones(2), np.array([0, 2], np.int64),
                         cells, np.ones(2), record="pressure", damped_record=True)
    d.set_wavelet(np.zeros(steps))
    d.state.copy_(d.torch.from_numpy(field))
    out = []
    for k in range(steps):   # every state on the way
        d.run(k, k + 1)
        out.append(d.state.cpu().numpy())
    d.close()
    return out


@pytest.mark.parametrize("shape", [(40, 46, 96), (23, 62, 128)])
def test_divergence_in_the_couplant(shape):
    rng = np.random.default_rng(8)
    C = np.zeros((2, 6, 6))
    C[0, :3, :3] = 300.0 * 1500.0 ** 2
    C[1] = np.diag([14e9, 14e9, 15e9, 3e9, 3e9, 3.4e9])
    rho = np.array([300.0, 917.0])
    mats = np.zeros(shape, np.uint16)
    mats[5:9, :, 40:60] = 1
    field = np.zeros((9,) + shape, np.float32)
    # a few strong cells far apart: the growth reaches the rest of the grid later
    for _ in range(6):
        z, y, x = [rng.integers(0, s) for s in shape]
        field[rng.integers(0, 3), z, y, x] = 1.0
    steps = 30
    got = _run(mats, C.reshape(2, 36), rho, field, steps)
    want = _run((1 - mats).astype(np.uint16), C[::-1].reshape(2, 36), rho[::-1], field, steps)
    assert np.isfinite(want[2]).all() and not np.isfinite(want[-1]).all()   # the run passes the limit
    for w, g in zip(want, got):
        assert np.array_equal(np.isnan(w), np.isnan(g))
        assert np.array_equal(np.where(np.isnan(w), 0, w).view(np.uint32), np.where(np.isnan(g), 0, g).view(np.uint32))
