"""Per-cell media on the pair kernels (GPU): the same bits, traces and all nine
fields, as the untiled kernels (taken when a tile is asked for), on one tile
and several, rows of every remainder, four coefficients and fewer, densities
that differ from cell to cell, with and without a damping volume."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,order", [((9, 10, 8), 8), ((12, 15, 31), 8), ((13, 33, 64), 4), ((10, 45, 99), 8),
                                         ((11, 40, 130), 6)])
@pytest.mark.parametrize("mask,record", [(False, "vz"), (True, "pressure")])
def test_pair_kernels_equal_untiled_per_cell(shape, order, mask, record):
    from pefdtd import fdtd
    from pefdtd.coeffs import taylor_coeffs
    rng = np.random.default_rng(4)
    n = int(np.prod(shape))
    C = np.zeros((n, 6, 6))
    C[:] = np.diag([14e9, 14e9, 15e9, 3e9, 3e9, 3.4e9])
    C += rng.normal(size=C.shape) * 2e8
    C = 0.5 * (C + C.transpose(0, 2, 1))
    rho = rng.uniform(300.0, 920.0, n)
    cells = np.array([shape[2] - 1, n // 2, n - 1], np.int64)
    sol = []
    for tile in ((0, 0), (32, 8)):
        d = fdtd.DeviceSolve(np.zeros(shape, np.uint16), C.reshape(n, 36), rho, 1e-4, 6e-9, taylor_coeffs(order),
                             cells[1:], np.ones(2), np.array([0, 2, 3], np.int64), cells, np.ones(3), record=record,
                             damped_record=True, sponge=None, variant="dense", tile=tile, chunk_steps=20,
                             damp_volume=np.random.default_rng(1).uniform(0.9, 1.0, shape) if mask else None)
        d.set_wavelet(np.sin(0.3 * np.arange(45)))
        d.state.copy_(d.torch.from_numpy(np.random.default_rng(2).normal(size=(9,) + shape).astype(np.float32) * 1e-6))
        for a, b in [(0, 30), (30, 33), (33, 45)]:
            d.run(a, b)
        sol.append(d)
    a, b = sol
    assert a.torch.equal(a.state, b.state)
    assert np.array_equal(a.traces_numpy(45), b.traces_numpy(45))
    for d in sol:
        d.close()
