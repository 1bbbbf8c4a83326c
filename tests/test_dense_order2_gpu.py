"""Per-cell media of order 2 (GPU): grids on both sides of the size at which the
untiled kernels take over from the pair kernels, rows of 16-byte units and not,
give the same bits with the dispatch's choice and with the untiled kernels
(taken when a tile is asked for)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 249 984 and 252 000 cells and, with rows of no 16-byte units, 249 984 and 250 047
@pytest.mark.parametrize("shape", [(31, 72, 112), (35, 72, 100), (31, 64, 126), (63, 63, 63), (9, 12, 16)])
def test_order_2_either_side_of_the_limit(shape):
    from pefdtd import fdtd
    rng = np.random.default_rng(4)
    n = int(np.prod(shape))
    C = np.zeros((n, 6, 6))
    C[:] = np.diag([14e9, 14e9, 15e9, 3e9, 3e9, 3.4e9])
    C += rng.normal(size=C.shape) * 2e8
    C = 0.5 * (C + C.transpose(0, 2, 1))
    rho = rng.uniform(300.0, 920.0, n)
    cells = np.array([shape[2] - 1, n // 2, n - 1], np.int64)
    field = rng.normal(size=(9,) + shape).astype(np.float32) * 1e-6
    out = []
    for tile in ((0, 0), (32, 8)):
        d = fdtd.DeviceSolve(np.zeros(shape, np.uint16), C.reshape(n, 36), rho, 1e-4, 6e-9, [1.0], cells[1:], np.ones(2),
                             np.array([0, 2, 3], np.int64), cells, np.ones(3), record="vz", damped_record=True,
                             sponge=None, variant="dense", tile=tile, chunk_steps=20)
        d.set_wavelet(np.sin(0.3 * np.arange(25)))
        d.state.copy_(d.torch.from_numpy(field))
        d.run(0, 25)
        out.append((d.state.cpu().numpy(), d.traces_numpy(25)))
        d.close()
    assert np.array_equal(out[0][0].view(np.uint32), out[1][0].view(np.uint32))
    assert np.array_equal(out[0][1], out[1][1])
