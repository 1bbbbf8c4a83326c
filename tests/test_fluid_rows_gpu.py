"""The pair stress kernel's couplant path (GPU; warps whose cells are all a
shear-free material 0) against the full product, bit for bit: the same medium
with its table rows in another order, so that row 0 is not the couplant. Grids
that are all couplant, half, and thin couplant layers; a couplant with one
shear constant; and fields holding infinities, NaN and values near overflow,
where a skipped product with a zero constant would show."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(mats, Ct, rho, poison, steps=14):
    from pefdtd import fdtd
    from pefdtd.coeffs import taylor_coeffs
    shape = mats.shape
    n = int(np.prod(shape))
    cells = np.array([n // 2, n // 3], np.int64)
    d = fdtd.DeviceSolve(mats, Ct, rho, 1e-4, 6e-9, taylor_coeffs(8), cells, np.ones(2), np.array([0, 2], np.int64),
                         cells, np.ones(2), record="pressure", damped_record=True)
    d.set_wavelet(np.sin(0.3 * np.arange(steps)))
    f = np.random.default_rng(2).normal(size=(9,) + shape).astype(np.float32) * np.float32(1e-6)
    if poison is not None:
        f[1].reshape(-1)[n // 2 + 3] = poison
        f[6].reshape(-1)[n // 4] = -poison
    d.state.copy_(d.torch.from_numpy(f))
    d.run(0, steps)
    out = d.state.cpu().numpy(), d.traces_numpy(steps)
    d.close()
    return out


@pytest.mark.parametrize("layout", ["all", "half", "layers"])
@pytest.mark.parametrize("shear", [0.0, 1.0e3])
@pytest.mark.parametrize("poison", [None, np.inf, np.nan, 3e38, 2e19])
def test_couplant_path_equals_full_product(layout, shear, poison):
    shape = (14, 40, 72)
    rng = np.random.default_rng(3)
    C = np.zeros((3, 6, 6))
    C[0, :3, :3] = 300.0 * 1500.0 ** 2
    C[0, 3, 3] = shear
    A = rng.normal(size=(2, 6, 6)) * 2e8
    C[1:] = np.diag([14e9, 14e9, 15e9, 3e9, 3e9, 3.4e9]) + A + A.transpose(0, 2, 1)
    rho = np.array([300.0, 917.0, 917.0])
    mats = np.zeros(shape, np.uint16)
    if layout == "half":
        mats[:, 18:, 30:] = rng.integers(1, 3, (14, 22, 42))
    elif layout == "layers":
        mats[::3] = 1
        mats[:, :, 37] = 2
    got = _run(mats, C.reshape(3, 36), rho, poison)
    order = np.array([1, 0, 2])   # rows 0 and 1 change places, and so do the indices
    want = _run(order[mats].astype(np.uint16), C[order].reshape(3, 36), rho[order], poison)
    for w, g in zip(want, got):   # NaN where NaN (payloads aside), else the same bits
        assert np.array_equal(np.isnan(w), np.isnan(g))
        assert np.array_equal(np.where(np.isnan(w), 0, w).view(np.uint32), np.where(np.isnan(g), 0, g).view(np.uint32))
