"""The two-cell adjoint kernels (GPU, FP32, even rows, 8-byte aligned buffers)
against the one-cell kernels, which an adjoint state moved by one element
runs: the adjoint fields and the scratch (strains, moved columns) bit for bit,
the stiffness gradient to the order of its float64 atomic sums, on grids of
one block and several with interior blocks, ragged last blocks, every order,
a sponge and a damping volume."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(d, L, lam, vp, scratch, res, shift):
    """One reverse step on copies of the fields, `shift` elements into their buffers."""
    from pefdtd import _capi, adjoint
    t = d.torch
    n = int(np.prod(d.shape))

    def place(x):
        buf = t.zeros(x.numel() + 4, dtype=x.dtype, device=x.device)
        buf[shift:shift + x.numel()] = x.reshape(-1)
        return buf, buf[shift:shift + x.numel()]
    keep, lam2 = place(lam)
    keep2, vp2 = place(vp)
    grad = t.zeros((d.cfg.n_mat, 21), dtype=t.float64, device=lam.device)
    a = adjoint._PeAdjoint()
    for i in range(3):
        a.lv[i] = lam2.data_ptr() + 4 * i * n
        a.v_prev[i] = vp2.data_ptr() + 4 * i * n
    for i in range(6):
        a.ls[i] = lam2.data_ptr() + 4 * (3 + i) * n
    a.scratch, a.grad = scratch.data_ptr(), grad.data_ptr()
    _capi.check(L.pe_solver_adjoint_step(d._h, C.byref(a), 3, res.data_ptr(),
                                         C.c_void_p(t.cuda.current_stream().cuda_stream)))
    t.cuda.synchronize()
    return lam2.clone(), scratch.clone(), grad


@pytest.mark.parametrize("shape,order", [((5, 6, 4), 8), ((9, 17, 34), 8), ((20, 40, 96), 8), ((18, 49, 98), 4),
                                         ((17, 33, 66), 6)])
@pytest.mark.parametrize("mask", [False, True])
def test_pairs_equal_one_cell_kernels(shape, order, mask):
    from pefdtd import adjoint, fdtd
    from pefdtd.coeffs import taylor_coeffs
    from pefdtd.damping import sponge_axis_profiles
    rng = np.random.default_rng(6)
    n = int(np.prod(shape))
    m = 5
    Cm = rng.normal(size=(m, 6, 6)) * 2e8 + np.diag([14e9, 14e9, 15e9, 3e9, 3e9, 3.4e9])
    Cm = 0.5 * (Cm + Cm.transpose(0, 2, 1))
    cells = np.array([n // 2, n - 1], np.int64)
    d = fdtd.DeviceSolve(rng.integers(0, m, shape).astype(np.uint16), Cm.reshape(m, 36), rng.uniform(300, 920, m), 1e-4,
                         6e-9, taylor_coeffs(order), cells, np.ones(2), np.array([0, 2], np.int64), cells, np.ones(2),
                         record="vz", damped_record=True, sponge=sponge_axis_profiles(shape, 3),
                         damp_volume=rng.uniform(0.9, 1.0, shape) if mask else None)
    d.set_wavelet(np.zeros(8))
    t = d.torch
    L = adjoint._bind()
    f = lambda k, s: t.from_numpy((rng.normal(size=(k,) + shape) * s).astype(np.float32)).cuda()  # noqa: E731
    lam, vp, res = f(9, 1.0), f(3, 1e-3), t.ones((8, 1), device="cuda")
    scratch = t.zeros((33,) + shape, device="cuda")
    got = _step(d, L, lam, vp, scratch, res, 0)
    want = _step(d, L, lam, vp, scratch.zero_(), res, 1)
    assert t.equal(got[0], want[0])
    assert t.equal(got[1], want[1])
    # the same terms summed in another order: n products of either sign
    assert (got[2] - want[2]).abs().max() <= 1e-12 * want[2].abs().max()
    d.close()
