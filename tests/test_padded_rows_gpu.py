"""Grids whose rows are not 16-byte multiples (GPU): runs of 8 and more steps
go through row-padded fields and the pair kernels, shorter ones step the
state in place with the one-column kernels. Both give the same bits, traces
and all nine fields, for every row remainder, on one tile and several, with
and without a damping volume, alone, in batches and in the adjoint's
recomputation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows of every remainder; one tile, tiles whose last column pair is half a
# pad, an interior tile, a single-cell last tile
SHAPES = [(9, 10, 5), (11, 17, 30), (12, 15, 31), (13, 33, 61), (10, 45, 99), (9, 40, 129)]


def _solve(shape, mask, record, variant, nt=45):
    from helpers import make_small
    from pefdtd import batch, fdtd
    rng = np.random.default_rng(5)
    nz, ny, nx = shape
    if min(shape) >= 12:
        p = make_small(nt=nt, shape=shape, n_grains=6, sponge=3, seed=7)
        sp = batch.spec_from_problem(p, record=record)
    else:   # too thin for a disk: random grains throughout
        p = make_small(nt=nt, shape=(16, 20, 24), n_grains=6, sponge=3, seed=7)
        sp = batch.spec_from_problem(p, record=record)
        sp["mats"] = rng.integers(0, len(sp["rho_t"]), shape).astype(np.uint16)
        sp["sponge"] = None
        cells = np.array([nx - 1, nz * ny * nx // 2, nz * ny * nx - 1], np.int64)
        sp.update(src_idx=cells[1:], src_w=np.ones(2), rec_idx=cells, rec_w=np.ones(3),
                  rec_off=np.array([0, 2, 3], np.int64))
    if mask:
        sp["damp_volume"] = rng.uniform(0.9, 1.0, shape).astype(np.float32)
    wav = sp.pop("wavelet")
    d = fdtd.DeviceSolve(**sp, dtype="float32", variant=variant, chunk_steps=20)
    d.set_wavelet(wav)
    d.state.copy_(d.torch.from_numpy(rng.normal(size=(9,) + shape).astype(np.float32) * 1e-6))
    return d, dict(sp, wavelet=wav)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("mask,record", [(False, "vz"), (True, "pressure")])
def test_padded_runs_equal_in_place_kernels(shape, mask, record):
    from pefdtd import batch
    want, sp = _solve(shape, mask, record, "column")
    got, _ = _solve(shape, mask, record, "tiled")
    start = want.state.clone()
    want.run(0, 45)
    for a, b in [(0, 30), (30, 33), (33, 45)]:   # padded (graph and rest), in place, padded again
        got.run(a, b)
    assert got.torch.equal(got.state, want.state)
    assert np.array_equal(got.traces_numpy(45), want.traces_numpy(45))
    # in a batch beside a solve with 16-byte rows, per-step launches and persistent
    other, sp4 = _solve((12, 24, 64), mask, record, "tiled")
    for persistent in (False, True):
        b = batch.BatchSolver([sp, sp4, sp], chunk_steps=20)
        b.set_persistent(persistent)
        for k in (0, 2):
            b.states[k].copy_(start)
        for a, e in [(0, 21), (21, 24), (24, 45)]:
            b.run(a, e)
        for k in (0, 2):
            assert b.torch.equal(b.states[k], want.state)
            assert np.array_equal(b.traces_numpy(45)[k], want.traces_numpy(45))
        b.close()
    for d in (want, got, other):
        d.close()


@pytest.mark.parametrize("shape", [(14, 21, 27), (13, 20, 34)])
def test_padded_adjoint_recomputation(shape):
    """Segments long enough to recompute through the padded fields (every=20)
    and segments stepped in place (every=5) give one gradient."""
    from helpers import make_small
    from pefdtd import adjoint
    p = make_small(nt=40, shape=shape, n_grains=4, sponge=3, seed=9)
    grads = []
    for every in (20, 5):
        prob = adjoint.Problem(p["mats"], p["rho_t"], p["h"], p["dt"], p["coeffs"], p["src_pts"], p["rec_groups"],
                               p["wavelet"], record="vz", sponge_width=p["sponge"], dtype="float32",
                               checkpoint_every=every)
        c21 = np.stack([p["Ct"].reshape(-1, 6, 6)[:, i, j] for i in range(6) for j in range(i, 6)], 1)
        a = prob.make_adjoint(c21)
        tr = a.forward()
        grads.append(a.backward(tr))
        a.solve.close()
    # the same terms; the float64 sums over cells are atomic, in any order
    scale = np.abs(grads[1]).max()
    assert np.abs(grads[0] - grads[1]).max() <= 1e-12 * scale
