"""Two-level checkpoints of solves on side streams (GPU): the device memory that
a wave of gradients holds at its peak stays within the memory plan, although
the host issues all segments ahead of the device; and the gradients equal those
of one level to the order of their float64 atomic sums."""
import numpy as np
import pytest

from helpers import make_small

pytestmark = pytest.mark.gpu


def test_inner_checkpoints_stay_within_the_plan():
    import torch
    from pefdtd import adjoint
    shape, nt, K, m = (64, 96, 96), 240, 40, 8
    out = {}
    for inner in (None, m):
        probs, tables, dobs = [], [], []
        for k in range(2):
            p = make_small(nt=nt, shape=shape, n_grains=6, sponge=4, seed=70 + k)
            probs.append(adjoint.Problem(p["mats"], p["rho_t"], p["h"], p["dt"], p["coeffs"], p["src_pts"],
                                         p["rec_groups"], p["wavelet"], record="vz", sponge_width=p["sponge"],
                                         dtype="float32", checkpoint_every=K, inner_every=inner))
            C = p["Ct"].reshape(-1, 6, 6)
            tables.append(np.stack([C[:, i, j] for i in range(6) for j in range(i, 6)], 1).astype(float))
            dobs.append(np.zeros((nt, 1)))
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_stats()["active_bytes.all.current"]
        got = adjoint.misfit_gradients(probs, tables, dobs, plan=False)
        peak = torch.cuda.memory_stats()["active_bytes.all.peak"] - held
        plan = 2 * adjoint.adjoint_bytes(shape, nt, K, inner_every=inner)
        assert peak <= plan, (inner, peak, plan)
        out[inner] = got
    for (J, g), (J1, g1) in zip(out[m], out[None]):
        assert J == J1
        assert np.abs(g - g1).max() <= 1e-12 * np.abs(g1).max()
