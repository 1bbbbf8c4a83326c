"""Performance cases: the work a user of pefdtd has it do.

Pulse-echo problems on ice disks in a fluid couplant, as the drivers of this
repository build them: a disk of Voronoi grains centred in the grid, a sponge
at the faces, a transducer patch on the top ice face that is both source and
receiver. Grids, grain counts, sponges and record lengths come from the
benchmark workloads (disk_small 64x96x96, disk_prod 160x256x256), the
reference's stored ladder traces (136x338x338, fluid damping mask), the
inversion's disks (64x96x96 to 128x160x160) and the small parity grids of
the tests.

Kinds of case
  call      forward_fused_labels: host labels and c-axes in, traces out
  steps     DeviceSolve kept on the device: a state restored from a
            checkpoint, advanced nt steps (also FP64, per-cell media)
  batch     BatchSolver: the azimuths of a sweep advanced together
  gradient  AdjointSolve: checkpointed forward run and reverse sweep of one
            solve, the stiffness gradient out
  misfits   misfit_gradients: one evaluation of a fabric inversion
  autograd  Problem.traces under torch.autograd, grain angles to misfit
  records   traces.envelope / analyse over a sweep's records

exact() restates the scheme in plain torch, float64.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

_PKG = os.path.join(os.getcwd(), "pulse-echo-azimuthal-simulation_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from pefdtd import adjoint, fdtd, traces  # noqa: E402
from pefdtd.batch import BatchSolver  # noqa: E402

DEV = "cuda"
# order-8 dispersion-optimised staggered coefficients are inputs of a solve;
# these are the Taylor ones, which any order can state exactly
COEFFS = {2: [1.0], 4: [9 / 8, -1 / 24], 6: [75 / 64, -25 / 384, 3 / 640],
          8: [1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168]}
ICE = dict(C11=13.93e9, C33=15.01e9, C44=3.01e9, C12=7.08e9, C13=5.77e9)
RHO_ICE, C_FLUID, RHO_FLUID = 917.0, 1500.0, 300.0
SPONGE_STRENGTH = 0.09
VOIGT = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))
UPPER = [(i, j) for i in range(6) for j in range(i, 6)]


# ------------------------------------------------------------------ listed
def listed():
    return [
        # a smoke-size solve through the drop-in call: set-up and launch latency
        dict(name="call_tiny", kind="call", nz=20, ny=24, nx=28, grains=8, nt=60, sponge=3,
             record="pressure", order=8),
        # disk_small through the drop-in call, an azimuth of a plain sweep loop
        dict(name="call_disk_small", kind="call", nz=64, ny=96, nx=96, grains=50, nt=600, sponge=20,
             record="vz", order=8),
        # disk_prod, the configuration the single-solve throughput is quoted on
        dict(name="steps_disk_prod", kind="steps", nz=160, ny=256, nx=256, grains=500, nt=200, sponge=32,
             record="vz", order=8, dtype="float32", mask=False, media="table"),
        # the reference's ladder specimen: rows that are not 16-byte multiples, fluid damping volume
        dict(name="steps_ladder", kind="steps", nz=136, ny=338, nx=338, grains=100, nt=100, sponge=24,
             record="pressure", order=8, dtype="float32", mask=True, media="table"),
        # a cropped corridor: small, every side odd
        dict(name="steps_odd", kind="steps", nz=61, ny=83, nx=117, grains=40, nt=200, sponge=8,
             record="vz", order=8, dtype="float32", mask=True, media="table"),
        # the FP64 check run of a disk_small solve
        dict(name="steps_f64", kind="steps", nz=64, ny=96, nx=96, grains=50, nt=200, sponge=20,
             record="vz", order=8, dtype="float64", mask=False, media="table"),
        # a smoothly varying medium: every cell its own stiffness (the dense entry points)
        dict(name="steps_percell", kind="steps", nz=64, ny=96, nx=96, grains=50, nt=200, sponge=12,
             record="vz", order=8, dtype="float32", mask=False, media="cell"),
        # a dozen azimuths of an azimuth sweep in one batch
        dict(name="batch_sweep", kind="batch", solves=12, nz=64, ny=96, nx=96, grains=50, nt=200, sponge=20,
             record="vz", order=8, mask=True),
        # the gradient of one inversion-size solve, checkpoints every 200 steps as the drivers keep them
        dict(name="gradient_disk", kind="gradient", nz=96, ny=160, nx=160, grains=200, nt=160, sponge=12,
             record="vz", order=8, dtype="float32", every=200, mask=False),
        # one evaluation of a small fabric inversion: four azimuths of a 64x96x96 disk
        dict(name="misfits_inversion", kind="misfits", solves=4, nz=64, ny=96, nx=96, grains=50, nt=120,
             sponge=12, record="vz", order=8, dtype="float32", every=200),
        # autograd at its default precision, from grain angles to the misfit
        dict(name="autograd_f64", kind="autograd", nz=40, ny=72, nx=72, grains=30, nt=80, sponge=8,
             record="vz", order=8, every=50),
        # post-processing of a 36-azimuth sweep of full-length records
        dict(name="records_sweep", kind="records", solves=36, nt=6000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "steps", "steps", "steps", "batch", "gradient", "misfits", "autograd", "records"])
    if kind == "records":
        return dict(kind=kind, solves=_logint(rng, 1, 72), nt=_logint(rng, 1200, 8000))
    most = {"call": 3_000_000, "steps": 12_000_000, "batch": 1_200_000, "gradient": 3_000_000,
            "misfits": 700_000, "autograd": 300_000}[kind]
    c = dict(kind=kind)
    dtype = rng.choice(["float32", "float32", "float32", "float64"])
    media = rng.choice(["table", "table", "table", "cell"])
    if kind == "steps":
        most = {"cell": 800_000, "table": most}[media]
        most = min(most, 3_000_000) if dtype == "float64" else most
    while True:
        ny = _logint(rng, 24, 360)
        nx = ny if rng.random() < 0.5 else _logint(rng, 24, 360)
        nz = _logint(rng, 16, 170)
        if nz * ny * nx <= most:
            break
    cells = nz * ny * nx
    c.update(nz=nz, ny=ny, nx=nx, grains=_logint(rng, 4, 600), sponge=min(nz // 4, rng.choice([0, 4, 8, 12, 20, 32])),
             record=rng.choice(["vz", "vz", "pressure"]), order=rng.choice([8, 8, 8, 4]))
    steps = {"call": 1.2e9, "steps": 1.5e9, "batch": 1.2e8, "gradient": 2e8, "misfits": 4e7, "autograd": 2e7}[kind]
    most_nt = {"call": 600, "steps": 200, "batch": 200, "gradient": 160, "misfits": 120, "autograd": 80}[kind]
    c["nt"] = max(20, min(most_nt, int(steps / cells)))
    if kind in ("steps", "gradient"):
        c["dtype"] = dtype
    if kind == "misfits":
        c["dtype"] = "float32"
    if kind == "steps":
        c["media"] = media
    if kind in ("steps", "batch", "gradient"):
        c["mask"] = rng.random() < 0.4
    if kind in ("batch", "misfits"):
        c["solves"] = rng.randint(2, 12 if kind == "batch" else 4)
    if kind in ("gradient", "misfits", "autograd"):
        c["every"] = rng.choice([50, 200])
    return c


# ------------------------------------------------------------------ inputs
def _labels(shape, grains, rng):
    """(nz, ny, nx) int16 material indices on the device: 0 the fluid, 1 + g
    in the Voronoi cell of seed g inside a centred disk."""
    nz, ny, nx = shape
    R = 0.5 * min(ny, nx) - 3.0
    m = max(1, nz // 10)
    seeds = np.stack([rng.uniform(0, nz, grains), rng.uniform(-R, R, grains) + 0.5 * ny,
                      rng.uniform(-R, R, grains) + 0.5 * nx], 1)
    sd = torch.as_tensor(seeds, dtype=torch.float64, device=DEV)
    y = torch.arange(ny, dtype=torch.float64, device=DEV)[:, None]
    x = torch.arange(nx, dtype=torch.float64, device=DEV)[None, :]
    disk = (y - 0.5 * (ny - 1)) ** 2 + (x - 0.5 * (nx - 1)) ** 2 <= R * R
    out = torch.zeros(shape, dtype=torch.int16, device=DEV)
    plane = torch.stack(torch.broadcast_tensors(y, x), -1).reshape(-1, 2)
    d_yx = torch.cdist(plane, sd[:, 1:]).square()
    for z in range(m, nz - m):
        d = d_yx + (z - sd[:, 0]) ** 2
        out[z] = torch.where(disk, d.argmin(1).reshape(ny, nx) + 1, 0).to(torch.int16)
    return out, m


def _probe(mats, z0):
    """Cells of the transducer patch on the first ice plane."""
    _, ny, nx = mats.shape
    r = min(ny, nx) / 8.0
    iy, ix = np.nonzero((np.arange(ny)[:, None] - 0.5 * (ny - 1)) ** 2
                        + (np.arange(nx)[None, :] - 0.5 * (nx - 1)) ** 2 <= r * r)
    return [(z0, int(a), int(b)) for a, b in zip(iy, ix)]


def _axes(n, rng):
    a = rng.normal(size=(n, 3)) * (0.4, 0.4, 1.0)
    return a / np.linalg.norm(a, axis=1, keepdims=True)


def _stiffness(a):
    """(..., 6, 6) Voigt stiffness of ice with c-axis a (..., 3), torch
    float64: the invariant form of a transversely isotropic tensor."""
    eye = torch.eye(3, dtype=a.dtype, device=a.device)
    c66 = 0.5 * (ICE["C11"] - ICE["C12"])
    b = ICE["C11"] + ICE["C33"] - 2 * ICE["C13"] - 4 * ICE["C44"]
    rows = []
    for i, j in VOIGT:
        row = []
        for k, l in VOIGT:
            t = ICE["C12"] * eye[i, j] * eye[k, l] + c66 * (eye[i, k] * eye[j, l] + eye[i, l] * eye[j, k])
            t = t + (ICE["C13"] - ICE["C12"]) * (eye[i, j] * a[..., k] * a[..., l] + eye[k, l] * a[..., i] * a[..., j])
            t = t + (ICE["C44"] - c66) * (eye[i, k] * a[..., j] * a[..., l] + eye[i, l] * a[..., j] * a[..., k]
                                          + eye[j, k] * a[..., i] * a[..., l] + eye[j, l] * a[..., i] * a[..., k])
            row.append(t + b * a[..., i] * a[..., j] * a[..., k] * a[..., l])
        rows.append(torch.stack(row, -1))
    return torch.stack(rows, -2)


def _table(axes):
    """(n + 1, 6, 6) float64 torch table, row 0 the fluid."""
    a = torch.as_tensor(axes, dtype=torch.float64)
    fluid = torch.zeros(1, 6, 6, dtype=torch.float64, device=a.device)
    fluid[:, :3, :3] = RHO_FLUID * C_FLUID * C_FLUID
    return torch.cat([fluid, _stiffness(a)])


def _tapers(shape, width):
    if width <= 0:
        return None
    out = []
    for n in shape:
        p, w = np.ones(n), min(int(width), n // 2)
        if w > 0:
            t = np.exp(-SPONGE_STRENGTH * (1.0 - np.arange(w) / w) ** 2 * w)
            p[:w], p[n - w:] = t, t[::-1]
        out.append(p.astype(np.float32))
    return tuple(out)


def _burst(nt, dt, f0, cycles=3):
    t = np.arange(nt) * dt
    d = cycles / f0
    return np.where(t < d, np.sin(2 * np.pi * f0 * t) * 0.5 * (1 - np.cos(2 * np.pi * t / d)), 0.0)


def _problem(case, seed):
    """Everything of one solve that exists before the call, host and device."""
    shape = (case["nz"], case["ny"], case["nx"])
    rng = np.random.default_rng(seed)
    mats, z0 = _labels(shape, case["grains"], rng)
    h = 1e-4 if max(shape) > 128 else 2e-4
    dt = 0.3 * h / 4000.0
    axes = _axes(case["grains"], rng)
    pts = _probe(mats, z0)
    w = 1.0 / len(pts)
    # a burst a few tens of steps long, so that short runs carry it whole
    wav = _burst(case["nt"], dt, 1.0 / (24 * dt)) * rng.uniform(0.5, 1.5)
    mask = None
    if case.get("mask"):
        mask = torch.where(mats == 0, 0.97, 0.9998).to(torch.float32)
    p = dict(shape=shape, mats=mats, axes=axes, h=h, dt=dt, nt=case["nt"], coeffs=COEFFS[case["order"]],
             pts=pts, w=w, wavelet=wav, sponge=case["sponge"], tapers=_tapers(shape, case["sponge"]), mask=mask,
             record=case["record"])
    rho = np.full(case["grains"] + 1, RHO_ICE)
    rho[0] = RHO_FLUID
    p["rho_t"] = rho
    idx = np.array([(a * shape[1] + b) * shape[2] + c for a, b, c in pts], np.int64)
    p["idx"] = idx
    p["wts"] = np.full(len(idx), w)
    return p


def _field(shape, seed, dtype):
    """A filled wavefield: smooth random v and s, at a pulse's amplitudes."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    small = [max(2, n // 5) for n in shape]
    a = torch.randn([1, 9] + small, generator=g, device=DEV, dtype=torch.float32)
    f = torch.nn.functional.interpolate(a, size=shape, mode="trilinear", align_corners=True)[0]
    f[:3] *= 3e-10
    f[3:] *= 1e-3
    return f.to(dtype).contiguous()


def _cell_media(p):
    """Per-cell medium: the c-axis turns smoothly through the ice."""
    nz, ny, nx = p["shape"]
    z, y, x = torch.meshgrid(*[torch.linspace(0, 1, n, dtype=torch.float64, device=DEV) for n in p["shape"]],
                             indexing="ij")
    k = float(p["axes"][0, 0])
    th, ph = 0.6 + 0.5 * torch.sin(3.0 * x + 2.0 * y + k), 2.0 * z + y + k
    a = torch.stack([th.sin() * ph.cos(), th.sin() * ph.sin(), th.cos()], -1).reshape(-1, 3)
    C = _stiffness(a)
    fluid = (p["mats"] == 0).reshape(-1)
    C[fluid] = 0.0
    C[fluid, :3, :3] = RHO_FLUID * C_FLUID * C_FLUID
    C = 0.5 * (C + C.transpose(-1, -2))
    rho = torch.where(fluid, RHO_FLUID, RHO_ICE).to(torch.float64)
    return C.reshape(-1, 36), rho


def _np_dtype(case):
    return np.float64 if case.get("dtype") == "float64" else np.float32


def _solve_args(p, case):
    """Positional arguments of DeviceSolve (keywords of a batch spec)."""
    nd = _np_dtype(case)
    if case.get("media") == "cell":
        C, rho = _cell_media(p)
        Ct, rho_t = C.cpu().numpy().astype(nd), rho.cpu().numpy().astype(nd)
        mats = np.zeros(p["shape"], np.uint16)
    else:
        Ct = _table(p["axes"]).reshape(-1, 36).numpy().astype(nd)
        rho_t, mats = p["rho_t"].astype(nd), p["mats"].cpu().numpy().astype(np.uint16)
    return dict(mats=mats, Ct=Ct, rho_t=rho_t, h=p["h"], dt=p["dt"], coeffs=np.array(p["coeffs"]), src_idx=p["idx"],
                src_w=p["wts"].astype(nd), rec_off=np.array([0, len(p["idx"])], np.int64), rec_idx=p["idx"],
                rec_w=p["wts"].astype(nd), record=p["record"], damped_record=True, sponge=p["tapers"],
                damp_volume=None if p["mask"] is None else p["mask"].cpu().numpy())


def _adjoint_problem(p, case):
    return adjoint.Problem(p["mats"].cpu().numpy(), p["rho_t"], p["h"], p["dt"], p["coeffs"],
                           [(q, p["w"]) for q in p["pts"]], [(p["pts"], p["wts"])], p["wavelet"], record=p["record"],
                           sponge_width=p["sponge"], damp_mask=None if p["mask"] is None else p["mask"].cpu().numpy(),
                           dtype=case.get("dtype", "float64"), checkpoint_every=case["every"])


def _observed(p):
    """A recorded trace to fit: a burst at the record's amplitude."""
    amp = 1e-10 if p["record"] == "vz" else 1e-4
    return amp * _burst(p["nt"], p["dt"], 1.0 / (30 * p["dt"]), 2)[:, None]


def _table21(axes):
    C = _table(axes)
    return torch.stack([C[:, i, j] for i, j in UPPER], -1)


def _angles(axes):
    return np.arccos(np.clip(axes[:, 2], -1, 1)), np.arctan2(axes[:, 1], axes[:, 0])


def _sub_seed(seed, k):
    return seed * 64 + k


def _records(case, seed):
    """Records of a sweep: a direct burst, an echo and a decaying coda."""
    rng = np.random.default_rng(seed)
    n = case["nt"]
    dt = 6.0e-5 / n
    t = np.arange(n) * dt
    out = []
    for _ in range(case["solves"]):
        te = 52e-6 + rng.uniform(-0.5e-6, 0.5e-6)
        f = 2e6 * rng.uniform(0.8, 1.2)
        x = np.exp(-((t - 2e-6) * f / 2) ** 2) * np.sin(2 * np.pi * f * t)
        x += 0.3 * np.exp(-((t - te) * f / 2) ** 2) * np.sin(2 * np.pi * f * (t - te))
        x += 0.02 * np.convolve(rng.normal(size=n), np.hanning(9), "same") * np.exp(-t / 2e-5)
        out.append((x * 1e-9).astype(np.float32))
    return out, dt


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "records":
        recs, dt = _records(case, seed)
        return dict(case=case, recs=recs, dt=dt)
    if kind in ("batch", "misfits"):
        ps = [_problem(case, _sub_seed(seed, k)) for k in range(case["solves"])]
        if kind == "misfits":
            return dict(case=case, problems=[_adjoint_problem(p, case) for p in ps],
                        tables=[_table21(p["axes"]).numpy() for p in ps], dobs=[_observed(p) for p in ps])
        b = BatchSolver([dict(_solve_args(p, case), wavelet=p["wavelet"]) for p in ps])
        b.set_persistent(True)
        return dict(case=case, batch=b, start=[_field(p["shape"], _sub_seed(seed, k), torch.float32)
                                               for k, p in enumerate(ps)])
    p = _problem(case, seed)
    if kind == "call":
        return dict(case=case, lab=p["mats"].cpu().numpy().astype(np.int32) - 1, axes=p["axes"], p=p,
                    src=[(q, p["w"]) for q in p["pts"]], rec=[(p["pts"], p["wts"])])
    if kind == "autograd":
        th, ph = _angles(p["axes"])
        return dict(case=case, problem=_adjoint_problem(p, case), theta=th, phi=ph,
                    dobs=torch.as_tensor(_observed(p)))
    solve = fdtd.DeviceSolve(**_solve_args(p, case), dtype=case["dtype"],
                             variant="dense" if case.get("media") == "cell" else "tiled")
    solve.set_wavelet(p["wavelet"])
    if kind == "gradient":
        return dict(case=case, adj=adjoint.AdjointSolve(solve, case["every"]),
                    dobs=torch.as_tensor(_observed(p), device=DEV).to(solve.tdt))
    return dict(case=case, solve=solve, start=_field(p["shape"], seed, solve.tdt))


# ------------------------------------------------------------------ run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "records":
        return {"env": traces.envelope(s["recs"]), "figures": np.array(traces.analyse(s["recs"], s["dt"]))}
    if kind == "call":
        p = s["p"]
        return fdtd.forward_fused_labels(s["lab"], s["axes"], p["h"], p["dt"], p["nt"], s["src"], p["wavelet"],
                                         s["rec"], coeffs=p["coeffs"], sponge_width=p["sponge"],
                                         sponge_strength=SPONGE_STRENGTH, c_couplant=C_FLUID, rho_couplant=RHO_FLUID,
                                         record=p["record"], damped_record=True)
    if kind == "steps":
        d = s["solve"]
        d.state.copy_(s["start"])
        d.run(0, case["nt"])
        return {"state": d.state, "traces": d.traces}
    if kind == "batch":
        b = s["batch"]
        for st, a in zip(b.states, s["start"]):
            st.copy_(a)
        b.run(0, case["nt"])
        return {"states": list(b.states), "traces": list(b.traces)}
    if kind == "gradient":
        tr = s["adj"].forward()
        return {"traces": tr, "grad": s["adj"].backward(tr - s["dobs"])}
    if kind == "misfits":
        got = adjoint.misfit_gradients(s["problems"], s["tables"], s["dobs"])
        return {"J": [j for j, _ in got], "grad": [g for _, g in got]}
    th = torch.tensor(s["theta"], requires_grad=True)
    ph = torch.tensor(s["phi"], requires_grad=True)
    tr = s["problem"].traces(adjoint.ice_table21(th, ph, C_FLUID, RHO_FLUID, dict(ICE, rho=RHO_ICE)))
    J = 0.5 * ((tr - s["dobs"]) ** 2).sum()
    J.backward()
    return {"traces": tr.detach(), "theta": th.grad, "phi": ph.grad}


# ------------------------------------------------------------------ work
def work(case):
    if case["kind"] == "records":
        n = case["solves"] * case["nt"]
        return {"bytes": 4 * n + 8 * n, "flops": 5 * n * math.log2(case["nt"]) * 2}
    es = 8 if case.get("dtype") == "float64" or case["kind"] == "autograd" else 4
    cells = case["nz"] * case["ny"] * case["nx"] * case.get("solves", 1)
    # a step reads and writes nine fields and reads the label (or 22 medium values) of each cell
    per = 18 * es + (22 * es if case.get("media") == "cell" else 2) + (4 if case.get("mask") else 0)
    flops = 9 * 3 * case["order"] // 2 * 2 + 6 + 18 * 4 + 36 * 2 + 6 * 3 + 3 * 5
    passes = 1
    if case["kind"] in ("gradient", "misfits", "autograd"):
        # forward, recomputation, and a reverse step over v, the adjoint state and the label
        per, flops = 2 * per + (3 + 18) * es + 2, 2 * flops + 2 * flops
    n = cells * case["nt"] * passes
    return {"bytes": n * per, "flops": n * flops}


# ------------------------------------------------------------------ exact
def _tap(f, axis, c, forward):
    n = f.shape[axis]
    out = torch.zeros_like(f)
    for j, cj in enumerate(c):
        m = n - 2 * j - 1
        if m > 0:
            out.narrow(axis, j if forward else j + 1, m).add_(
                f.narrow(axis, 2 * j + 1, m) - f.narrow(axis, 0, m), alpha=cj)
    return out


def _half(f, axis, d):
    """Mean of f and its neighbour at +-1 along axis, zero where there is none."""
    n = f.shape[axis]
    out = torch.zeros_like(f)
    if n > 1:
        out.narrow(axis, 0 if d > 0 else 1, n - 1).copy_(0.5 * (f.narrow(axis, 0, n - 1) + f.narrow(axis, 1, n - 1)))
    return out


_POS = ((0, 0, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1))   # centre, yz, xz, xy as (z, y, x) half cells
_AT = (0, 0, 0, 1, 2, 3)


def _move(g, J, P):
    for axis in range(3):
        d = _POS[P][axis] - _POS[_AT[J]][axis]
        if d:
            g = _half(g, axis, d)
    return g


def _face(rho, axis):
    out = rho.clone()
    n = rho.shape[axis]
    if n > 1:
        out.narrow(axis, 0, n - 1).copy_(0.5 * (rho.narrow(axis, 0, n - 1) + rho.narrow(axis, 1, n - 1)))
    return out


class _Exact:
    """The scheme in plain torch float64, one step at a time."""

    def __init__(self, p, C, rho):
        """C: {(I, J): map or per-cell tensor} for I <= J; rho: per cell."""
        self.p, self.C = p, C
        self.faces = [_face(rho, a) for a in (2, 1, 0)]
        d = torch.ones(p["shape"], dtype=torch.float64, device=DEV)
        if p["tapers"] is not None:
            z, y, x = [torch.as_tensor(t, device=DEV) for t in p["tapers"]]
            d = ((z[:, None, None] * y[None, :, None]) * x[None, None, :]).double()
        if p["mask"] is not None:
            d = (d.float() * p["mask"]).double()
        self.damp = d
        self.idx = torch.as_tensor(p["idx"], device=DEV)
        self.wts = torch.as_tensor(p["wts"], device=DEV)

    def step(self, n, *f):
        p, c = self.p, self.p["coeffs"]
        vx, vy, vz = f[:3]
        ih = 1.0 / p["h"]
        F, B = (lambda a, ax: _tap(a, ax, c, True)), (lambda a, ax: _tap(a, ax, c, False))
        g = [B(vx, 2) * ih, B(vy, 1) * ih, B(vz, 0) * ih, (F(vz, 1) + F(vy, 0)) * ih, (F(vz, 2) + F(vx, 0)) * ih,
             (F(vy, 2) + F(vx, 1)) * ih]
        s = []
        for P in range(4):
            q = [_move(g[J], J, P) for J in range(6)]
            for i in [i for i in range(6) if _AT[i] == P]:
                acc = 0.0
                for J in range(6):
                    acc = acc + self.C[(min(i, J), max(i, J))] * q[J]
                s.append(f[3 + i] * self.damp + p["dt"] * acc)
        src = torch.zeros(p["shape"], dtype=torch.float64, device=DEV)
        src.view(-1)[self.idx] = float(p["wavelet"][n]) * self.wts
        s = [a + src if i < 3 else a for i, a in enumerate(s)]
        k = p["dt"] / p["h"]
        ax = F(s[0], 2) + B(s[5], 1) + B(s[4], 0)
        ay = B(s[5], 2) + F(s[1], 1) + B(s[3], 0)
        az = B(s[4], 2) + B(s[3], 1) + F(s[2], 0)
        v = [(a + k * b / r) * self.damp for a, b, r in zip((vx, vy, vz), (ax, ay, az), self.faces)]
        if p["record"] == "vz":
            t = (v[2].reshape(-1)[self.idx] * self.wts).sum()
        else:
            t = (-(((s[0] + s[1] + s[2]) * self.damp).reshape(-1)[self.idx]) / 3.0 * self.wts).sum()
        return tuple(v) + tuple(s) + (t,)

    def run(self, f, grad=False):
        f, tr = tuple(f), []
        for n in range(self.p["nt"]):
            if grad:
                out = torch.utils.checkpoint.checkpoint(self.step, n, *f, use_reentrant=False)
            else:
                out = self.step(n, *f)
            f, t = out[:9], out[9]
            tr.append(t)
        return f, torch.stack(tr)[:, None]


def _maps(p, c21):
    """{(I, J): map} from a (n_mat, 21) table, and the density."""
    m = p["mats"].long().reshape(-1)
    c = c21.to(DEV)
    C = {ij: c[:, k].index_select(0, m).reshape(p["shape"]) for k, ij in enumerate(UPPER)}
    return C, torch.as_tensor(p["rho_t"], device=DEV).index_select(0, m).reshape(p["shape"])


def _exact_solve(p, case):
    if case.get("media") == "cell":
        C, rho = _cell_media(p)
        return _Exact(p, {(i, j): C[:, 6 * i + j].reshape(p["shape"]) for i, j in UPPER}, rho.reshape(p["shape"]))
    return _Exact(p, *_maps(p, _table21(p["axes"])))


def _zeros(p):
    return [torch.zeros(p["shape"], dtype=torch.float64, device=DEV) for _ in range(9)]


def _exact_gradient(p, c21):
    """(traces, J, dJ/dc21) for J = 0.5 ||traces - observed||^2."""
    c = c21.detach().clone().requires_grad_(True)
    E = _Exact(p, *_maps(p, c))
    _, tr = E.run(_zeros(p), grad=True)
    r = tr - torch.as_tensor(_observed(p), device=DEV)
    J = 0.5 * (r * r).sum()
    J.backward()
    return tr.detach(), float(J.detach()), c.grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "records":
        recs, _ = _records(case, seed)
        env = []
        for x in recs:
            n = len(x)
            X = torch.fft.fft(torch.as_tensor(x, device=DEV).double())
            h = torch.zeros(n, dtype=torch.float64, device=DEV)
            h[0] = 1
            h[1:(n + 1) // 2] = 2
            if n % 2 == 0:
                h[n // 2] = 1
            env.append(torch.fft.ifft(X * h).abs().cpu().numpy())
        return {"env": env, "figures": None}
    if kind in ("batch", "misfits"):
        ps = [_problem(case, _sub_seed(seed, k)) for k in range(case["solves"])]
        if kind == "misfits":
            got = [_exact_gradient(p, _table21(p["axes"])) for p in ps]
            return {"J": [j for _, j, _ in got], "grad": [g.numpy() for _, _, g in got]}
        with torch.no_grad():
            got = [_exact_solve(p, case).run(_field(p["shape"], _sub_seed(seed, k), torch.float32).double())
                   for k, p in enumerate(ps)]
        return {"states": [torch.stack(f) for f, _ in got], "traces": [t for _, t in got]}
    p = _problem(case, seed)
    if kind == "gradient":
        tr, _, g = _exact_gradient(p, _table21(p["axes"]))
        return {"traces": tr, "grad": g.numpy()}
    if kind == "autograd":
        th, ph = [torch.tensor(a, requires_grad=True) for a in _angles(p["axes"])]
        c21 = _table21(torch.stack([th.sin() * ph.cos(), th.sin() * ph.sin(), th.cos()], -1))
        tr, _, g = _exact_gradient(p, c21)
        (c21 * g).sum().backward()
        return {"traces": tr.cpu(), "theta": th.grad, "phi": ph.grad}
    with torch.no_grad():
        if kind == "call":
            return _exact_solve(p, case).run(_zeros(p))[1]
        f, tr = _exact_solve(p, case).run(_field(p["shape"], seed, torch.float64 if case["dtype"] == "float64"
                                                 else torch.float32).double())
    return {"state": torch.stack(f), "traces": tr}
