"""Performance cases of the library's public entry points.

Every case is one call (or one update) that a program built on this library makes, at sizes taken
from the workload definitions (mcmatlab_b200/configs.py), the tests and the benchmark, or generic
ones. All entry points take and return host arrays, as MATLAB's MEX calls do, so a pass runs from
host inputs to host outputs; only the resident heat state keeps its grids on the device between
calls, as model.simulateHeatDistribution does.

Kinds of cases:

* mc        one photon-packet transport run (native.mc_run): the heart of model.runMonteCarlo
* mc_batch  several models in one launch (native.mc_run_batch): parameter sweeps
* mc_grad   transport with derivatives (native.mc_grad): fitting optical properties
* heat      one update of a heat simulation: grids resident on the device (native.HeatState), or
            the whole call from host grids (native.heat_forward)
* adjoint   a heat run with its gradients (native.heat_adjoint): treatment planning
* normals   interface normals of a geometry with several refractive indices
            (native.interface_normals): before every run with mismatched interfaces
* binning   sub-media binning of one medium whose properties depend on the local fluence rate,
            temperature or damage (native.downsample_params): before such a run

Outputs that the library computes in single precision and hands out in FP64 containers (sensor
temperatures, perturbation derivatives, the objective and dJ/dc) are returned as float32.
"""
import math

import numpy as np
import torch

from mcmatlab_b200 import mexargs, native, prep
from mcmatlab_b200 import model as mm

GAS_R = 8.3144598
ZERO_C = 273.15
MC_STEPS = 150   # propagation sub-steps of an ordinary packet in tissue
MC_FLOPS = 60    # floating-point operations of a sub-step with its share of a scattering event


def listed():
    return [
        # the smallest transport call: a quick look at a coarse grid, or one of many calls of an
        # optimisation loop; launches, copies and the longest packet count here
        dict(name="mc_preview", kind="mc", nx=30, ny=30, nz=30, packets=10000, matched=False, source="pencil",
             boundary=1, wavelengths=1, collector="none", far=0),
        # the ordinary transport call: the 100^3 skin cube with refraction, 1e6 packets
        dict(name="mc_cube", kind="mc", nx=100, ny=100, nz=100, packets=1000000, matched=False, source="pencil",
             boundary=1, wavelengths=1, collector="none", far=0),
        # a spectroscopy set-up: ragged grid, cyclic sides, two wavelengths, Gaussian beam, a
        # time-resolved fibre and the far field
        dict(name="mc_fibre", kind="mc", nx=117, ny=83, nz=141, packets=400000, matched=False, source="gaussian",
             boundary=3, wavelengths=2, collector="fibre", far=40),
        # a sweep of six models of different sizes in one launch
        dict(name="mc_sweep", kind="mc_batch", models=6, nx=96, ny=101, nz=88, packets=100000, matched=False),
        # one evaluation of a fit: derivatives for every medium of a 128^3 cube
        dict(name="mc_fit", kind="mc_grad", nx=128, ny=128, nz=128, packets=1000000, bins=32, matched=False),
        # the smallest heat call: a coarse ragged grid from host arrays, few steps, with sensors
        dict(name="heat_preview", kind="heat", nx=31, ny=27, nz=40, steps=20, light=True, damage=True, sinked=False,
             media=3, factor=1.5, sensors=3, resident=False),
        # the ordinary heat update: the 100^3 cube, light on, damage, grids resident
        dict(name="heat_cube", kind="heat", nx=100, ny=100, nz=100, steps=100, light=True, damage=True, sinked=False,
             media=4, factor=0.9, sensors=2, resident=True),
        # the largest heat update: 18 million voxels cooling between heat-sinked faces
        dict(name="heat_large", kind="heat", nx=300, ny=300, nz=200, steps=150, light=False, damage=False, sinked=True,
             media=4, factor=0.9, sensors=0, resident=True),
        # a deep, narrow grid with one axis above 512 voxels and large time steps, from host arrays
        dict(name="heat_deep", kind="heat", nx=45, ny=37, nz=640, steps=60, light=True, damage=False, sinked=False,
             media=4, factor=15.0, sensors=1, resident=False),
        # gradients of damage and peak temperature over a heat run
        dict(name="heat_adjoint", kind="adjoint", nx=120, ny=111, nz=90, steps=40, sinked=False, media=4, factor=0.9,
             store_all=False),
        # smoothed interface normals of a 100 x 100 x 120 tissue block
        dict(name="normals", kind="normals", nx=100, ny=100, nz=120, smooth=True, media=4),
        # 300 000 voxels of a temperature-dependent medium into 40 sub-media
        dict(name="binning", kind="binning", n=300000, bins=40),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["mc"] * 4 + ["mc_batch", "mc_grad"] + ["heat"] * 5 + ["adjoint", "normals", "binning"])
    if kind == "mc":
        boundary = rng.choice([1, 1, 2, 3])
        return dict(kind=kind, nx=_logint(rng, 20, 160), ny=_logint(rng, 20, 160), nz=_logint(rng, 20, 160),
                    packets=_logint(rng, 5000, 1000000), matched=rng.random() < 0.3,
                    source=rng.choice(["pencil", "gaussian", "isotropic", "plane"]), boundary=boundary,
                    wavelengths=rng.choice([1, 1, 2, 3]), collector=rng.choice(["none", "fibre", "lens"]),
                    far=rng.choice([0, 0, 30]))
    if kind == "mc_batch":
        return dict(kind=kind, models=rng.randint(2, 8), nx=_logint(rng, 24, 110), ny=_logint(rng, 24, 110),
                    nz=_logint(rng, 24, 110), packets=_logint(rng, 5000, 100000), matched=rng.random() < 0.5)
    if kind == "mc_grad":
        return dict(kind=kind, nx=_logint(rng, 32, 128), ny=_logint(rng, 32, 128), nz=_logint(rng, 32, 128),
                    packets=_logint(rng, 20000, 1000000), bins=rng.choice([16, 32, 50]), matched=rng.random() < 0.3)
    if kind == "heat":
        nx, ny, nz = _logint(rng, 24, 300), _logint(rng, 24, 300), _logint(rng, 24, 300)
        if rng.random() < 0.1:
            nx, ny, nz = _logint(rng, 24, 60), _logint(rng, 24, 60), _logint(rng, 513, 800)
        damage = rng.random() < 0.6
        most = max(1, min(100 if damage else 300, 1000000000 // (nx * ny * nz)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_logint(rng, min(10, most), most), light=rng.random() < 0.6,
                    damage=damage, sinked=rng.random() < 0.4, media=rng.randint(2, 8),
                    factor=rng.choice([0.9, 1.5, 1.5, 15.0]), sensors=rng.choice([0, 1, 4]), resident=rng.random() < 0.6)
    if kind == "adjoint":
        return dict(kind=kind, nx=_logint(rng, 24, 120), ny=_logint(rng, 24, 120), nz=_logint(rng, 24, 100),
                    steps=rng.randint(12, 48), sinked=rng.random() < 0.4, media=rng.randint(2, 6),
                    factor=rng.choice([0.9, 1.5]), store_all=rng.random() < 0.3)
    if kind == "normals":
        return dict(kind=kind, nx=_logint(rng, 24, 110), ny=_logint(rng, 24, 110), nz=_logint(rng, 24, 110),
                    smooth=rng.random() < 0.7, media=rng.randint(2, 5))
    return dict(kind=kind, n=_logint(rng, 2000, 500000), bins=rng.randint(5, 60))


# ------------------------------------------------------------------------------------------------
# Photon transport
# ------------------------------------------------------------------------------------------------

def _skin_model(nx, ny, nz, packets, matched, seed):
    """A layered skin block 1 mm wide: air, epidermis, dermis and a vessel along y, with optical
    properties and layer depths that vary with the seed."""
    rng = np.random.default_rng(seed)
    mua = np.array([1e-8, 10.0, 1.0, 200.0]) * np.array([1.0, *rng.uniform(0.7, 1.4, 3)])
    mus = np.array([1e-8, 150.0, 100.0, 100.0]) * np.array([1.0, *rng.uniform(0.8, 1.2, 3)])
    depth, thick = rng.uniform(0.008, 0.012), rng.uniform(0.005, 0.008)
    vx, vz, vr = rng.uniform(-0.004, 0.004), rng.uniform(0.037, 0.043), rng.uniform(0.008, 0.012)

    def media(params):
        # shorter wavelengths are absorbed and scattered more strongly
        names = ("air", "epidermis", "dermis", "vessel")
        return [mm.mediumProperties(name=names[k],
                                    mua=(lambda w, k=k: float(mua[k] * (532.0 / w) ** (1.0 if k else 0.0))),
                                    mus=(lambda w, k=k: float(mus[k] * (532.0 / w) ** (0.8 if k else 0.0))),
                                    g=1.0 if k == 0 else 0.9, n=1.0 if k == 0 else 1.3) for k in range(4)]

    def geom(X, Y, Z, params):
        M = np.full(X.shape, 3.0)
        M[Z < depth + thick] = 2
        M[Z < depth] = 1
        M[(X - vx) ** 2 + (Z - vz) ** 2 < vr ** 2] = 4
        return M

    m = mm.model()
    m.G.nx, m.G.ny, m.G.nz = nx, ny, nz
    m.G.Lx = m.G.Ly = m.G.Lz = 0.1
    m.G.mediaPropertiesFunc, m.G.geomFunc = media, geom
    m.MC.nPhotonsRequested = float(packets)
    m.MC.seed = seed
    m.MC.matchedInterfaces = matched
    m.MC.wavelength = 532.0
    m.MC.boundaryType = 1
    m.MC.silentMode = True
    return m


def _mc_input(case, seed):
    m = _skin_model(case["nx"], case["ny"], case["nz"], case["packets"], case["matched"], seed)
    MC = m.MC
    MC.boundaryType = case["boundary"]
    MC.farFieldRes = case["far"]
    if case["wavelengths"] > 1:
        MC.wavelength = np.linspace(532.0, 700.0, case["wavelengths"])
        MC.spectrumFunc = lambda w: 1.0
    LS = MC.lightSource
    if case["source"] == "gaussian":
        LS.sourceType = 4
        LS.FPID.radialDistr, LS.FPID.radialWidth = 1, 0.01
        LS.AID.radialDistr, LS.AID.radialWidth = 1, 0.05
    elif case["source"] == "isotropic":
        LS.sourceType = 1
        LS.zFocus = 0.03
        LS.emitterLength = 0.02
    elif case["source"] == "plane":
        LS.sourceType = 2
    else:
        LS.sourceType = 0
    if case["collector"] != "none":
        MC.useLightCollector = True
        LC = MC.lightCollector
        LC.x, LC.y, LC.z, LC.theta, LC.phi = 0.0, 0.0, -0.05, 0.0, math.pi / 2
        LC.tStart, LC.tEnd, LC.nTimeBins = 0.0, 2e-11, 60
        if case["collector"] == "fibre":
            LC.f, LC.diam, LC.NA, LC.res = math.inf, 0.1, 0.5, 1
        else:
            LC.f, LC.diam, LC.fieldSize, LC.res, LC.nTimeBins = 0.1, 0.1, 0.1, 40, 0
    m.G.updateGeometry()
    return mexargs.prepare_mc(m, 1, normals=native.interface_normals)


def _mc_output(out):
    keep = [k for k in sorted(out) if k.startswith("NI_") or k in ("NFR", "image", "farField")]
    return {**{k: out[k] for k in keep}, "nPhotons": int(out["nPhotons"]), "nPhotonsCollected": int(out["nPhotonsCollected"])}


def _mc_bytes(nx, ny, nz, nL, matched, far, collector, boundary):
    L = nx * ny * nz
    b = L * (1 + (0 if matched else 8)) + 4 * L * nL
    b += 4 * nL * (far * far + {"none": 0, "fibre": 62, "lens": 1600}[collector])
    faces = {1: 2 * (nx * ny + nx * nz + ny * nz), 2: 25 * nx * ny, 3: 2 * nx * ny}[boundary]
    return b + 4 * nL * faces


# ------------------------------------------------------------------------------------------------
# Heat
# ------------------------------------------------------------------------------------------------

def _heat_input(case, seed):
    """A heated block: `media` - 1 layers along z and an ellipsoid (the only medium that is
    damaged), a beam-like heat source and a warm, slightly uneven start temperature."""
    rng = np.random.default_rng(seed)
    nx, ny, nz, nM = case["nx"], case["ny"], case["nz"], case["media"]
    d = (0.1 / 100, 0.1 / 100, 0.1 / 100)
    x, y = (np.arange(nx) + 0.5) / nx - 0.5, (np.arange(ny) + 0.5) / ny - 0.5
    z = (np.arange(nz) + 0.5) / nz
    TC, VHC = rng.uniform(0.002, 0.006, nM), rng.uniform(3.0, 4.2, nM)
    if nM > 2:
        TC[0], VHC[0] = 0.00026, 0.0012  # air on top
    top = np.sort(rng.uniform(0.08, 0.9, max(nM - 2, 0)))
    layer = np.searchsorted(top, z).astype(np.uint8)
    c = (rng.uniform(-0.1, 0.1), rng.uniform(-0.1, 0.1), rng.uniform(0.4, 0.6))
    r = rng.uniform(0.12, 0.25, 3)
    M = np.empty((nx, ny, nz), dtype=np.uint8, order="F")
    M[...] = layer[None, None, :] + 1
    q = (((x - c[0]) / r[0]) ** 2)[:, None, None] + (((y - c[1]) / r[1]) ** 2)[None, :, None] + (((z - c[2]) / r[2]) ** 2)[None, None, :]
    inside = q < 1
    M[inside] = nM
    beam = (np.exp(-(x / 0.2) ** 2)[:, None, None] * np.exp(-(y / 0.2) ** 2)[None, :, None] * np.exp(-z / 0.4)[None, None, :])
    NA = 2000.0 * beam * np.where(VHC > 0.1, VHC, 0.0)[M - 1]  # 2000 K/s in the beam; the air absorbs nothing
    cond, Q = prep.calc_dTdt_arrays(VHC, TC, *d, NA, 1.0, M)
    dt = case["factor"] * float(np.min(VHC / TC)) / (2 * sum(1 / s ** 2 for s in d))
    A, E = np.zeros(nM), np.zeros(nM)
    A[-1], E[-1] = 7.6e66, 4.48e5
    li = w = None
    if case.get("sensors"):
        ax = [(np.arange(n) + 0.5) * s for n, s in zip((nx, ny, nz), d)]
        li, w = prep.convert_temp_sensor_pos(rng.uniform(0.1, 0.9, (case["sensors"], 3)) * [a[-1] for a in ax], *ax)
    hp = mexargs.heat_mex_params(M, A, E, cond, Q, True, int(case["sinked"]), li, w, case.get("light", True), case["steps"], dt)
    a, b, e = rng.uniform(2.0, 6.0, 3)
    T0 = np.empty((nx, ny, nz), dtype=np.float32, order="F")
    T0[...] = 48.0 + 2.0 * (np.sin(a * x + 1)[:, None, None] * np.cos(b * y)[None, :, None] * np.sin(e * z)[None, None, :])
    return dict(T0=T0, hp=hp, M=M, inside=inside)


def _work_heat(case):
    L = case["nx"] * case["ny"] * case["nz"]
    # per step: T read and written, the medium, the source while the light is on, the damage of
    # the ellipsoid's voxels; about 50 operations for the stencils and the three line solves
    per = 9 + (4 if case.get("light", True) else 0)
    return {"bytes": float(L * per * case["steps"] + 12 * L), "flops": 50.0 * L * case["steps"]}


def _exact_heat(case, seed):
    """The Douglas-Gunn step in FP64: per axis a tridiagonal solve along whole lines."""
    s = _heat_input(case, seed)
    hp = s["hp"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = torch.from_numpy(np.ascontiguousarray(s["T0"])).to(dev, torch.float64)
    M = torch.from_numpy(np.ascontiguousarray(s["M"]).astype(np.int64) - 1).to(dev)
    Q = torch.from_numpy(np.ascontiguousarray(hp["dTdt_abs"])).to(dev, torch.float64).reshape(T.shape)
    cond = torch.from_numpy(np.ascontiguousarray(hp["dTdtperdeltaT"])).to(dev, torch.float64)
    A = torch.from_numpy(hp["A"].ravel()).to(dev)
    E = torch.from_numpy(hp["E"].ravel()).to(dev)
    dt, nt, nM = hp["dt"], int(hp["steps"]), len(A)
    held = torch.zeros_like(M, dtype=torch.bool)
    if hp["heatBoundaryType"]:
        for ax in range(3):
            held.narrow(ax, 0, 1).fill_(True)
            held.narrow(ax, T.shape[ax] - 1, 1).fill_(True)
    free = (~held).to(torch.float64)
    axes = []
    for ax in range(3):  # the axis first: couplings of row i to its lower (a) and upper (b) neighbour
        Mt, Ft = M.movedim(ax, 0).contiguous(), free.movedim(ax, 0).contiguous()
        a, b = torch.zeros_like(Ft), torch.zeros_like(Ft)
        a[1:] = cond[Mt[1:], Mt[:-1], ax] * Ft[1:]
        b[:-1] = cond[Mt[:-1], Mt[1:], ax] * Ft[:-1]
        ha, hb = dt / 2 * a, dt / 2 * b
        inv = torch.empty_like(ha)
        inv[0] = 1 / (1 + ha[0] + hb[0])
        for i in range(1, inv.shape[0]):
            inv[i] = 1 / (1 + ha[i] + hb[i] - ha[i] * hb[i - 1] * inv[i - 1])
        fw = torch.zeros_like(ha)
        fw[1:] = ha[1:] * inv[:-1]
        axes.append((a, b, fw, hb * inv, inv))

    def spread(u, ax):  # D_ax u, axis first
        a, b = axes[ax][:2]
        v = u.movedim(ax, 0).contiguous()
        o = torch.zeros_like(v)
        o[1:] += a[1:] * (v[:-1] - v[1:])
        o[:-1] += b[:-1] * (v[1:] - v[:-1])
        return o.movedim(0, ax)

    def solve(u, ax):
        fw, bw, inv = axes[ax][2:]
        v = u.movedim(ax, 0).contiguous()
        for i in range(1, v.shape[0]):
            v[i].addcmul_(fw[i], v[i - 1])
        v *= inv
        for i in range(v.shape[0] - 2, -1, -1):
            v[i].addcmul_(bw[i], v[i + 1])
        return v.movedim(0, ax)

    log_a = torch.where(E != 0, torch.log(torch.where(A > 0, A, torch.ones_like(A))), torch.zeros_like(A))
    hot = (E != 0)[M]
    omega = torch.zeros_like(T) if case["damage"] else None
    peak = torch.full((nM,), -math.inf, dtype=torch.float64, device=dev)
    heat = Q * free if hp["lightsOn"] else torch.zeros_like(Q)
    li = np.asarray(hp["tempSensorCornerIdxs"]).ravel().astype(np.int64)
    w = np.asarray(hp["tempSensorInterpWeights"]).reshape(len(li), 3) if len(li) else None
    seen = []

    def sense():
        row = []
        for k, l in enumerate(li):
            i, j, m = l % T.shape[0], l // T.shape[0] % T.shape[1], l // (T.shape[0] * T.shape[1])
            c = T[i:i + 2, j:j + 2, m:m + 2]
            for t in reversed(w[k]):  # z, then y, then x
                c = (1 - t) * c[..., 0] + t * c[..., 1]
            row.append(c)
        seen.append(torch.stack(row))

    for _ in range(nt):
        if len(li):
            sense()
        dx, dy, dz = (spread(T, ax) for ax in range(3))
        u = solve(T + dt * (heat + dy + dz) + dt / 2 * dx, 0)
        u = solve(u - dt / 2 * dy, 1)
        u = solve(u - dt / 2 * dz, 2)
        if omega is not None:
            mid = (0.5 * (u + T) + ZERO_C)[hot]
            omega[hot] += dt * torch.exp(log_a[M[hot]] - E[M[hot]] / (GAS_R * mid))
        T = u.contiguous()
        for m in range(nM):
            if bool((M == m).any()) if _ == 0 else math.isfinite(float(peak[m])):
                peak[m] = torch.maximum(peak[m], T[M == m].max())
    if len(li):
        sense()
    out = {"T": T.cpu().numpy(), "peaks": peak.reshape(1, -1).cpu().numpy()}
    if omega is not None:
        out["damage"] = omega.cpu().numpy()
    if len(li):
        out["sensors"] = torch.stack(seen, 1).cpu().numpy()
    return out


# ------------------------------------------------------------------------------------------------
# The interface
# ------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "mc":
        s["input"] = _mc_input(case, seed)
    elif kind == "mc_batch":
        rng = np.random.default_rng(case["models"])  # the models' sizes go with the case, not with the seed
        one = dict(source="gaussian", wavelengths=1, collector="none", far=0, matched=case["matched"])
        s["inputs"] = []
        for k in range(case["models"]):
            n = [max(16, int(case[a] * rng.uniform(0.6, 1.0))) for a in ("nx", "ny", "nz")]
            packets = int(case["packets"] * rng.uniform(0.5, 1.5))
            s["inputs"].append(_mc_input({**one, "nx": n[0], "ny": n[1], "nz": n[2], "packets": packets,
                                          "boundary": 3 if k % 2 else 1}, seed * 64 + k))
    elif kind == "mc_grad":
        s["input"] = _mc_input({**case, "source": "pencil", "boundary": 1, "wavelengths": 1, "collector": "none", "far": 0}, seed)
        s["bins"] = case["bins"]
        cx, cy, cz = case["nx"] // 2, case["ny"] // 2, case["nz"] // 4
        s["box"] = (cx - 4, cx + 4, cy - 4, cy + 4, cz, cz + 8)
    elif kind == "heat":
        h = _heat_input(case, seed)
        s.update(T0=h["T0"], hp=h["hp"], n=(case["nx"], case["ny"], case["nz"]), damage=case["damage"])
        s["omega"] = np.zeros(s["n"], dtype=np.float32, order="F") if case["damage"] else None
        s["state"] = native.HeatState(s["T0"], s["omega"], s["hp"], *s["n"]) if case["resident"] else None
    elif kind == "adjoint":
        h = _heat_input({**case, "light": True, "sensors": 0}, seed)
        n = (case["nx"], case["ny"], case["nz"])
        spare = np.zeros(n, dtype=np.float32, order="F")
        spare[:, :, : max(1, n[2] // 4)] = 1.0 / (n[0] * n[1] * max(1, n[2] // 4))
        s.update(T0=h["T0"], hp=h["hp"], n=n, wd=np.asfortranarray(h["inside"].astype(np.float32)), wp=spare,
                 checkpoints=case["steps"] if case["store_all"] else 0)
    elif kind == "normals":
        M = _heat_input({**case, "steps": 1, "sinked": False, "factor": 0.9}, seed)["M"]
        index = np.array([1.0, 1.33, 1.4, 1.45, 1.5])[: case["media"]]
        s.update(M=M, index=index, length=0.002 if case["smooth"] else 0.0)
    else:
        rng = np.random.default_rng(seed)
        n = case["n"]
        T = 37.0 + 40.0 * rng.beta(1.2, 4.0, n)  # a temperature field, and properties that follow it
        par = np.empty((3, n), dtype=np.float32, order="F")
        par[0] = 1.0 + 0.04 * (T - 37.0) + 0.02 * rng.standard_normal(n)
        par[1] = 100.0 * np.exp(-(T - 37.0) / 60.0)
        par[2] = 0.9 - 0.001 * (T - 37.0)
        s.update(par=par, bins=case["bins"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "mc":
        return _mc_output(native.mc_run(s["input"]))
    if kind == "mc_batch":
        return [_mc_output(o) for o in native.mc_run_batch(s["inputs"])]
    if kind == "mc_grad":
        out, g = native.mc_grad(s["input"], nRadialBins=s["bins"], radialBinWidth=0.05 / s["bins"], box=s["box"])
        return {"forward": _mc_output(out), "grad": {k: np.asarray(v, dtype=np.float32) for k, v in g.items()}}
    if kind == "heat":
        if s["state"] is not None:
            sensors, peaks = s["state"].step(s["hp"])
            T, omega = s["state"].read()
        else:
            T, omega, sensors, peaks = native.heat_forward(s["T0"], s["omega"], s["hp"], *s["n"])
        out = {"T": T, "peaks": peaks}
        if omega is not None:
            out["damage"] = omega
        if sensors.size:
            out["sensors"] = sensors.astype(np.float32)
        return out
    if kind == "adjoint":
        g = native.heat_adjoint(s["T0"], s["hp"], *s["n"], damageWeight=s["wd"], peakWeight=s["wp"], nCheckpoints=s["checkpoints"])
        return {"J": np.float32(g["J"]), "dJ_dc": g["dJ_dc"].astype(np.float32), "dJ_dQ": g["dJ_dQ"], "dJ_dT0": g["dJ_dT0"]}
    if kind == "normals":
        return native.interface_normals(s["M"], s["index"], 0.001, 0.001, 0.001, s["length"])
    return list(native.downsample_params(s["par"], s["bins"]))


def work(case):
    kind = case["kind"]
    if kind == "mc":
        return {"bytes": float(_mc_bytes(case["nx"], case["ny"], case["nz"], case["wavelengths"], case["matched"], case["far"],
                                         case["collector"], case["boundary"])),
                "flops": float(case["packets"]) * MC_STEPS * MC_FLOPS}
    if kind == "mc_batch":
        one = _mc_bytes(case["nx"], case["ny"], case["nz"], 1, case["matched"], 0, "none", 1)
        return {"bytes": 0.5 * case["models"] * one, "flops": float(case["models"] * case["packets"]) * MC_STEPS * MC_FLOPS}
    if kind == "mc_grad":
        return {"bytes": float(_mc_bytes(case["nx"], case["ny"], case["nz"], 1, case["matched"], 0, "none", 1)),
                "flops": float(case["packets"]) * MC_STEPS * 2 * MC_FLOPS}
    if kind == "heat":
        return _work_heat(case)
    if kind == "adjoint":  # the run and, going back, each step's state, its three solves and the gradients
        w = _work_heat(case)
        return {"bytes": 3 * w["bytes"], "flops": 3 * w["flops"]}
    if kind == "normals":
        L = case["nx"] * case["ny"] * case["nz"]
        # fast transforms along three axes, there and back, for three components per class
        flops = 30.0 * L + (case["media"] * 3 * 6 * 2.5 * L * math.log2(max(L, 2)) / 3 if case["smooth"] else 0.0)
        return {"bytes": 9.0 * L, "flops": flops}
    return {"bytes": 13.0 * case["n"], "flops": 9.0 * case["n"] * case["bins"]}


def exact(case, seed):
    """FP64 values where there are any: a packet's path has none (its decisions amplify rounding),
    smoothed normals far from every interface are directions of rounding noise, binning selects
    input values, and the adjoint's FP64 run would need every line solve's history."""
    return _exact_heat(case, seed) if case["kind"] == "heat" else None
