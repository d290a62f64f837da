"""Performance cases of the time-step loop, each one output interval of a run
under way: ``run`` advances the domain by the interval's steps and takes what
the output step writes (slice, monitor rows, field maxima, the running-DFT
plane, or whole fields), as the drop-in executable's loop does.  One case
puts a batch of requests through the serving loop.

``exact`` is the same loop in plain torch float64 (dense arrays, one tensor
operation per term of the update equations), sharing only the inputs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from php_fdtd_b200 import Material, Simulation, Source, make_desc
from php_fdtd_b200.serving import DftSpec, Server
from php_fdtd_b200.workloads import cone_tip_box, drude_lorentz_eps, lattice_16atom, lattice_2atom

C0 = 299792458.0
EPS0 = 8.854e-12
MU0 = math.pi * 4e-7
HZ_PER_CM = 0.03e12
ROT20 = 0.3490658504
ROT30 = 0.5235987756


def listed():
    return [
        # the shortest useful interval on a small grid: launches and read-out latency are all of it
        {"name": "glass_32_fp64", "scene": "glass", "nx": 32, "ny": 32, "nz": 32, "cell": 10e-9, "pml": 4,
         "steps": 10, "warm": 30, "precision": "fp64", "nfreq": 0, "volumes": False},
        # the two-atom polar slab (96^3, a slice every 20 steps): the everyday phonon-polariton run, both precisions
        {"name": "polar_96_fp64", "scene": "polar", "nx": 96, "ny": 96, "nz": 96, "cell": 10e-9, "pml": 10,
         "steps": 20, "warm": 200, "precision": "fp64", "nfreq": 0, "volumes": False},
        {"name": "polar_96_fp32", "scene": "polar", "nx": 96, "ny": 96, "nz": 96, "cell": 10e-9, "pml": 10,
         "steps": 20, "warm": 200, "precision": "fp32", "nfreq": 0, "volumes": False},
        # metal tip (tensor ADE) over a rotated lossy anisotropic slab, running DFT above it: the repository's
        # benchmark workload at its grid and its output interval, both precisions
        {"name": "tip_256_fp64", "scene": "tip", "nx": 256, "ny": 256, "nz": 256, "cell": 5e-9, "pml": 12,
         "steps": 50, "warm": 230, "precision": "fp64", "nfreq": 1, "volumes": False},
        {"name": "tip_256_fp32", "scene": "tip", "nx": 256, "ny": 256, "nz": 256, "cell": 5e-9, "pml": 12,
         "steps": 50, "warm": 230, "precision": "fp32", "nfreq": 1, "volumes": False},
        # 16-atom lattice: the ion pass (DMM contraction) carries the step, both precisions
        {"name": "lattice16_256_fp64", "scene": "lattice16", "nx": 256, "ny": 256, "nz": 128, "cell": 10e-9, "pml": 10,
         "steps": 20, "warm": 200, "precision": "fp64", "nfreq": 0, "volumes": False},
        {"name": "lattice16_256_fp32", "scene": "lattice16", "nx": 256, "ny": 256, "nz": 128, "cell": 10e-9, "pml": 10,
         "steps": 20, "warm": 200, "precision": "fp32", "nfreq": 0, "volumes": False},
        # the large single domain (half the edge of the 1024 x 1024 x 512 one): rotated two-atom slab, tip, a DFT
        # plane at three wavenumbers, both precisions
        {"name": "tipslab_512_fp64", "scene": "tipslab", "nx": 512, "ny": 512, "nz": 256, "cell": 8e-9, "pml": 16,
         "steps": 30, "warm": 200, "precision": "fp64", "nfreq": 3, "volumes": False},
        {"name": "tipslab_512_fp32", "scene": "tipslab", "nx": 512, "ny": 512, "nz": 256, "cell": 8e-9, "pml": 16,
         "steps": 50, "warm": 200, "precision": "fp32", "nfreq": 3, "volumes": False},
        # the mode that reproduces the reference bit for bit, on a ragged grid of anisotropic media; whole E fields
        # taken at the end of the interval
        {"name": "crystal_101_strict", "scene": "crystal", "nx": 101, "ny": 67, "nz": 53, "cell": 10e-9, "pml": 6,
         "steps": 100, "warm": 100, "precision": "fp64-strict", "nfreq": 1, "volumes": True},
        # ragged grid, rotated lossy and anisotropic media, |E| on an x plane
        {"name": "crystal_201_fp32", "scene": "crystal", "nx": 201, "ny": 173, "nz": 131, "cell": 10e-9, "pml": 8,
         "steps": 50, "warm": 200, "precision": "fp32", "nfreq": 0, "volumes": False},
        # serving: independent requests of uneven size through admission, stepping and read-back
        {"name": "serving_6_fp32", "scene": "serving", "requests": 6, "edge_lo": 64, "edge_hi": 128, "pml": 8,
         "steps": 1200, "precision": "fp32"},
    ]


# per scene: (smallest, largest) edge along x/y and along z, precisions
RANGES = {
    "glass": (24, 256, 24, 256, ("fp64", "fp32", "fp64-strict")),
    "polar": (48, 256, 48, 256, ("fp64", "fp32")),
    "tip": (64, 288, 64, 288, ("fp64", "fp32")),
    "tipslab": (128, 512, 96, 256, ("fp64", "fp32")),
    "crystal": (40, 256, 40, 200, ("fp64", "fp32", "fp64-strict")),
    "lattice16": (32, 256, 32, 128, ("fp64", "fp32")),
}
MAX_CELLS = 512 * 512 * 256
MAX_CELLS_LATTICE = 256 * 256 * 128


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if rng.random() < 0.08:
        return {"scene": "serving", "requests": rng.randint(2, 6), "edge_lo": 64, "edge_hi": rng.randint(72, 120),
                "pml": 8, "steps": log_int(200, 1000), "precision": "fp32"}
    scene = rng.choice(sorted(RANGES))
    lo, hi, zlo, zhi, precisions = RANGES[scene]
    cap = MAX_CELLS_LATTICE if scene == "lattice16" else MAX_CELLS
    nx, ny, nz = log_int(lo, hi), log_int(lo, hi), log_int(zlo, zhi)
    if nx * ny * nz > cap:
        nz = max(zlo, cap // (nx * ny))
    precision = rng.choice(precisions)
    limit = 8e6 if precision == "fp64-strict" else 40e6 if scene == "lattice16" else 8e8
    steps = max(2, min(log_int(5, 60), int(limit / (nx * ny * nz))))
    return {"scene": scene, "nx": nx, "ny": ny, "nz": nz,
            "cell": rng.choice([5e-9, 8e-9, 10e-9]), "pml": rng.randint(4, max(4, min(16, min(nx, ny, nz) // 6))),
            "steps": steps, "warm": 200, "precision": precision,
            "nfreq": rng.choice([0, 1, 3]), "volumes": nx * ny * nz < 1e6 and rng.random() < 0.25}


# ------------------------------------------------------------------- inputs


def _tip_material(nu_cm):
    e = drude_lorentz_eps(nu_cm)
    return dict(eps_re=np.eye(3) * e.real, eps_im=np.eye(3) * e.imag, use_ade=1)


def _inputs(case, seed):
    """Medium [nx][ny][nz], material records, sources, output positions."""
    rng = np.random.default_rng(seed)
    scene, nx, ny, nz, L, dl = (case[q] for q in ("scene", "nx", "ny", "nz", "pml", "cell"))
    dt = dl / (C0 * math.sqrt(3.0)) * 0.99
    med = np.zeros((nx, ny, nz), np.int32)
    mats = [dict()]
    jx, jy = (int(v) for v in rng.integers(-3, 4, size=2))
    cx, cy = nx // 2 + jx, ny // 2 + jy
    # fields of about 1e6 V/m: a driven near field, lattice displacements far below the divergence guard
    amp = 1e12 * float(rng.uniform(0.5, 2.0))
    f = HZ_PER_CM * float(rng.uniform(850.0, 1400.0))
    slice_at, comp = ("z", nz // 2), "Ez"
    # a weak sine at the polariton wavenumber (quasi-static over these few steps), and a wave that fills the domain
    sine = dict(type=1, x=cx, y=cy, component="z", amplitude=0.01 * amp, frequency=f)
    wave = dict(type=1, x=cx + 2, y=cy - 2, component="z", amplitude=amp,
                frequency=float(rng.uniform(0.9, 1.1)) / (21 * dt))
    slab = max(2, round(40 * nz / 96))
    if scene == "glass":
        med[:, :, :nz // 3] = 1
        mats.append(dict(eps_re=np.eye(3) * float(rng.uniform(2.0, 4.0))))
        zs = nz // 2
    elif scene == "polar":
        qv, qm, dmm = lattice_2atom(int(rng.integers(1 << 30)))
        med[:, :, :slab] = 1
        mats.append(dict(eps_re=np.diag([4.9, 4.9, 2.95]), natom=2, qezv=qv, qezm=qm, dmm=dmm))
        slice_at, zs = ("z", slab + 2), min(nz - L - 2, slab + max(3, nz // 6))
    elif scene in ("tip", "tipslab"):
        if scene == "tip":
            slab = max(2, round(40 * nz / 256))
            a, b, c = 6.0 * float(rng.uniform(0.9, 1.1)), 3.5, 2.8
            mats.append(dict(eps_re=np.diag([a, b, c]), eps_im=np.diag([0.4, 0.2, 0.1]), anglez=ROT30))
        else:
            slab = max(2, round(64 * nz / 512))
            qv, qm, dmm = lattice_2atom(int(rng.integers(1 << 30)))
            mats.append(dict(eps_re=np.diag([4.9, 4.9, 2.95]), natom=2, qezv=qv, qezm=qm, dmm=dmm, anglex=ROT20))
        med[:, :, :slab] = 1
        mats.append(_tip_material(f / HZ_PER_CM))
        box, sub = cone_tip_box(nx, ny, nz, dl, dl, (nx // 2, ny // 2), slab + 2, 20e-9, 15.0, top_k=nz - L - 2)
        med[box][sub] = 2
        slice_at, zs = ("z", slab + 1), min(nz - L - 2, slab + 2 + nz // 4)
    elif scene == "lattice16":
        qv, qm, dmm = lattice_16atom(int(rng.integers(1 << 30)))
        slab = nz // 2
        med[:, :, :slab] = 1
        mats.append(dict(eps_re=np.diag([5.8, 6.6, 4.4]), natom=16, qezv=qv, qezm=qm, dmm=dmm))
        comp, slice_at, zs = "Ex", ("z", slab + 2), min(nz - L - 2, slab + max(2, nz // 10))
        sine["component"] = wave["component"] = "x"
    elif scene == "crystal":
        mats += [dict(eps_re=np.diag([6.0, 3.5, 2.8]), eps_im=np.diag([0.4, 0.2, 0.1]), anglez=ROT30),
                 dict(eps_re=np.array([[4.0, 0.7, 0.2], [0.7, 3.0, -0.3], [0.2, -0.3, 2.5]])),
                 dict(eps_re=np.diag([5.0, 2.0, 3.0]), eps_im=np.array([[0, 0, 0], [0, 0, 0.1], [0, 0.1, 0]]),
                      anglex=ROT20),
                 dict(eps_re=np.eye(3) * 2.25, sigma=500.0)]
        med[:, :, :nz // 3] = 1
        x0, y0 = nx // 6 + jx, ny // 6 + jy
        med[x0:x0 + nx // 2, y0:y0 + ny // 2, nz // 3:nz // 2] = 2
        med[x0:x0 + nx // 3, y0 + ny // 3:y0 + (2 * ny) // 3, nz // 3:(3 * nz) // 5] = 3
        med[nx // 2:, ny // 2:, nz // 3:nz // 3 + max(1, nz // 8)] = 4
        comp, slice_at, zs = "E", ("x", nx // 2), (2 * nz) // 3
    else:
        raise ValueError(scene)
    sine["z"] = wave["z"] = int(zs)
    return {"nx": nx, "ny": ny, "nz": nz, "L": L, "dl": dl, "dt": dt, "medium": med, "mats": mats,
            "sources": [sine, wave], "frequency": f, "comp": comp, "slice": slice_at,
            "monitor": (nx // 2 + min(nx // 8, 7), ny // 2 - min(ny // 8, 5),
                        min(slab, nz - 2) - 1 if scene != "glass" else nz // 2),
            "dft_z": min(nz - 1, slice_at[1] + 1) if slice_at[0] == "z" else nz // 2,
            "dft_f": [f, 1.2 * f, 1.0 / (21 * dt)][: case["nfreq"]]}


def _holder(s, precision):
    mats = [Material(**{k: (tuple(np.ravel(v)) if k.startswith("eps") else v) for k, v in m.items()})
            for m in s["mats"]]
    return make_desc(s["medium"], mats, [Source(**q) for q in s["sources"]], dx=s["dl"], dy=s["dl"], dz=s["dl"],
                     dt=s["dt"], pml_thickness=s["L"], precision=precision, source_frequency=s["frequency"],
                     epsilon0=EPS0, mu0=MU0)


def _requests(case, seed):
    """Serving requests: polar slab, tip, sine source, uneven grids and step
    counts (the case's own, so that the planes keep their shapes)."""
    rng, size = np.random.default_rng(seed), np.random.default_rng(case["steps"] + 7 * case["requests"])
    out = []
    for _ in range(case["requests"]):
        lo, hi = math.log(case["edge_lo"]), math.log(case["edge_hi"])
        nx, ny, nz = (int(round(math.exp(size.uniform(lo, hi)))) for _ in range(3))
        sub = {"scene": "tipslab", "nx": nx, "ny": ny, "nz": nz, "pml": case["pml"], "cell": 10e-9, "nfreq": 1}
        s = _inputs(sub, int(rng.integers(1 << 30)))
        s["steps"] = int(size.integers(case["steps"] // 2, case["steps"] + 1))
        del s["sources"][1:]  # the sine alone
        out.append(s)
    return out


def prepare(case, seed):
    if case["scene"] == "serving":
        reqs = [(_holder(s, case["precision"]), s["steps"], DftSpec("Ez", s["dft_z"], s["dft_f"]))
                for s in _requests(case, seed)]
        return {"case": case, "server": Server(32 << 30), "requests": reqs}
    s = _inputs(case, seed)
    sim = Simulation(_holder(s, case["precision"]))
    sim.step(case["warm"])
    i, j, k = s["monitor"]
    sim.probe_set(i, j, k + 1, k)
    dft = sim.dft_add("Ez", s["dft_z"], s["dft_f"]) if s["dft_f"] else None
    sim.prepare(case["steps"])
    sim.sync()
    return {"case": case, "sim": sim, "slice": (s["comp"], *s["slice"]), "dft": dft,
            "natom": s["mats"][int(s["medium"][i, j, k])].get("natom", 0)}


# --------------------------------------------------------------------- run


def _rows(rows, natom, real):
    """Monitor rows by quantity (they differ by orders of magnitude)."""
    out = {"E": rows[:, 0:3], "D": rows[:, 3:6], "H": rows[:, 6:9]}
    if natom:
        out["r"], out["v"] = rows[:, 9:9 + 3 * natom], rows[:, 9 + 3 * natom:]
    return {k: np.ascontiguousarray(v, dtype=real) for k, v in out.items()}


def run(state):
    case = state["case"]
    if case["scene"] == "serving":
        srv = state["server"]
        order = {srv.submit(h, n, d): q for q, (h, n, d) in enumerate(state["requests"])}
        planes = [None] * len(order)
        while order:
            for info in srv.poll(timeout_ms=1000):
                if info["status"] != 0:
                    raise RuntimeError(info["error"])
                planes[order.pop(info["job"])] = srv.fetch_dft(info).astype(np.complex64)
        return {"dft": planes}
    sim = state["sim"]
    # an FP32 run's values carry single precision and are kept so, as its slice files are
    single = case["precision"] == "fp32"
    real = np.float32 if single else np.float64
    sim.step(case["steps"])
    f = sim.frame_wait(sim.frame_begin(diag=True, slice=state["slice"], probe=True))
    out = {"slice": f["slice"], "rows": _rows(f["rows"], state["natom"], real),
           "max": np.array([f["diag"]["max_e"], f["diag"]["max_ex"], f["diag"]["max_r"]], dtype=real)}
    if state["dft"] is not None:
        out["dft"] = sim.dft_read(state["dft"])[0].astype(np.complex64 if single else np.complex128)
    if case["volumes"]:
        out["volumes"] = [sim.read_volume(c).astype(real) for c in ("Ex", "Ey", "Ez")]
    return out


def work(case):
    """Per step E, H, the CPML state and the ADE and lattice state read once and
    written once (a domain's state does not stay on the chip between steps),
    and the material id read; the outputs once."""
    if case["scene"] == "serving":
        total = {"bytes": 0.0, "flops": 0.0}
        for s in _requests(case, 0):
            sub = {"scene": "tipslab", "nx": s["nx"], "ny": s["ny"], "nz": s["nz"], "pml": s["L"], "cell": s["dl"],
                   "steps": s["steps"], "precision": case["precision"], "nfreq": 1, "volumes": False}
            for k, v in work(sub).items():
                total[k] += v
        return total
    scene, nx, ny, nz, L = (case[q] for q in ("scene", "nx", "ny", "nz", "pml"))
    w = 4 if case["precision"] == "fp32" else 8
    cells = nx * ny * nz
    atoms = {"polar": (2, round(40 * nz / 96)), "lattice16": (16, nz // 2),
             "tipslab": (2, round(64 * nz / 512))}.get(scene, (0, 0))
    acells = nx * ny * max(2, atoms[1]) if atoms[0] else 0
    pml = 2 * L * (ny * nz + nx * nz + nx * ny)
    words = 12 * cells + 8 * pml + 12 * atoms[0] * acells
    flops = 40 * cells + 24 * pml + acells * (2 * (3 * atoms[0]) ** 2 + 54 * atoms[0])
    out = 4 * nx * ny + 16 * case["nfreq"] * nx * ny + (3 * cells * w if case["volumes"] else 0)
    return {"bytes": float(case["steps"] * (words * w + cells) + out), "flops": float(case["steps"] * flops)}


# ------------------------------------------------------------------- exact


def _axis(n, L, d, dt, dev):
    """CPML profile of one axis: kappa, b, c per cell (cubic grading)."""
    kap, b, c = np.ones(n), np.ones(n), np.zeros(n)
    smax = -4.0 * math.log(1e-6) / (2.0 * math.sqrt(MU0 / EPS0) * d * L) if L else 0.0
    for i in range(n):
        q = i if i < L else n - 1 - i if i >= n - L else -1
        if q < 0:
            continue
        r = (L - q) / L
        s, kap[i], a = smax * r ** 3, 1.0 + 6.0 * r ** 3, 0.05 * (1.0 - r)
        aw = s / (kap[i] * EPS0) + a / EPS0
        b[i] = math.exp(-aw * dt)
        c[i] = s / (kap[i] ** 2 * EPS0) * (b[i] - 1.0) / aw if aw > 1e-30 else 0.0
    return [torch.tensor(v, dtype=torch.float64, device=dev) for v in (kap, b, c)]


def _adj(m):
    out = np.empty((3, 3))
    for r in range(3):
        for s in range(3):
            sub = np.delete(np.delete(m, s, 0), r, 1)
            out[r, s] = (-1) ** (r + s) * (sub[0, 0] * sub[1, 1] - sub[0, 1] * sub[1, 0])
    return out


class _Medium:
    """One material's coefficients and the flat indices of its cells."""

    def __init__(self, m, where, f, dt, dev):
        re = np.asarray(m.get("eps_re", np.eye(3)), float).reshape(3, 3)
        im = np.asarray(m.get("eps_im", np.zeros((3, 3))), float).reshape(3, 3)
        # the solver's inverse of eps: determinants and adjugates of the real and imaginary parts apart
        dr, di = np.linalg.det(re), (np.linalg.det(im) if im.any() else 0.0)
        inv = (dr * _adj(re) + di * _adj(im)) / (dr * dr + di * di)
        s = m.get("sigma", 0.0) * dt / (2 * EPS0)
        lf = 1.0 / (1.0 + s)
        self.keep = 1.0 - s * lf
        az, ax = m.get("anglez", 0.0), m.get("anglex", 0.0)
        rot = np.eye(3)
        if az:
            rot[0:2, 0:2] = [[math.cos(az), -math.sin(az)], [math.sin(az), math.cos(az)]]
        elif ax:
            rot[1:3, 1:3] = [[math.cos(-ax), -math.sin(-ax)], [math.sin(-ax), math.cos(-ax)]]
        t = lambda a: torch.tensor(np.asarray(a, float), dtype=torch.float64, device=dev)  # noqa: E731
        self.rot, self.inv, self.where = t(rot), t(inv * (lf / EPS0)), where
        self.ade, self.natom = bool(m.get("use_ade")), m.get("natom", 0)
        self.loss = t(im * (dt * f * 2.0 * 3.14159265 * EPS0)) if im.any() and not self.ade else None
        if self.ade:
            e1 = re - 20.0 * np.eye(3)
            g = -(im @ np.linalg.inv(e1)) * f * 2.0 * math.pi
            w = -f * f * 4.0 * math.pi ** 2 * e1 + f * 2.0 * math.pi * (g @ im)
            self.gp, self.gm = t(np.linalg.inv(np.eye(3) + g * dt / 2)), t(np.eye(3) - g * dt / 2)
            self.w = t(w * (EPS0 * dt * dt))
            self.P = torch.zeros((where.numel(), 3), dtype=torch.float64, device=dev)
            self.Po = torch.zeros_like(self.P)
        if self.natom:
            n = self.natom
            self.zv = t(np.reshape(m["qezv"], (n, 3, 3)).transpose(1, 0, 2).reshape(3, 3 * n))
            self.zm = t(np.reshape(m["qezm"], (n, 3, 3)).transpose(0, 2, 1).reshape(3 * n, 3))
            self.dmm = t(np.reshape(m["dmm"], (3 * n, 3 * n)))
            self.r = torch.zeros((where.numel(), 3 * n), dtype=torch.float64, device=dev)
            self.v = torch.zeros_like(self.r)


class _Exact:
    def __init__(self, s):
        self.s, dev = s, "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny, nz = s["nx"], s["ny"], s["nz"]
        z = lambda *n: torch.zeros(n, dtype=torch.float64, device=dev)  # noqa: E731
        # [component][x][y][z with a zero plane on either side]
        self.E, self.D, self.H = z(3, nx, ny, nz + 2), z(3, nx, ny, nz + 2), z(3, nx, ny, nz + 2)
        self.psi = {q: z(nx, ny, nz) for q in ("hxy", "hxz", "hyx", "hyz", "hzx", "hzy",
                                               "dxy", "dxz", "dyx", "dyz", "dzx", "dzy")}
        ax = [_axis(n, s["L"], s["dl"], s["dt"], dev) for n in (nx, ny, nz)]
        self.kx, self.bx, self.cx = (v.view(-1, 1, 1) for v in ax[0])
        self.ky, self.by, self.cy = (v.view(1, -1, 1) for v in ax[1])
        self.kz, self.bz, self.cz = (v.view(1, 1, -1) for v in ax[2])
        med = torch.tensor(s["medium"], device=dev)
        pad = torch.full((nx, ny, nz + 2), -1, dtype=torch.int32, device=dev)
        pad[:, :, 1:-1] = med
        self.media = []
        for q, m in enumerate(s["mats"]):
            where = (pad.view(-1) == q).nonzero().view(-1)
            if where.numel():
                self.media.append(_Medium(m, where, s["frequency"], s["dt"], dev))
        inner = torch.zeros((nx, ny, nz + 2), dtype=torch.bool, device=dev)
        inner[1:-1, 1:-1, 1:-1] = True
        self.lossy = [(m, m.where[inner.view(-1)[m.where]]) for m in self.media if m.loss is not None]
        self.t, self.rows, self.dft, self.taking = 0, [], None, False

    def _psi(self, name, sl, b, c, d):
        """The old CPML term, replaced by b psi + c d."""
        p = self.psi[name][sl]
        old = p.clone()
        p.mul_(b).add_(c * d)
        return old

    def step(self):
        s = self.s
        dt, dl = s["dt"], s["dl"]
        Ex, Ey, Ez = self.E
        Hx, Hy, Hz = self.H
        # H: cells i < nx-1, j < ny-1
        a, m = slice(0, -1), slice(1, -1)
        sl = (a, a, slice(None))
        up = slice(2, None)
        kx, bx, cx = self.kx[a], self.bx[a], self.cx[a]
        ky, by, cy = self.ky[:, a], self.by[:, a], self.cy[:, a]
        kz, bz, cz = self.kz, self.bz, self.cz
        g = 1.0 / (dl * MU0)
        ddx = lambda F: (F[1:, :-1, m] - F[:-1, :-1, m]) * g  # noqa: E731
        ddy = lambda F: (F[:-1, 1:, m] - F[:-1, :-1, m]) * g  # noqa: E731
        ddz = lambda F: (F[a, a, up] - F[a, a, m]) * g  # noqa: E731
        dzy, dyz, dzx, dxz, dyx, dxy = ddy(Ez), ddz(Ey), ddx(Ez), ddz(Ex), ddx(Ey), ddy(Ex)
        Hx[a, a, m] += dt * (-dzy / ky + self._psi("hyx", sl, by, cy, -dzy) + dyz / kz + self._psi("hzx", sl, bz, cz, dyz))
        Hy[a, a, m] += dt * (dzx / kx + self._psi("hxy", sl, bx, cx, dzx) - dxz / kz + self._psi("hzy", sl, bz, cz, -dxz))
        Hz[a, a, m] += dt * (-dyx / kx + self._psi("hxz", sl, bx, cx, -dyx) + dxy / ky + self._psi("hyz", sl, by, cy, dxy))
        del dzy, dyz, dzx, dxz, dyx, dxy
        # D: interior in x and y
        sl = (m, m, slice(None))
        kx, bx, cx = self.kx[m], self.bx[m], self.cx[m]
        ky, by, cy = self.ky[:, m], self.by[:, m], self.cy[:, m]
        dn = slice(0, -2)
        g = 1.0 / dl
        ddx = lambda F: (F[1:-1, m, m] - F[:-2, m, m]) * g  # noqa: E731
        ddy = lambda F: (F[m, 1:-1, m] - F[m, :-2, m]) * g  # noqa: E731
        ddz = lambda F: (F[m, m, m] - F[m, m, dn]) * g  # noqa: E731
        dzy, dyz, dxz, dzx, dyx, dxy = ddy(Hz), ddz(Hy), ddz(Hx), ddx(Hz), ddx(Hy), ddy(Hx)
        Dx, Dy, Dz = self.D
        Dx[m, m, m] += dt * (dzy / ky + self._psi("dyx", sl, by, cy, dzy) - dyz / kz + self._psi("dzx", sl, bz, cz, -dyz))
        Dy[m, m, m] += dt * (-dzx / kx + self._psi("dxy", sl, bx, cx, -dzx) + dxz / kz + self._psi("dzy", sl, bz, cz, dxz))
        Dz[m, m, m] += dt * (dyx / kx + self._psi("dxz", sl, bx, cx, dyx) - dxy / ky + self._psi("dyz", sl, by, cy, -dxy))
        del dzy, dyz, dxz, dzx, dyx, dxy
        E3, D3 = self.E.view(3, -1), self.D.view(3, -1)
        for md, where in self.lossy:
            D3[:, where] -= md.loss @ E3[:, where]
        time = self.t * dt
        for q in s["sources"]:
            self.D["xyz".index(q["component"]), q["x"], q["y"], q["z"] + 1] += q["amplitude"] * math.sin(2 * math.pi * q["frequency"] * time) * dt
        # D -> E, ADE, ions, in the crystal frame
        for md in self.media:
            d = md.rot @ D3[:, md.where]
            if md.natom:
                d -= md.zv @ md.r.T
            if md.ade:
                e = md.rot @ E3[:, md.where]
                n = (2.0 * md.P - md.Po @ md.gm.T + (md.w @ e).T) @ md.gp.T
                md.Po, md.P = md.P, n
                e = (d - n.T) / (EPS0 * 20.0) * md.keep
            else:
                e = (md.inv @ d) * md.keep
            if md.natom:
                acc = e.T @ md.zm.T - md.r @ md.dmm.T
                md.r += md.v * dt + 0.5 * acc * dt * dt
                md.v += acc * dt
            E3[:, md.where] = md.rot.T @ e
        if self.taking:
            i, j, k = s["monitor"]
            row = [F[:, i, j, k + 2] for F in (self.E, self.D, self.H)]
            if self.atom is not None:
                md, q = self.atom
                row += [md.r[q], md.v[q]]
            self.rows.append(torch.cat(row))
        self.accumulate()
        self.t += 1

    def accumulate(self):
        if self.dft is not None:
            x = self.E[2, :, :, self.s["dft_z"] + 1]
            for q, f in enumerate(self.s["dft_f"]):
                ph = -2.0 * math.pi * f * (self.t * self.s["dt"])
                self.dft[q] += x * complex(math.cos(ph), math.sin(ph))

    def take(self):
        """Monitor rows and DFT samples from the next step on."""
        s = self.s
        i, j, k = s["monitor"]
        flat = (i * s["ny"] + j) * (s["nz"] + 2) + k + 1
        self.atom = None
        for md in self.media:
            hit = (md.where == flat).nonzero()
            if hit.numel() and md.natom:
                self.atom = (md, int(hit))
        self.taking = True
        if s["dft_f"]:
            self.dft = torch.zeros((len(s["dft_f"]), s["nx"], s["ny"]), dtype=torch.complex128, device=self.E.device)

    def volume(self, c):
        return self.E[c, :, :, 1:-1].contiguous().cpu().numpy()


def exact(case, seed):
    if case["scene"] == "serving":
        planes = []
        for s in _requests(case, seed):
            x = _Exact(s)
            x.take()
            x.taking = False
            for _ in range(s["steps"]):
                x.step()
            planes.append(x.dft.cpu().numpy())
        return {"dft": planes}
    s = _inputs(case, seed)
    x = _Exact(s)
    for _ in range(case["warm"]):
        x.step()
    x.take()
    for _ in range(case["steps"]):
        x.step()
    axis, pos = s["slice"]
    F = {"z": lambda: x.E[:, :, :, pos + 2], "x": lambda: x.E[:, pos, :, 1:-1], "y": lambda: x.E[:, :, pos, 1:-1]}[axis]()
    plane = F.square().sum(0).sqrt() if s["comp"] == "E" else F["xyz".index(s["comp"][1])]
    rows = torch.stack(x.rows).cpu().numpy()
    mag = x.E.square().sum(0).sqrt()
    max_r = max([float(m.r.abs().max()) for m in x.media if m.natom], default=0.0)
    out = {"slice": plane.contiguous().cpu().numpy().ravel(),
           "rows": _rows(rows, x.atom[0].natom if x.atom else 0, np.float64),
           "max": np.array([float(mag.max()), float(x.E[0].abs().max()), max_r])}
    if x.dft is not None:
        out["dft"] = x.dft.cpu().numpy()
    if case["volumes"]:
        out["volumes"] = [x.volume(c) for c in range(3)]
    return out
