"""The work that programs have this library do, as timed cases.

A case is a dict of plain values; prepare() makes the frame and the system
(batch, server) that a program would hold, run() is one pass through the
public entry points: a segment of MD steps ending with the read-out of the
frame, a force pass on new coordinates, a batch of replicas, or a set of
requests served to the end.  exact() restates the same pass in plain torch
FP64 (padded cells, torch.fft for the smooth-PME sum).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import atomiverse_b200 as A
from atomiverse_b200 import workloads as W

MIXED = 1
FLUID_RHO = 0.8442
STATE = ("x", "y", "z", "vx", "vy", "vz")
FULL = STATE + ("fx", "fy", "fz")


def listed():
    return [
        # the smallest replica of a ladder: every step is launch latency
        dict(name="fluid_256", kind="fluid", cx=4, cy=4, cz=4, drop=0, precision=0,
             thermostat=0, t_star=1.44, stress=0, steps=100),
        # the plain LJ fluid every MD user starts with (4,000 atoms, NVE)
        dict(name="fluid_4000", kind="fluid", cx=10, cy=10, cz=10, drop=0, precision=0,
             thermostat=0, t_star=1.44, stress=0, steps=100),
        # an ordinary replica in a slab box with vacancies: Langevin, mixed, virial
        dict(name="fluid_slab_langevin", kind="fluid", cx=23, cy=17, cz=9, drop=37, precision=1,
             thermostat=2, t_star=1.1, stress=1, steps=50),
        # the precision study's fluid, both builds: a million atoms
        dict(name="fluid_1m", kind="fluid", cx=63, cy=63, cz=63, drop=0, precision=0,
             thermostat=0, t_star=0.72, stress=0, steps=40),
        dict(name="fluid_1m_mixed", kind="fluid", cx=63, cy=63, cz=63, drop=0, precision=1,
             thermostat=0, t_star=0.72, stress=0, steps=20),
        # a small salt melt with PME and Nose-Hoover: latency of the whole chain
        dict(name="melt_1728", kind="melt", nx=12, ny=12, nz=12, order=4, precision=0, steps=50),
        # a middling melt in an uneven box, mixed precision
        dict(name="melt_22k_mixed", kind="melt", nx=36, ny=28, nz=22, order=4, precision=1,
             steps=40),
        # the headline melt: 262,144 ions, 192^3 mesh, FP64
        dict(name="melt_262k", kind="melt", nx=64, ny=64, nz=64, order=4, precision=0, steps=20),
        # a three-type LJ mixture under a thermostat and a barostat
        dict(name="mixture_npt", kind="mixture", cells=15, precision=0, steps=40),
        # single-point forces, energy and virial of a water box (per-type LJ,
        # exclusions, PME) on new coordinates
        dict(name="water_forces", kind="water", m=20, precision=1),
        # a ladder of replicas advanced together
        dict(name="ladder_24", kind="batch", systems=24, n_min=256, n_max=32768, steps=50),
        # a burst of requests served to the end: fluids and melts
        dict(name="serve_10", kind="serve", requests=10, n_min=500, n_max=20000, steps=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fluid", "fluid", "fluid", "melt", "melt", "mixture", "water", "batch",
                       "serve"])
    if kind == "fluid":
        n = _log_int(rng, 300, 900000)
        c = (n / 4.0) ** (1.0 / 3.0)
        cx = max(4, int(round(c * rng.uniform(0.7, 1.4))))
        cy = max(4, int(round(c * rng.uniform(0.7, 1.4))))
        cz = max(4, min(int(round(n / (4.0 * cx * cy))), 250000 // (cx * cy)))
        return dict(kind=kind, cx=cx, cy=cy, cz=cz, drop=rng.randint(0, cx * cy * cz // 16),
                    precision=rng.randint(0, 1), thermostat=rng.choice([0, 0, 1, 2]),
                    t_star=round(rng.uniform(0.7, 1.5), 3), stress=rng.randint(0, 1),
                    steps=20 if n > 100000 else rng.choice([25, 50, 100]))
    if kind == "melt":
        n = _log_int(rng, 600, 200000)
        c = n ** (1.0 / 3.0)
        nx = max(8, 2 * int(round(c * rng.uniform(0.75, 1.3) / 2)))
        ny = max(8, 2 * int(round(c * rng.uniform(0.75, 1.3) / 2)))
        nz = max(8, min(2 * int(round(n / (nx * ny) / 2)), 2 * (262144 // (2 * nx * ny))))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, order=rng.choice([4, 4, 6]),
                    precision=rng.randint(0, 1), steps=20 if n > 30000 else rng.choice([20, 40]))
    if kind == "mixture":
        return dict(kind=kind, cells=_log_int(rng, 6, 30), precision=rng.randint(0, 1),
                    steps=rng.choice([20, 40]))
    if kind == "water":
        return dict(kind=kind, m=_log_int(rng, 7, 24), precision=rng.randint(0, 1))
    if kind == "batch":
        return dict(kind=kind, systems=_log_int(rng, 3, 32), n_min=256,
                    n_max=_log_int(rng, 1000, 32768), steps=rng.choice([20, 50]))
    return dict(kind=kind, requests=rng.randint(3, 10), n_min=500,
                n_max=_log_int(rng, 1000, 20000), steps=rng.choice([20, 40]))


# ------------------------------------------------------------------ inputs

def _frame(pos, vel, mass, charge):
    f = {k: np.ascontiguousarray(pos[:, i]) for i, k in enumerate("xyz")}
    f.update({"v" + k: np.ascontiguousarray(vel[:, i]) for i, k in enumerate("xyz")})
    f["mass"], f["charge"] = mass, charge
    f["tag"] = np.arange(1, len(mass) + 1, dtype=np.int64)
    return f


def _fluid(c, seed):
    """FCC Lennard-Jones fluid in reduced units, cx x cy x cz cells, `drop`
    sites removed at random."""
    rng = np.random.default_rng(seed)
    a = (4.0 / FLUID_RHO) ** (1.0 / 3.0)
    nc = np.array([c["cx"], c["cy"], c["cz"]])
    g = np.stack(np.meshgrid(*[np.arange(k) for k in nc], indexing="ij"), -1).reshape(-1, 3)
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]) + 0.25
    pos = ((g[:, None, :] + base[None]) * a).reshape(-1, 3)
    if c["drop"]:
        keep = np.ones(len(pos), bool)
        keep[rng.choice(len(pos), c["drop"], replace=False)] = False
        pos = pos[keep]
    n = len(pos)
    T = c["t_star"] / W.KB
    mass = np.ones(n)
    vel = W.maxwell_velocities(mass, T, rng)
    desc = dict(n_atoms=n, box=tuple(float(v) for v in nc * a), precision=c["precision"],
                nl_cutoff=2.5, nl_skin=0.3, lj_enabled=1, lj_epsilon=1.0, lj_sigma=1.0,
                lj_cutoff=2.5, dt=0.005 * W.TAU_LJ_FS, thermostat=c["thermostat"], temperature=T,
                tau=0.5 * W.TAU_LJ_FS, damp=W.TAU_LJ_FS, seed=int(seed) % 1000003 + 1,
                stress_required=c["stress"])
    return desc, _frame(pos, vel, mass, np.zeros(n)), {}


def _melt(c, seed):
    """Jittered rock-salt lattice of +-1 e ions at 1200 K (the headline
    melt's parameters), nx x ny x nz sites."""
    rng = np.random.default_rng(seed)
    nc = np.array([c["nx"], c["ny"], c["nz"]])
    g = np.stack(np.meshgrid(*[np.arange(k) for k in nc], indexing="ij"), -1).reshape(-1, 3)
    L = nc * 2.82
    pos = (g + 0.5) * 2.82 + rng.uniform(-0.2, 0.2, size=g.shape)
    even = g.sum(1) % 2 == 0
    charge = np.where(even, 1.0, -1.0)
    mass = np.where(even, 23.0, 35.45)
    rc = min(12.0, 0.5 * float(L.min()) - 1.05)
    alpha = W.recommend_alpha(rc, 1e-5)
    grid = tuple(192 if k == 64 else W.good_fft_size(math.ceil(k * 2.82 / 0.94)) for k in nc)
    desc = dict(n_atoms=len(g), box=tuple(float(v) for v in L), precision=c["precision"],
                nl_cutoff=rc, nl_skin=1.0, lj_enabled=1, lj_epsilon=0.5 / W.KJMOL_PER_EV,
                lj_sigma=3.0, lj_cutoff=rc, coul_enabled=1, coul_alpha=alpha, coul_cutoff=rc,
                pme_enabled=1, pme_alpha=alpha, pme_order=c["order"], pme_grid=grid, dt=2.0,
                thermostat=1, temperature=1200.0, tau=100.0)
    return desc, _frame(pos, W.maxwell_velocities(mass, 1200.0, rng), mass, charge), {}


def _mixture(c, seed):
    """Three-type LJ mixture (an explicit cross term, one type without an
    LJ site), Nose-Hoover and a Berendsen barostat."""
    rng = np.random.default_rng(seed)
    a = (4.0 / FLUID_RHO) ** (1.0 / 3.0)
    pos = W.fcc_sites(c["cells"], a) + 0.25 * a
    pos += rng.uniform(-0.06, 0.06, size=pos.shape)
    n, L = len(pos), c["cells"] * a
    T = 1.0 / W.KB
    mass = np.ones(n)
    desc = dict(n_atoms=n, box=(L, L, L), precision=c["precision"], nl_cutoff=2.5, nl_skin=0.3,
                lj_enabled=1, lj_epsilon=1.0, lj_sigma=1.0, lj_cutoff=2.5,
                dt=0.002 * W.TAU_LJ_FS, thermostat=1, temperature=T, tau=0.5 * W.TAU_LJ_FS,
                stress_required=1)
    f = _frame(pos, W.maxwell_velocities(mass, T, rng), mass, np.zeros(n))
    f["type"] = rng.integers(0, 3, size=n).astype(np.int32)
    opts = dict(lj_types=[(0, 0, 1.0, 1.0), (1, 1, 0.5, 0.88), (0, 1, 1.5, 0.8),
                          (2, 2, 0.0, 1.0)],
                barostat=dict(P_target=1.0, tau_P=50.0, dt=desc["dt"], bulk_modulus=10.0))
    return desc, f, opts


def _water(c, seed):
    """SPC/E-like molecules on a cubic lattice at random orientations; LJ on
    the oxygens, intramolecular pairs excluded."""
    rng = np.random.default_rng(seed)
    m, sp = c["m"], 3.1
    L = m * sp
    o = (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * sp
    u = rng.normal(size=o.shape)
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w = rng.normal(size=o.shape)
    w -= (w * u).sum(1, keepdims=True) * u
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    ang = math.radians(109.47)
    pos = np.stack([o, o + u, o + u * math.cos(ang) + w * math.sin(ang)], 1).reshape(-1, 3)
    pos = np.mod(pos, L)
    k = len(o)
    t = 3 * np.arange(k, dtype=np.int64) + 1
    rc = min(9.0, 0.5 * L - 1.05)
    alpha = W.recommend_alpha(rc, 1e-5)
    K = W.good_fft_size(math.ceil(L / 1.0))
    desc = dict(n_atoms=3 * k, box=(L, L, L), precision=c["precision"], nl_cutoff=rc, nl_skin=1.0,
                lj_enabled=1, lj_epsilon=0.0067, lj_sigma=3.166, lj_cutoff=rc, coul_enabled=1,
                coul_alpha=alpha, coul_cutoff=rc, pme_enabled=1, pme_alpha=alpha, pme_order=4,
                pme_grid=(K, K, K), dt=1.0, stress_required=1)
    f = _frame(pos, np.zeros_like(pos), np.tile([15.9994, 1.008, 1.008], k),
               np.tile([-0.8476, 0.4238, 0.4238], k))
    f["type"] = np.tile(np.array([0, 1, 1], np.int32), k)
    bonds = np.concatenate([np.stack([t, t + 1], 1), np.stack([t, t + 2], 1)])
    opts = dict(lj_types=[(0, 0, 0.0067, 3.166)],
                special_bonds=dict(lj=(0.0, 0.0, 0.0), coul=(0.0, 0.0, 0.0), bonds=bonds))
    return desc, f, opts


def _replicas(c, seed):
    """Systems of a ladder: sizes log-uniform, temperatures 0.70 to 1.50."""
    rng = np.random.default_rng(seed)
    k = c["systems"]
    out = []
    # one size per equal share of the log range, so that the total is alike for every seed
    for j, u in enumerate(rng.permutation(k)):
        n = int(round(c["n_min"] * (c["n_max"] / c["n_min"]) ** ((u + 0.5) / k)))
        d = math.ceil((n / 4.0) ** (1.0 / 3.0))
        s = dict(cx=d, cy=d, cz=max(4, math.ceil(n / (4 * d * d))), precision=MIXED,
                 thermostat=2, t_star=0.7 * (1.5 / 0.7) ** (j / max(k - 1, 1)), stress=0)
        s["cx"] = s["cy"] = max(4, d)
        s["drop"] = max(0, min(4 * s["cx"] * s["cy"] * s["cz"] - n, s["cx"] * s["cy"] * s["cz"] // 16))
        out.append(_fluid(s, int(rng.integers(1 << 31))))
    return out


def _requests(c, seed):
    """Fluids (3 of 5) and melts (2 of 5) of log-spaced sizes, mixed precision."""
    rng = np.random.default_rng(seed)
    k = c["requests"]
    out = []
    for j in range(k):
        n = c["n_min"] * (c["n_max"] / c["n_min"]) ** ((j + 0.5) / k)
        s = int(rng.integers(1 << 31))
        if j % 5 in (0, 2, 4):
            d = max(4, round((n / 4.0) ** (1.0 / 3.0)))
            out.append(_fluid(dict(cx=d, cy=d, cz=d, drop=0, precision=MIXED, thermostat=0,
                                   t_star=1.44, stress=0), s))
        else:
            d = max(8, 2 * round(n ** (1.0 / 3.0) / 2))
            out.append(_melt(dict(nx=d, ny=d, nz=d, order=4, precision=MIXED), s))
    order = rng.permutation(k)
    return [out[i] for i in order]


_MAKE = dict(fluid=_fluid, melt=_melt, mixture=_mixture, water=_water)


# -------------------------------------------------------------------- runs

class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    st.ctx = A.Context(0)
    kind = case["kind"]
    if kind == "batch":
        st.batch = A.Batch(st.ctx, [(d, f) for d, f, _ in _replicas(case, seed)])
        st.batch.compute_forces()
    elif kind == "serve":
        st.requests = [(A.make_desc(**d), f) for d, f, _ in _requests(case, seed)]
        st.server = A.Server(st.ctx, 8 << 30)
    else:
        desc, frame, opts = _MAKE[kind](case, seed)
        st.sys = A.System(st.ctx, desc, frame, **opts)
        st.frame = frame
        if kind != "water":
            st.sys.compute_forces()
    return st


def _scalars(sc, stress):
    out = dict(energy=sc["energy"], kinetic=sc["kinetic"])
    if stress:
        out["stress"] = sc["stress"]
    return out


def run(st):
    c = st.case
    if c["kind"] == "batch":
        b = st.batch
        b.step(c["steps"])
        got = [b.download(k, STATE) for k in range(len(b.sizes))]
        out = {k: np.concatenate([f[k] for f, _ in got]) for k in STATE}
        out["energy"] = np.array([s["energy"] for _, s in got])
        return out
    if c["kind"] == "serve":
        s = st.server
        ids = [s.submit(d, f, c["steps"]) for d, f in st.requests]
        s.tick(20)
        while s.stats()["queued"] + s.stats()["running"]:
            s.tick(20)
        got = [s.collect(i) for i in ids]
        out = {k: np.concatenate([f[k] for f, _ in got]) for k in STATE}
        out["energy"] = np.array([r["scalars"]["energy"] for _, r in got])
        return out
    s = st.sys
    if c["kind"] == "water":  # single point: new coordinates in, forces out
        s.upload(st.frame)
        s.compute_forces()
        f, sc = s.download(("fx", "fy", "fz"))
        return dict(f, energy=sc["energy"], stress=sc["stress"])
    s.step(c["steps"])
    f, sc = s.download(FULL)
    stress = bool(c.get("stress")) or c["kind"] == "mixture"
    out = dict(f, **_scalars(sc, stress))
    if c["kind"] == "mixture":
        out["box"] = sc["box"]
    return out


# ------------------------------------------------------------ work, limits

def _work_system(n, vol, rc, coul, mesh, order):
    """Bytes and operations of one force evaluation and step: each pair
    inside the cutoff once, the mesh sums once, the state read and written
    once."""
    pairs = 0.5 * n * (n / vol) * 4.0 / 3.0 * math.pi * rc ** 3
    flops = pairs * (60.0 if coul else 30.0) + 40.0 * n
    byts = n * 20 * 8.0
    if mesh:
        k3 = float(mesh[0] * mesh[1] * mesh[2])
        flops += 5.0 * k3 * math.log2(k3) + 10.0 * k3 + n * order ** 3 * 12.0
        byts += 2 * 8.0 * k3
    return byts, flops


def work(case):
    kind = case["kind"]
    fluid_vol = 1.0 / FLUID_RHO

    def fluid(n):
        return _work_system(n, n * fluid_vol, 2.5, False, None, 0)

    def melt(nx, ny, nz, order):
        L = [k * 2.82 for k in (nx, ny, nz)]
        rc = min(12.0, 0.5 * min(L) - 1.05)
        return _work_system(nx * ny * nz, L[0] * L[1] * L[2], rc, True,
                            [math.ceil(v / 0.94) for v in L], order)

    steps = case.get("steps", 1)
    if kind == "fluid":
        b, f = fluid(4 * case["cx"] * case["cy"] * case["cz"] - case["drop"])
    elif kind == "melt":
        b, f = melt(case["nx"], case["ny"], case["nz"], case["order"])
    elif kind == "mixture":
        b, f = fluid(4 * case["cells"] ** 3)
    elif kind == "water":
        L = case["m"] * 3.1
        b, f = _work_system(3 * case["m"] ** 3, L ** 3, min(9.0, 0.5 * L - 1.05), True, [L] * 3, 4)
    elif kind == "batch":
        k = case["systems"]
        s = [fluid(case["n_min"] * (case["n_max"] / case["n_min"]) ** ((j + 0.5) / k))
             for j in range(k)]
        b, f = sum(v[0] for v in s), sum(v[1] for v in s)
    else:
        b = f = 0.0
        k = case["requests"]
        for j in range(k):
            n = case["n_min"] * (case["n_max"] / case["n_min"]) ** ((j + 0.5) / k)
            d = max(8.0, n ** (1.0 / 3.0))
            w = fluid(n) if j % 5 in (0, 2, 4) else melt(d, d, d, 4)
            b, f = b + w[0], f + w[1]
    return {"bytes": b * steps, "flops": f * steps}


def tolerance(case):
    """About four times the distance from exact() after two passes of a
    state.  FP64: 3e-13 in the fluids, 2e-11 with the mesh (its charges are
    2^-40 fixed point); a virial that is nearly zero carries the fixed-point
    step of its sums (2e-12).  FP32 sums: 3e-6 after a trajectory of a
    hundred steps; the energy of a water box is a small difference of large
    terms (5e-5)."""
    kind = case["kind"]
    if kind in ("batch", "serve") or case["precision"] == MIXED:
        return {"rel": 2e-4 if kind == "water" else 1.5e-5}
    if kind in ("melt", "water"):
        return {"rel": 8e-11}
    return {"rel": 1e-11 if kind == "mixture" or case["stress"] else 2e-12}


# ------------------------------------------------------------------- exact

def _pair_sums(d2, ok, qq, eps4, sig6, lj_rc2, alpha, c_rc2, shift):
    """Force over distance and energies of masked pairs at squared distance d2."""
    safe = torch.where(ok, d2, torch.ones_like(d2))
    inv2 = 1.0 / safe
    fr = torch.zeros_like(d2)
    e = torch.zeros_like(d2)
    if eps4 is not None:
        r6 = inv2 ** 3 * sig6
        m = ok & (d2 < lj_rc2)
        fr += torch.where(m, 6.0 * eps4 * inv2 * r6 * (2.0 * r6 - 1.0), 0.0)
        e += torch.where(m, eps4 * r6 * (r6 - 1.0) - shift, 0.0)
    if qq is not None:
        r = torch.sqrt(safe)
        m = ok & (d2 < c_rc2)
        ec = qq * torch.erfc(alpha * r) / r
        fc = (ec + qq * (2.0 * alpha / math.sqrt(math.pi)) * torch.exp(-alpha ** 2 * safe)) * inv2
        fr += torch.where(m, fc, 0.0)
        e += torch.where(m, ec, 0.0)
    return fr, e


class _Exact:
    """One system in plain torch FP64."""

    def __init__(self, desc, frame, opts):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.d = desc
        self.L = t(desc["box"])
        self.x = torch.stack([t(frame[k]) for k in ("x", "y", "z")], 1)
        self.x -= self.L * torch.floor(self.x / self.L)
        self.v = torch.stack([t(frame[k]) for k in ("vx", "vy", "vz")], 1)
        self.m, self.q = t(frame["mass"]), t(frame["charge"])
        self.tag = np.asarray(frame["tag"]).astype(np.uint64)
        self.n = len(self.m)
        self.baro = opts.get("barostat")
        self.types = None
        self.has_coul = bool(desc.get("coul_enabled"))
        s2 = desc["lj_cutoff"] ** -2
        if opts.get("lj_types"):
            co = opts["lj_types"]
            nt = int(frame["type"].max()) + 1
            eps, sig = np.zeros((nt, nt)), np.ones((nt, nt))
            diag = {i: (e, s) for i, j, e, s in co if i == j}
            for i in range(nt):
                for j in range(nt):
                    if i in diag and j in diag:
                        eps[i, j] = math.sqrt(diag[i][0] * diag[j][0])
                        sig[i, j] = 0.5 * (diag[i][1] + diag[j][1])
            for i, j, e, s in co:
                eps[i, j] = eps[j, i] = e
                sig[i, j] = sig[j, i] = s
            self.types = torch.as_tensor(frame["type"].astype(np.int64), device=self.dev)
            self.eps4, self.sig6 = t(4.0 * eps), t(sig ** 6)
            r6 = s2 ** 3 * self.sig6
            self.shift = self.eps4 * r6 * (r6 - 1.0)
        else:
            self.eps4, self.sig6 = 4.0 * desc["lj_epsilon"], desc["lj_sigma"] ** 6
            r6 = s2 ** 3 * self.sig6
            self.shift = self.eps4 * r6 * (r6 - 1.0)
        self.excluded = None
        if opts.get("special_bonds"):
            b = np.asarray(opts["special_bonds"]["bonds"]) - 1  # 1-2, and 1-3 through the oxygen
            k = len(b) // 2
            both = np.concatenate([b, np.stack([b[:k, 1], b[k:, 1]], 1)])
            self.excluded = torch.as_tensor(both, device=self.dev)
        self.f = torch.zeros_like(self.x)
        self.xi, self.vscale, self.step = 0.0, 1.0, 0

    # ---- forces

    def _block(self, xi, xj, ai, aj, same):
        """Forces on the atoms ai from aj (index -1: empty), and sums."""
        d = xi[..., :, None, :] - xj[..., None, :, :]
        d -= self.L * torch.round(d / self.L)
        d2 = (d * d).sum(-1)
        ok = (ai >= 0)[..., :, None] & (aj >= 0)[..., None, :]
        if same:
            ok &= ai[..., :, None] != aj[..., None, :]
        si, sj = ai.clamp(min=0), aj.clamp(min=0)
        qq = None
        if self.has_coul:
            qq = 14.399645 * self.q[si][..., :, None] * self.q[sj][..., None, :]
        e4, s6, sh = self.eps4, self.sig6, self.shift
        if self.types is not None:
            ti, tj = self.types[si][..., :, None], self.types[sj][..., None, :]
            e4, s6, sh = e4[ti, tj], s6[ti, tj], sh[ti, tj]
        dd = self.d
        fr, e = _pair_sums(d2, ok, qq, e4, s6, dd["lj_cutoff"] ** 2, dd.get("coul_alpha", 0.0),
                           dd.get("coul_cutoff", 0.0) ** 2, sh)
        f = torch.einsum("...ij,...ijk->...ik", fr, d)
        self.e_pair += 0.5 * float(e.sum())
        if dd.get("stress_required") or self.baro:
            w = torch.einsum("...ija,...ij,...ijb->ab", d, fr, d)
            self.W += 0.5 * w
        return f

    def forces(self):
        n, dev = self.n, self.dev
        rc = max(self.d["lj_cutoff"], self.d.get("coul_cutoff", 0.0))
        self.e_pair = 0.0
        self.W = torch.zeros(3, 3, dtype=torch.float64, device=dev)
        f = torch.zeros_like(self.x)
        nc = torch.floor(self.L / rc).long()
        if n <= 3000 or int(nc.min()) < 3:
            idx = torch.arange(n, device=dev)
            for b in range(0, n, max(1, 20_000_000 // n)):
                ai = idx[b:b + max(1, 20_000_000 // n)]
                f[ai] += self._block(self.x[ai], self.x, ai, idx, True)
        else:
            c = torch.minimum((self.x / self.L * nc).long(), nc - 1)
            cell = (c[:, 0] * nc[1] + c[:, 1]) * nc[2] + c[:, 2]
            ncell = int(nc.prod())
            order = torch.argsort(cell)
            cnt = torch.bincount(cell, minlength=ncell)
            start = torch.cumsum(cnt, 0) - cnt
            M = int(cnt.max())
            table = torch.full((ncell, M), -1, dtype=torch.long, device=dev)
            cs = cell[order]
            table[cs, torch.arange(n, device=dev) - start[cs]] = order
            ids = torch.arange(ncell, device=dev)
            c3 = torch.stack([ids // (nc[1] * nc[2]), (ids // nc[2]) % nc[1], ids % nc[2]], 1)
            step = max(1, 20_000_000 // (M * M))
            for b in range(0, ncell, step):
                ai = table[b:b + step]
                xi = self.x[ai.clamp(min=0)]
                acc = torch.zeros_like(xi)
                for ox in (-1, 0, 1):
                    for oy in (-1, 0, 1):
                        for oz in (-1, 0, 1):
                            o = torch.tensor([ox, oy, oz], device=dev)
                            k3 = (c3[b:b + step] + o) % nc
                            aj = table[(k3[:, 0] * nc[1] + k3[:, 1]) * nc[2] + k3[:, 2]]
                            acc += self._block(xi, self.x[aj.clamp(min=0)], ai, aj,
                                               (ox, oy, oz) == (0, 0, 0))
                on = ai >= 0
                f[ai[on]] = acc[on]
        self.energy = self.e_pair
        if self.excluded is not None:
            i, j = self.excluded[:, 0], self.excluded[:, 1]
            d = self.x[i] - self.x[j]
            d -= self.L * torch.round(d / self.L)
            r = torch.sqrt((d * d).sum(1))
            e = 14.399645 * self.q[i] * self.q[j] / r
            fv = (e / r ** 2)[:, None] * d
            f.index_add_(0, i, -fv)
            f.index_add_(0, j, fv)
            self.energy -= float(e.sum())
            self.W -= torch.einsum("ia,ib->ab", d, fv)
        if self.d.get("pme_enabled"):
            f += self._mesh()
        self.f = f

    def _splines(self, u, order):
        """B-spline weights M_n(frac + n - 1 - k) and their derivatives."""
        w = [1.0 - u, u]
        for k in range(3, order + 1):
            if k == order:
                dw = [-w[0]] + [w[j - 1] - w[j] for j in range(1, order - 1)] + [w[order - 2]]
            new = []
            for j in range(k):
                a = w[j - 1] if j > 0 else None
                b = w[j] if j < k - 1 else None
                t = 0.0
                if a is not None:
                    t = t + (u + (k - 1 - j)) * a
                if b is not None:
                    t = t + ((j + 1) - u) * b
                new.append(t / (k - 1))
            w = new
        return torch.stack(w, 1), torch.stack(dw, 1)

    def _mesh(self):
        dd, dev, n = self.d, self.dev, self.n
        K, p = dd["pme_grid"], dd["pme_order"]
        alpha = dd["pme_alpha"]
        th, dth, ix = [], [], []
        for a in range(3):
            u = self.x[:, a] / self.L[a] * K[a]
            fl = torch.floor(u)
            w, dw = self._splines(u - fl, p)
            th.append(w)
            dth.append(dw)
            ix.append((fl.long()[:, None] + torch.arange(p, device=dev) - (p - 1)) % K[a])
        flat = ((ix[0][:, :, None, None] * K[1] + ix[1][:, None, :, None]) * K[2]
                + ix[2][:, None, None, :]).reshape(n, -1)

        def prod(a, b, c):
            return (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(n, -1)

        grid = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=dev)
        grid.index_add_(0, flat.reshape(-1), (self.q[:, None] * prod(*th)).reshape(-1))
        S = torch.fft.fftn(grid.reshape(K))
        m2, ms, B = 0.0, [], 1.0
        zero = torch.zeros(1, dtype=torch.float64, device=dev)
        w0 = self._splines(zero, p)[0][0]
        for a in range(3):
            k = torch.arange(K[a], device=dev, dtype=torch.float64)
            ph = torch.exp(2j * math.pi * k[:, None] * torch.arange(p, device=dev) / K[a])
            b = 1.0 / (ph * w0).sum(1).abs() ** 2
            mm = torch.where(k > K[a] / 2, k - K[a], k) / self.L[a]
            shape = [1, 1, 1]
            shape[a] = K[a]
            ms.append(mm.reshape(shape))
            m2 = m2 + ms[a] ** 2
            B = B * b.reshape(shape)
        V = float(self.L.prod())
        m2s = m2.clone()
        m2s[0, 0, 0] = 1.0
        G = 14.399645 / (math.pi * V) * torch.exp(-math.pi ** 2 * m2s / alpha ** 2) / m2s * B
        G[0, 0, 0] = 0.0
        em = 0.5 * G * S.abs() ** 2
        self.energy += float(em.sum())
        self.energy -= 14.399645 * alpha / math.sqrt(math.pi) * float((self.q ** 2).sum())
        fac = 2.0 * (1.0 / m2s + math.pi ** 2 / alpha ** 2)
        for a in range(3):
            for b in range(3):
                w = -fac * ms[a] * ms[b] + (1.0 if a == b else 0.0)
                self.W[a, b] += (em * w).sum()
        phi = torch.fft.ifftn(S * G).real.reshape(-1) * (K[0] * K[1] * K[2])
        g = phi[flat]
        out = torch.stack([(g * prod(dth[0], th[1], th[2])).sum(1) * K[0] / self.L[0],
                           (g * prod(th[0], dth[1], th[2])).sum(1) * K[1] / self.L[1],
                           (g * prod(th[0], th[1], dth[2])).sum(1) * K[2] / self.L[2]], 1)
        return -self.q[:, None] * out

    # ---- integration

    def _ke(self):
        return 0.5 * W.MVV2E * float((self.m[:, None] * self.v ** 2).sum())

    def _gauss(self):
        with np.errstate(over="ignore"):
            s = (np.uint64(self.d["seed"]) * np.uint64(0x9E3779B97F4A7C15)
                 + np.uint64(self.step) * np.uint64(0xBF58476D1CE4E5B9)
                 + self.tag * np.uint64(0xD6E8FEB86659FD93))

            def u01():
                nonlocal s
                s = s + np.uint64(0x9E3779B97F4A7C15)
                z = s
                z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
                z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
                z = z ^ (z >> np.uint64(31))
                return (z >> np.uint64(11)).astype(np.float64) / 9007199254740992.0

            def polar():
                r = np.sqrt(-2.0 * np.log(np.maximum(u01(), 1e-300)))
                a = 2.0 * np.pi * u01()
                return r * np.cos(a), r * np.sin(a)

            (a, b), (c, _) = polar(), polar()
        return torch.as_tensor(np.stack([a, b, c], 1), device=self.dev)

    def advance(self, steps):
        d = self.d
        dt, kind = d["dt"], d.get("thermostat", 0)
        ftm2v = 1.0 / W.MVV2E
        dtfm = (0.5 * dt * ftm2v / self.m)[:, None]
        ndof = 3 * self.n - 3
        kT = W.KB * d.get("temperature", 0.0)
        for _ in range(steps):
            self.v = self.v * self.vscale + dtfm * self.f
            self.x = self.x + dt * self.v
            self.x -= self.L * torch.floor(self.x / self.L)
            sa = 1.0
            if kind == 1:
                Q = ndof * kT * d["tau"] ** 2
                self.xi += 0.5 * dt * (2.0 * self._ke() - ndof * kT) / Q
                sa = math.exp(-0.5 * dt * self.xi)
            self.forces()
            self.v = self.v * sa
            if kind == 2:
                g1 = 1.0 / (d["damp"] * ftm2v)
                g2 = math.sqrt(2.0 * kT / (d["damp"] * dt * W.MVV2E)) / ftm2v
                self.f = (self.f - g1 * self.m[:, None] * self.v
                          + g2 * torch.sqrt(self.m)[:, None] * self._gauss())
            self.v = self.v + dtfm * self.f
            self.vscale = 1.0
            ke = self._ke()
            if kind == 1:
                self.xi += 0.5 * dt * (2.0 * ke - ndof * kT) / Q
                self.vscale = math.exp(-0.5 * dt * self.xi)
                ke *= self.vscale ** 2
            self.kinetic = ke
            self.step += 1
            if self.baro:
                b = self.baro
                P = (2.0 * ke + float(self.W.diagonal().sum())) / (3.0 * float(self.L.prod()))
                mu3 = 1.0 - dt / (b["tau_P"] * b["bulk_modulus"]) * (b["P_target"] - P)
                mu = min(max(mu3, 0.5), 2.0) ** (1.0 / 3.0)
                self.L = self.L * mu
                self.x = self.x * mu

    def state(self, keys):
        v = self.v * self.vscale
        cols = dict(x=self.x[:, 0], y=self.x[:, 1], z=self.x[:, 2], vx=v[:, 0], vy=v[:, 1],
                    vz=v[:, 2], fx=self.f[:, 0], fy=self.f[:, 1], fz=self.f[:, 2])
        return {k: cols[k].cpu().numpy() for k in keys}

    def stress(self):
        w = self.W
        return torch.stack([w[0, 0], w[1, 1], w[2, 2], w[0, 1], w[0, 2], w[1, 2]]).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        items = (_replicas if kind == "batch" else _requests)(case, seed)
        if sum(d["n_atoms"] * case["steps"] for d, _, _ in items) > 2e7:
            return None
        done = []
        for it in items:
            e = _Exact(*it)
            e.forces()
            e.advance(case["steps"])
            done.append(e)
        states = [e.state(STATE) for e in done]
        out = {k: np.concatenate([s[k] for s in states]) for k in STATE}
        out["energy"] = np.array([e.energy for e in done])
        return out
    e = _Exact(*_MAKE[kind](case, seed))
    e.forces()
    if kind == "water":
        return dict(e.state(("fx", "fy", "fz")), energy=e.energy, stress=e.stress())
    e.advance(case["steps"])
    out = e.state(FULL)
    out.update(energy=e.energy, kinetic=e.kinetic)
    if case.get("stress") or kind == "mixture":
        out["stress"] = e.stress()
    if kind == "mixture":
        out["box"] = e.L.cpu().numpy()
    return out
