"""What a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values.  `listed()` names the standing ones, `draw()`
gives one more of the same ranges, `prepare()` builds what a program holds
before the call (a context with its state, from the seed alone), `run()` is one
pass through the public entry points, `work()` counts what a pass cannot do
without, and `exact()` restates the pass in 64 bits with plain torch.

Kinds of case:
  run       restore a state, step it `steps` times, read the state back into
            CUDA tensors: a chunk of a simulation between two outputs
  source    the source-term loop: read the state, form tendencies from it,
            hand them over, step
  exchange  the state in from pinned host arrays, one step, the state out
  ensemble  members of uneven size stepped together
  adjoint   a window forward and its gradients
  keysort   the stable key sort without allocation

Atmospheres (cells, particles per cell and physics of this repository's
configurations; the box follows the lattice, so a lattice of any size keeps
the spacing and the cells):
  bubble    the 2,097,152-particle moist bubble: 150 x 150 x 40 m cells,
            0.6 particles per cell, a sort every step
  small     the 65,536-particle box: 200 x 200 x 50 m cells, 0.26 per cell,
            displacement-gated sorts
  dense     the 262,144-particle adjoint box: the same cells, 1.05 per cell
  large     the 16,777,216-particle run: 160 x 160 x 20 m cells, 0.54 per cell
  reference the reference's own physics and cells, one particle per cell, its
            displacement-gated sorts
"""
import ctypes
import math

import numpy as np
import torch

import sph_cuda_gb300 as sph
from sph_cuda_gb300 import abi
from sph_cuda_gb300.adjoint import AdjointWindow

# lattice spacing [m] and cell edge asked for [m] of each atmosphere
_ATM = {
    "bubble": ((156.25, 156.25, 62.5), (150.0, 150.0, 40.0)),
    "small": ((312.5, 312.5, 78.125), (200.0, 200.0, 50.0)),
    "dense": ((156.25, 156.25, 78.125), (200.0, 200.0, 50.0)),
    "large": ((156.25, 156.25, 39.0625), (160.0, 160.0, 20.0)),
    "reference": ((1000.0, 1000.0, 100.0), (1000.0, 1000.0, 100.0)),
}
_PRESET = {"bubble": "bubble2m", "small": "small65k", "dense": "adjoint262k", "large": "large16m",
           "reference": "reference"}
_FIELDS = ("x", "y", "z", "u", "v", "w", "th", "qv", "qc", "rho", "ax", "ay", "az")
_MOST = 256 ** 3 * 3   # particle-steps of the largest listed case


def listed():
    return [
        # one step of the smallest ensemble member by itself: launches and latency
        {"name": "single_step_16k", "kind": "run", "atm": "small", "lx": 20, "ly": 20, "lz": 41, "steps": 1,
         "developed": False},
        # the small preset between two looks at it, at the reference's sort cadence
        {"name": "small_65k", "kind": "run", "atm": "small", "lx": 32, "ly": 32, "lz": 64, "steps": 10,
         "developed": False},
        # an ordinary run on a ragged lattice, a sort every step
        {"name": "bubble_475k", "kind": "run", "atm": "bubble", "lx": 97, "ly": 83, "lz": 59, "steps": 10,
         "developed": False},
        # the headline workload
        {"name": "bubble_2m", "kind": "run", "atm": "bubble", "lx": 128, "ly": 128, "lz": 128, "steps": 10,
         "developed": False},
        # the same later on: updrafts, clustered particles, cloud and rain
        {"name": "bubble_2m_developed", "kind": "run", "atm": "bubble", "lx": 128, "ly": 128, "lz": 128, "steps": 10,
         "developed": True},
        # the reference's own configuration at its own cadence
        {"name": "reference_2m", "kind": "run", "atm": "reference", "lx": 128, "ly": 128, "lz": 128, "steps": 10,
         "developed": False},
        # the largest configuration
        {"name": "large_16m", "kind": "run", "atm": "large", "lx": 256, "ly": 256, "lz": 256, "steps": 3,
         "developed": False},
        # a model's tendencies every step
        {"name": "source_262k", "kind": "source", "atm": "dense", "lx": 64, "ly": 64, "lz": 64, "steps": 2,
         "developed": False},
        # a host program that owns the state
        {"name": "exchange_475k", "kind": "exchange", "atm": "bubble", "lx": 97, "ly": 83, "lz": 59, "steps": 1,
         "developed": False},
        # an ensemble of uneven members
        {"name": "ensemble_16", "kind": "ensemble", "members": 16, "lo": 16384, "hi": 524288, "steps": 5},
        # gradients over a window
        {"name": "adjoint_262k", "kind": "adjoint", "atm": "dense", "lx": 64, "ly": 64, "lz": 64, "steps": 6,
         "every": 3, "developed": False},
        # the key sort of a caller that must not allocate
        {"name": "keysort_300k", "kind": "keysort", "n": 300007, "bits": 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, lo, hi):
    """Lattice counts of about a log-uniform number of particles, each axis its own size."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    e = (n / (a * b)) ** (1.0 / 3.0)
    return max(12, int(round(e * a))), max(12, int(round(e * b))), max(12, int(round(e)))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["source", "exchange", "ensemble", "adjoint", "keysort"])
    if kind == "keysort":
        return {"kind": kind, "n": _log_int(rng, 10000, 524288), "bits": rng.choice([21, 24, 27, 30])}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(4, 24), "lo": 16384, "hi": _log_int(rng, 65536, 524288),
                "steps": rng.randint(2, 6)}
    if kind == "adjoint":
        lx, ly, lz = _lattice(rng, 30000, 300000)
        steps = rng.randint(3, 8)
        return {"kind": kind, "atm": rng.choice(["dense", "small"]), "lx": lx, "ly": ly, "lz": lz, "steps": steps,
                "every": rng.randint(2, 4), "developed": False}
    atm = rng.choice(sorted(_ATM))
    # the big sizes stay within the reference's 1024 cells per axis on every atmosphere
    lx, ly, lz = _lattice(rng, 16384, 6000000 if kind == "run" else 600000)
    n = lx * ly * lz
    steps = 1 if kind == "exchange" else max(1, min(rng.choice([1, 2, 5, 10]), _MOST // n))
    if kind == "source":
        steps = min(steps, 3)
    return {"kind": kind, "atm": atm, "lx": lx, "ly": ly, "lz": lz, "steps": steps,
            "developed": kind == "run" and rng.random() < 0.4}


# ---------------------------------------------------------------------------
# configurations and states
# ---------------------------------------------------------------------------
def _params(case):
    """The atmosphere's parameters on the case's lattice."""
    lat = (case["lx"], case["ly"], case["lz"])
    n = lat[0] * lat[1] * lat[2]
    spacing, edge = _ATM[case["atm"]]
    if case["atm"] == "reference":
        p = sph.preset("reference", *lat)
        p.dt_request = 0.25
        return p
    p = sph.preset(_PRESET[case["atm"]])
    box = [a * s for a, s in zip(lat, spacing)]
    p.nx, p.ny, p.nz = (int(b // e) for b, e in zip(box, edge))
    p.dx, p.dy, p.dz = box[0] / p.nx, box[1] / p.ny, box[2] / p.nz
    p.lat_nx, p.lat_ny, p.lat_nz = lat
    p.n_particles = n
    return p


def _ensemble_params(case, seed):
    """Sizes from the case, not from the seed, so that every seed costs the same."""
    members = sph.ensemble_members(case["members"], seed=11, lo=case["lo"], hi=case["hi"])
    for k, p in enumerate(members):
        p.seed = seed * 64 + k
    return members


class _Air:
    """The run constants of a parameter set in 64 bits, with the reference's sounding."""
    G, RD, CP, P0, LV, SIG = 9.80665, 287.05, 1004.0, 1.0e5, 2.501e6, 1.0 / math.pi

    def __init__(self, p):
        f = np.float32
        self.n = (int(p.nx), int(p.ny), int(p.nz))
        self.d = tuple(float(a) for a in (p.dx, p.dy, p.dz))
        self.inv32 = tuple(float(f(1) / f(a)) for a in self.d)   # cells come from the rounded float product
        self.L = tuple(float(f(n) * f(a)) for n, a in zip(self.n, self.d))
        self.N = int(p.n_particles)
        self.ncell = self.n[0] * self.n[1] * self.n[2]
        for k in ("th0", "n2", "cs", "qv_mode", "qv0", "rh", "rh_bl", "z_bl", "sponge_sigma", "sponge_frac",
                  "dthdt_cap", "surface_flux", "c_h", "c_e", "beta_moist", "v_bg", "dts_skin", "ramp", "qc_auto",
                  "rate_auto", "v_rain", "theta_cap", "qv_cap", "accretion", "rain_evap", "k_accr", "cfl",
                  "adaptive_dt", "sort_every", "permute_acc"):
            setattr(self, k, getattr(p, k))
        self.alpha, self.beta = float(p.alpha_av), float(p.beta_av)
        self.h_av = p.h_av if p.h_av > 0 else 2.0 * self.d[2]
        self.eta2 = (0.01 * self.h_av) ** 2
        self.a = self.G ** 2 / (self.CP * self.th0 * self.n2)
        self.v_cell = self.d[0] * self.d[1] * self.d[2]
        self.pmass = self.P0 / (self.RD * self.th0) * self.v_cell * self.ncell / self.N
        self.mm = self.pmass / self.v_cell
        static = p.cfl * min(self.d) / p.cs
        self.dt_cap = min(p.dt_request, static) if p.dt_request > 0 else static

    def th_ref(self, z):
        return self.th0 * torch.exp(self.n2 * z / self.G)

    def ex_ref(self, z):
        return 1.0 - self.a * (1.0 - torch.exp(-self.n2 * z / self.G))

    def p_ref(self, z):
        return self.P0 * self.ex_ref(z) ** (self.CP / self.RD)

    def rho_ref(self, z):
        return self.p_ref(z) / (self.RD * self.th_ref(z) * self.ex_ref(z))

    def esat(self, T):
        return 611.2 * torch.exp(17.67 * (T - 273.15) / (T - 273.15 + 243.5))

    def qsat(self, T, p):
        es = torch.minimum(self.esat(T), 0.5 * p)
        return 0.622 * es / (p - 0.378 * es)

    def qv_ref(self, z):
        if self.qv_mode == abi.QV_REFERENCE:
            return self.qv0 * torch.exp(-z / 2500.0) * torch.exp(-torch.clamp(z - 5000.0, min=0.0) / 1000.0)
        q = self.qsat(self.th_ref(z) * self.ex_ref(z), self.p_ref(z))
        return torch.where(z < self.z_bl, self.rh_bl, self.rh) * q

    def thv_ref(self, z):
        return self.th_ref(z) * (1.0 + 0.608 * self.qv_ref(z))

    def cells(self, x, y, z):
        """Cell of a position: the rounded float product, truncated and clamped."""
        return [torch.clamp((c.float() * torch.tensor(i, dtype=torch.float32, device=c.device)).to(torch.int64), 0, n - 1)
                for c, i, n in zip((x, y, z), self.inv32, self.n)]


def _state(p, seed, lattice, developed):
    """A moist state on a jittered lattice, as float32 CUDA tensors in lattice
    order: warm bubbles that rise and draw air in below, vapour near
    saturation and cloud water inside them, light rain in their cells.
    Developed: updrafts of tens of metres per second, a disordered lattice and
    particles drawn together by eddies of some sixteen cells (up to eight times
    the mean density, a mean of about one and a half neighbours for each one
    of the lattice, as a run has after some hundred steps)."""
    A = _Air(p)
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    dev, f64 = "cuda", torch.float64
    i = torch.arange(A.N, device=dev)
    nx, ny, nz = lattice
    ijk = (i % nx, (i // nx) % ny, i // (nx * ny))
    jit = 0.45 if developed else 0.25
    q = [(k.to(f64) + 0.5 + jit * (2.0 * torch.rand(A.N, generator=g, device=dev, dtype=f64) - 1.0)) * (L / n)
         for k, L, n in zip(ijk, A.L, lattice)]
    nb = 3
    at = torch.rand(nb, 3, generator=g, device=dev, dtype=f64).tolist()
    speed = 35.0 if developed else 3.0
    warm = torch.zeros(A.N, device=dev, dtype=f64)
    vel = [0.5 * torch.randn(A.N, generator=g, device=dev, dtype=f64) for _ in range(3)]
    for b in range(nb):
        c = [(0.2 + 0.6 * at[b][0]) * A.L[0], (0.2 + 0.6 * at[b][1]) * A.L[1], (0.2 + 0.3 * at[b][2]) * A.L[2]]
        r = [max(0.08 * A.L[0], 2.5 * A.d[0]), max(0.08 * A.L[1], 2.5 * A.d[1]), max(0.14 * A.L[2], 2.5 * A.d[2])]
        d = [a - m for a, m in zip(q, c)]
        e = torch.exp(-sum((a / s) ** 2 for a, s in zip(d, r)))
        warm = warm + e
        vel[0] = vel[0] - 0.15 * speed * e * d[0] / r[0]
        vel[1] = vel[1] - 0.15 * speed * e * d[1] / r[1]
        vel[2] = vel[2] + speed * e
    if developed:
        amp = 0.5 if A.N < 0.7 * A.ncell else 0.35
        for k in range(3):
            turns = max(1, round(A.n[k] / 16))
            ph = 2.0 * math.pi * (q[k] * (turns / A.L[k]))
            q[k] = q[k] + amp * A.L[k] / (2.0 * math.pi * turns) * torch.sin(ph)
    top = [torch.tensor(L, dtype=torch.float32, device=dev) for L in A.L]
    x, y, z = (torch.minimum(torch.clamp(a.float(), min=0.0), torch.nextafter(t, torch.zeros_like(t)))
               for a, t in zip(q, top))
    zd = z.to(f64)
    th = A.th_ref(zd) + 2.0 * warm + 0.05 * torch.randn(A.N, generator=g, device=dev, dtype=f64)
    qs = A.qsat(th * A.ex_ref(zd), A.p_ref(zd))
    qv = torch.clamp(torch.minimum(A.qv_ref(zd) * (1.0 + 0.4 * warm), 1.02 * qs), 0.0, 0.05)
    qc = torch.where(warm > 0.5, (2.0e-3 if developed else 4.0e-4) * warm, torch.zeros_like(warm))
    rho = A.rho_ref(zd) * (1.0 + 1.0e-3 * warm)
    s = dict(x=x, y=y, z=z, u=vel[0], v=vel[1], w=vel[2], th=th, qv=qv, qc=qc, rho=rho)
    for k in ("ax", "ay"):
        s[k] = torch.zeros(A.N, device=dev)
    s["az"] = 0.05 * warm
    s = {k: v.float().contiguous() for k, v in s.items()}
    cx, cy, cz = A.cells(s["x"], s["y"], s["z"])
    rain = torch.zeros(A.ncell, device=dev, dtype=torch.float32)
    rain[((cz * A.n[1] + cy) * A.n[0] + cx)[warm > 0.3]] = float(1.0e-4 * A.v_cell)   # about 0.1 g of rain a kg
    return s, rain


def _host(t):
    return {k: v.cpu().numpy() for k, v in t.items()}


def _context(p, s, rain):
    sim = sph.Asph(p)
    sim.set_state(_host(s))
    sim.set_rain(rain.cpu().numpy())
    return sim


def _lat(case):
    return case["lx"], case["ly"], case["lz"]


def _buffers(n):
    return [torch.empty(n, 4, device="cuda", dtype=torch.float32) for _ in range(3)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "keysort":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        keys = _keys(case, g)
        return {"kind": kind, "keys": keys, "sorted": torch.empty_like(keys), "perm": torch.empty_like(keys),
                "bits": case["bits"], "lib": sph.library()}
    if kind == "ensemble":
        members = _ensemble_params(case, seed)
        ens = sph.Ensemble(members)
        total = ens.n_particles
        st = {"kind": kind, "ens": ens, "steps": case["steps"], "snaps": [], "out": _buffers(total)}
        for k, p in enumerate(members):
            s, rain = _state(p, seed * 64 + k, (p.lat_nx, p.lat_ny, p.lat_nz), False)
            m = ens.member(k)
            m.set_state(_host(s))
            m.set_rain(rain.cpu().numpy())
            m.sort_build()
            st["snaps"].append(m.snapshot())
        return st
    p = _params(case)
    s, rain = _state(p, seed, _lat(case), case["developed"])
    sim = _context(p, s, rain)
    st = {"kind": kind, "sim": sim, "steps": case["steps"]}
    if kind == "exchange":
        # the host program's arrays, pinned; the state goes in and out in the context's order
        st["in"] = {k: s[k].cpu().pin_memory().numpy() for k in _FIELDS}
        st["out"] = {k: torch.empty(p.n_particles, dtype=torch.float32, pin_memory=True).numpy() for k in _FIELDS}
        st["rain"] = sim.snapshot()
        return st
    if kind == "adjoint":
        sim.sort_build()
        st["window"] = AdjointWindow(sim, case["steps"], case["every"])
        st["theta0"] = sim.get_state(("th",))["th"]
        st["dqc"], st["dxyz"] = (v.cpu().numpy() for v in _loss(p.n_particles, seed))
        return st
    sim.sort_build()
    if kind == "source":
        sim.enable_source()
        st["tend"] = torch.zeros(p.n_particles, 4, device="cuda", dtype=torch.float32)
    st["snap"] = sim.snapshot()
    st["out"] = _buffers(p.n_particles)
    return st


def _keys(case, g):
    """Keys all over the range, a quarter of them twice."""
    n = case["n"]
    keys = torch.randint(0, 1 << case["bits"], (n,), generator=g, device="cuda", dtype=torch.int64)
    keys[:n // 4] = keys[n // 4:2 * (n // 4)]
    return keys.to(torch.int32)


def _loss(n, seed):
    """dL/d(final cloud water) and dL/d(final positions) of a misfit, as a caller hands them over."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2)
    dqc = torch.randn(n, generator=g, device="cuda", dtype=torch.float32) / n
    dxyz = 1.0e-6 * torch.randn(3 * n, generator=g, device="cuda", dtype=torch.float32) / n
    return dqc, dxyz


def _tendencies(thq, out):
    """A cheap stand-in for a model's output: cooling of cloudy air, relaxation of vapour."""
    out[:, 0] = -1.0e-4 - 1.0e-2 * thq[:, 2]
    out[:, 1] = -1.0e-5 * thq[:, 1]
    out[:, 2] = -1.0e-5 * thq[:, 2]
    return out


def run(state):
    kind = state["kind"]
    if kind == "keysort":
        ptr = [ctypes.c_void_p(state[k].data_ptr()) for k in ("keys", "sorted", "perm")]
        st = state["lib"].asph_sort_keys_noalloc(*ptr, state["keys"].numel(), state["bits"],
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != abi.ASPH_OK:
            raise RuntimeError("key sort failed: %d" % st)
        return {"keys": state["sorted"], "perm": state["perm"]}
    if kind == "ensemble":
        ens = state["ens"]
        for k, snap in enumerate(state["snaps"]):
            ens.member(k).restore(snap)
        ens.step(state["steps"])
        pos, vel, thq = state["out"]
        at = 0
        for k in range(len(ens)):
            m = ens.member(k)
            m.state_device(pos[at:at + m.N], vel[at:at + m.N], thq[at:at + m.N])
            at += m.N
        return {"pos": pos, "vel": vel, "thq": thq}
    sim = state["sim"]
    if kind == "exchange":
        sim.restore(state["rain"])   # the rain grid and the clock of the pass; the particles come from the host
        sim.set_state(state["in"])
        sim.step(1)
        return sim.get_state(_FIELDS, out=state["out"])
    if kind == "adjoint":
        fin = state["window"].forward(state["theta0"])
        dth, da, db = state["window"].backward(dL_dqc=state["dqc"], dL_dxyz=state["dxyz"])
        return {"theta": fin["th"], "qv": fin["qv"], "qc": fin["qc"],
                "xyz": np.stack([fin["x"], fin["y"], fin["z"]]), "dtheta0": dth, "dalpha": da, "dbeta": db}
    pos, vel, thq = state["out"]
    sim.restore(state["snap"])
    if kind == "source":
        for _ in range(state["steps"]):
            sim.state_device(thq=thq)
            sim.set_source_device(_tendencies(thq, state["tend"]))
            sim.step(1)
    else:
        sim.step(state["steps"])
    sim.state_device(pos, vel, thq)
    return {"pos": pos, "vel": vel, "thq": thq}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(n, ncell, crowd):
    """One step of n particles: thirteen fields in and out and the rain grid in
    and out; per particle the window's candidate tests (125 cells, 8
    operations each), the accepted pairs (a ball of radius two cells, 20
    operations in the density and 60 in the momentum sums) and about 300 of
    point physics."""
    ppc = crowd * n / ncell
    return 104.0 * n + 8.0 * ncell, n * (125.0 * ppc * 8.0 + 33.5 * ppc * 80.0 + 300.0)


def work(case):
    kind = case["kind"]
    if kind == "keysort":
        return {"bytes": 12.0 * case["n"], "flops": 0.0}
    if kind == "ensemble":
        w = [_step_work(p.n_particles, p.nx * p.ny * p.nz, 1.0) for p in _ensemble_params(case, 0)]
        return {"bytes": case["steps"] * sum(a for a, _ in w), "flops": case["steps"] * sum(b for _, b in w)}
    p = _params(case)
    b, f = _step_work(p.n_particles, p.nx * p.ny * p.nz, 1.5 if case["developed"] else 1.0)
    # an adjoint pass steps the window and takes the reverse of it, about twice the step's operations
    reps = 3 * case["steps"] if kind == "adjoint" else case["steps"]
    return {"bytes": b * reps, "flops": f * reps}


# ---------------------------------------------------------------------------
# the same passes in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """The step in 64 bits with plain torch.  What one step hands to the next
    is rounded to float32, as the framework's state is; a particle's cell is
    defined by its float32 position."""

    def __init__(self, p, s, rain):
        self.A = _Air(p)
        self.s = {k: s[k].double() for k in _FIELDS}
        self.rain = rain.double()
        self.dt, self.simt, self.since_sort, self.step_no, self.do_sort = self.A.dt_cap, 0.0, 1e9, 0, True
        self.sorted_now = False
        self.lag = self.s["rho"]

    def order(self, move_acc, carry=()):
        """Stable sort by Morton key, the cell table and the surface flags."""
        A, s = self.A, self.s
        cx, cy, cz = A.cells(s["x"].detach(), s["y"].detach(), s["z"].detach())
        key = torch.zeros_like(cx)
        for b in range(10):
            for k, c in enumerate((cx, cy, cz)):
                key |= ((c >> b) & 1) << (3 * b + k)
        perm = torch.sort(key, stable=True).indices
        for k in list(s):
            if not (k in ("ax", "ay", "az") and not move_acc):
                s[k] = s[k][perm]
        cid = ((cz * A.n[1] + cy) * A.n[0] + cx)[perm]
        new = torch.ones(A.N, dtype=torch.bool, device=cid.device)
        new[1:] = cid[1:] != cid[:-1]
        at = torch.nonzero(new).flatten()
        self.first = torch.zeros(A.ncell, dtype=torch.int64, device=cid.device)
        self.count = torch.zeros_like(self.first)
        self.first[cid[at]] = at
        self.count[cid[at]] = torch.diff(at, append=torch.tensor([A.N], device=at.device))
        self.surf = (s["z"].detach().float() * torch.tensor(A.inv32[2], dtype=torch.float32, device=cid.device)).to(torch.int64) == 0
        self.sorted_now = True
        return [c[perm] for c in carry]

    def drift(self):
        A, s, dt = self.A, self.s, self.dt
        for v, a in (("u", "ax"), ("v", "ay"), ("w", "az")):
            s[v] = s[v] + 0.5 * dt * s[a]
        for k, v, L in (("x", "u", A.L[0]), ("y", "v", A.L[1])):
            q = s[k] + dt * s[v]
            q = _round32(q)
            q = torch.where(q < 0, q + L, q)
            s[k] = _round32(torch.where(q >= L, q - L, q))
        z, w = s["z"] + dt * s["w"], s["w"]
        low, high = z < 0, z > A.L[2]
        s["w"] = torch.where(low, w.abs(), torch.where(high, -w.abs(), w))
        s["z"] = _round32(torch.where(low, -z, torch.where(high, 2 * A.L[2] - z, z)))
        if A.surface_flux:
            r = min(max(self.simt / A.ramp, 0.0), 1.0)
            Ts = torch.tensor(A.th0 + A.dts_skin * r * r * (3 - 2 * r), dtype=torch.float64, device=z.device)
            qs = A.qsat(Ts, A.p_ref(torch.zeros_like(Ts)))
            on = self.surf & (s["z"] < A.d[2])
            Pi = (A.p_ref(s["z"]) / A.P0) ** (A.RD / A.CP)
            th = s["th"] + A.c_h * A.v_bg * (Ts - s["th"] * Pi) * dt / A.d[2]
            qv = s["qv"] + A.beta_moist * A.c_e * A.v_bg * (qs - s["qv"]) * dt / A.d[2]
            s["th"] = torch.where(on, torch.clamp(th, 100.0, A.theta_cap), s["th"])
            s["qv"] = torch.where(on, torch.clamp(qv, 0.0, A.qv_cap), s["qv"])

    def pairs(self):
        """Accepted pairs (self excluded) by window offset, each a list of index tensors."""
        A, s = self.A, self.s
        with torch.no_grad():
            x, y, z = (s[k].detach() for k in "xyz")
            c = A.cells(x, y, z)
            i = torch.arange(A.N, device=x.device)
            found = []
            for dz in range(-2, 3):
                for dy in range(-2, 3):
                    for dx in range(-2, 3):
                        jz = c[2] + dz
                        ok = (jz >= 0) & (jz < A.n[2])
                        cell = (jz.clamp(0, A.n[2] - 1) * A.n[1] + (c[1] + dy) % A.n[1]) * A.n[0] + (c[0] + dx) % A.n[0]
                        n = torch.where(ok, self.count[cell], 0)
                        end = torch.cumsum(n, 0)
                        ii = torch.repeat_interleave(i, n)
                        j = self.first[cell[ii]] + torch.arange(ii.numel(), device=x.device) - (end - n)[ii]
                        r2 = ((x[ii] - x[j]) / A.d[0]) ** 2 + ((y[ii] - y[j]) / A.d[1]) ** 2 + ((z[ii] - z[j]) / A.d[2]) ** 2
                        keep = (r2 < 4.0) & (r2 >= 1e-12)
                        found.append((ii[keep], j[keep]))
            return found

    def density(self, found):
        A, s = self.A, self.s
        rho_old = torch.clamp(s["rho"], min=1e-3)
        rref = A.rho_ref(s["z"])
        w0 = torch.full_like(rho_old, A.SIG)
        S2, T = w0 / rho_old, w0 / rho_old * (s["rho"] - rref)
        for i, j in found:
            q = _dist(A, s, i, j)[3].sqrt()
            t = 2.0 - q
            W = torch.where(q < 1.0, A.SIG * (1 - 1.5 * q * q + 0.75 * q ** 3), 0.25 * A.SIG * t ** 3)
            iw = W / rho_old[j]
            S2 = S2.index_add(0, i, iw)
            T = T.index_add(0, i, iw * (s["rho"][j] - rref[i]))
        rho = torch.minimum(torch.maximum(rref + T / S2, 0.5 * rref), 2.0 * rref)
        dd = torch.minimum(torch.maximum(rho - rref, -0.3 * rref), 0.3 * rref)
        self.prs = A.cs ** 2 * dd
        s["rho"] = rho

    def micro(self):
        A, s, dt = self.A, self.s, self.dt
        p = torch.clamp(A.p_ref(s["z"]) + self.prs, min=1.0)
        Pi = (p / A.P0) ** (A.RD / A.CP)
        th, qv, qc, r = s["th"], s["qv"], s["qc"], torch.clamp(s["rho"], min=1e-3)
        T = th * Pi
        wet = (qv > A.qsat(T, p)) | (qc > 0)
        lc = A.LV / A.CP
        dq = torch.zeros_like(T)
        for _ in range(3):
            Tn = T + lc * dq
            es = A.esat(Tn)
            den = p - 0.378 * es
            dqs = 0.622 * p * es * (17.67 * 243.5) / (Tn - 273.15 + 243.5) ** 2 / den ** 2
            dq = dq - (qv - dq - A.qsat(Tn, p)) / (-1.0 - dqs * lc)
            dq = torch.maximum(torch.minimum(dq, qv), -qc)
        dq = torch.where(wet, dq, torch.zeros_like(dq))
        qv, qc, th, T = qv - dq, qc + dq, th + lc * dq / Pi, T + lc * dq
        over = torch.clamp(qc - A.qc_auto, min=0.0) * (1.0 - math.exp(-A.rate_auto * dt))
        qc, dep = qc - over, over
        cx, cy, cz = A.cells(s["x"].detach(), s["y"].detach(), s["z"].detach())
        cid = (cz * A.n[1] + cy) * A.n[0] + cx
        if A.accretion or A.rain_evap:
            qr = torch.clamp(self.rain[cid], min=0.0) / (r * A.v_cell)
            has = qr > 0
            qr1 = torch.where(has, qr, torch.ones_like(qr))
            if A.accretion:
                da = torch.minimum(qc, dt * A.k_accr * qc * qr1 ** 0.875)
                da = torch.where(has & (qc > 0), da, torch.zeros_like(da))
                qc, dep = qc - da, dep + da
            if A.rain_evap:
                qvs = A.qsat(T, p)
                rq = 1e-3 * r * qr1
                C = 1.6 + 124.9 * rq ** 0.2046
                er = (1 - qv / qvs) * C * rq ** 0.525 / (1e-3 * r * (5.4e5 + 2.55e6 / (0.01 * p * qvs)))
                de = torch.minimum(qr, torch.minimum(dt * er, qvs - qv))
                de = torch.where(has & (qv < qvs), de, torch.zeros_like(de))
                qv, th, dep = qv + de, th - lc * de / Pi, dep - de
        self.delta = torch.zeros_like(self.rain).index_add(0, cid, dep * A.pmass)
        s["th"] = torch.clamp(th, 100.0, A.theta_cap)
        s["qv"], s["qc"] = torch.clamp(qv, 0.0, A.qv_cap), torch.clamp(qc, min=0.0)

    def momentum(self, found, source=None):
        A, s, dt = self.A, self.s, self.dt
        rho, prs = torch.clamp(s["rho"], min=1e-3), self.prs
        acc = [torch.zeros_like(rho) for _ in range(3)]
        heat = torch.zeros_like(rho)
        vel = (s["u"], s["v"], s["w"])
        for i, j in found:
            rx, ry, rz, r2 = _dist(A, s, i, j)
            q = r2.sqrt()
            k = A.SIG * torch.where(q < 1.0, -3.0 + 2.25 * q, -0.75 * (2.0 - q) ** 2 / q)
            vr = sum((v[i] - v[j]) * r for v, r in zip(vel, (rx, ry, rz)))
            mu = A.h_av * torch.clamp(vr, max=0.0) / (rx * rx + ry * ry + rz * rz + A.eta2)
            visc = (-A.alpha * A.cs * mu + A.beta * mu * mu) / ((0.5 * (rho[i] + rho[j])) ** 2 * rho[j])
            both = (prs[j] - prs[i]) / (rho[i] * rho[j]) + visc
            for c, (r, d) in enumerate(zip((rx, ry, rz), A.d)):
                gr = k * r / (d * d) * A.mm
                acc[c] = acc[c].index_add(0, i, -both * gr)
                heat = heat.index_add(0, i, visc * gr * vel[c][i])   # -(v . V)
        z = s["z"]
        thv = A.thv_ref(z)
        acc[2] = acc[2] + A.G * ((s["th"] * (1 + 0.608 * s["qv"]) - thv) / thv - s["qc"])
        Pi = (torch.clamp(A.p_ref(z) + prs, min=1.0) / A.P0) ** (A.RD / A.CP)
        dth = torch.clamp(heat / (A.CP * Pi), -A.dthdt_cap, A.dthdt_cap)
        if source is None:
            s["th"] = torch.clamp(s["th"] + dth * dt, 100.0, A.theta_cap)
        else:
            s["th"] = torch.clamp(s["th"] + (dth + source[0]) * dt, 100.0, A.theta_cap)
            s["qv"] = torch.clamp(s["qv"] + source[1] * dt, 0.0, A.qv_cap)
            s["qc"] = torch.clamp(s["qc"] + source[2] * dt, min=0.0)
        s["ax"], s["ay"], s["az"] = acc
        for v, a in zip("uvw", acc):
            s[v] = s[v] + 0.5 * dt * a
        zs = (1 - A.sponge_frac) * A.L[2]
        t = torch.clamp((z - zs) / (A.sponge_frac * A.L[2]), min=0.0)
        s["w"] = s["w"] / (1.0 + A.sponge_sigma * t * t * dt)

    def fall(self):
        A = self.A
        cur = (self.rain + self.delta).view(A.n[2], -1)
        if A.accretion or A.rain_evap:
            cur = torch.clamp(cur, min=0.0)
        f = min(A.v_rain * self.dt / A.d[2], 1.0)
        above = torch.zeros_like(cur)
        above[:-1] = cur[1:]
        self.rain = _round32((cur * (1 - f) + above * f).reshape(-1))

    def control(self, fixed=False):
        A, s = self.A, self.s
        self.simt += self.dt
        self.since_sort = (0.0 if self.sorted_now else self.since_sort) + self.dt
        self.sorted_now = False
        self.step_no += 1
        top = [float(s[v].detach().abs().max()) for v in "uvw"]
        need = 0.9 * A.cfl * min(d / (A.cs + m) for d, m in zip(A.d, top))
        if A.adaptive_dt and not fixed:
            self.dt = min(A.dt_cap, need)
        gap = min(max(min(0.3 * A.d[2] / max(top[2], 0.5), 0.3 * A.d[0] / max(top[0], top[1], 0.5)), self.dt), 15.0)
        self.do_sort = self.step_no % A.sort_every == 0 if A.sort_every > 0 else self.since_sort >= gap

    def step(self, source=None):
        self.lag = self.s["rho"]
        if self.do_sort:
            got = self.order(self.A.permute_acc, () if source is None else source)
            source = source if source is None else got
            self.lag = self.s["rho"]
        self.drift()
        self.rest(source, False)

    def window_step(self):
        """The adjoint's step: the sort moved after the drift, dt fixed."""
        self.drift()
        self.order(self.A.permute_acc)
        self.lag = self.s["rho"]
        self.rest(None, True)

    def rest(self, source, fixed):
        found = self.pairs()
        self.density(found)
        self.micro()
        self.momentum(found, source)
        self.fall()
        for k in self.s:
            self.s[k] = _round32(self.s[k])
        self.control(fixed)

    def tensors(self):
        s, zero = self.s, torch.zeros_like(self.s["x"])
        return {"pos": torch.stack([s["x"], s["y"], s["z"], self.lag], 1),
                "vel": torch.stack([s["u"], s["v"], s["w"], zero], 1),
                "thq": torch.stack([s["th"], s["qv"], s["qc"], zero], 1)}


def _round32(v):
    """float32 rounding with the identity as its derivative."""
    return v + (v.detach().float().double() - v.detach()) if v.requires_grad else v.float().double()


def _dist(A, s, i, j):
    rx, ry, rz = (s[k][i] - s[k][j] for k in "xyz")
    return rx, ry, rz, (rx / A.d[0]) ** 2 + (ry / A.d[1]) ** 2 + (rz / A.d[2]) ** 2


def exact(case, seed):
    kind = case["kind"]
    if kind == "keysort":
        keys = _keys(case, torch.Generator(device="cuda").manual_seed(int(seed)))
        r = torch.sort(keys.to(torch.int64), stable=True)
        return {"keys": r.values.to(torch.int32), "perm": r.indices.to(torch.int32)}
    if kind == "ensemble":
        got = []
        for k, p in enumerate(_ensemble_params(case, seed)):
            s, rain = _state(p, seed * 64 + k, (p.lat_nx, p.lat_ny, p.lat_nz), False)
            e = _Exact(p, s, rain)
            e.order(True)
            for _ in range(case["steps"]):
                e.step()
            got.append(e.tensors())
        return {k: torch.cat([g[k] for g in got]) for k in ("pos", "vel", "thq")}
    p = _params(case)
    s, rain = _state(p, seed, _lat(case), case["developed"])
    e = _Exact(p, s, rain)
    if kind == "exchange":
        e.step()
        return {k: e.s[k] for k in _FIELDS}
    e.order(e.A.permute_acc)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, e)
    for _ in range(case["steps"]):
        if kind == "source":
            t = _tendencies(e.tensors()["thq"].float(), torch.zeros(e.A.N, 4, device="cuda")).double()
            e.step([t[:, k] for k in range(3)])
        else:
            e.step()
    return e.tensors()


def _exact_adjoint(case, seed, e):
    """The window and its gradients by automatic differentiation, the sorts, the pairs and dt held fixed."""
    theta0 = e.s["th"].clone().requires_grad_(True)
    alpha = torch.tensor(e.A.alpha, dtype=torch.float64, device="cuda", requires_grad=True)
    beta = torch.tensor(e.A.beta, dtype=torch.float64, device="cuda", requires_grad=True)
    e.s["th"], e.A.alpha, e.A.beta = theta0, alpha, beta
    for _ in range(case["steps"]):
        e.window_step()
    dqc, dxyz = (v.double() for v in _loss(e.A.N, seed))
    xyz = torch.stack([e.s[k] for k in "xyz"])
    L = (dqc * e.s["qc"]).sum() + (dxyz * xyz.reshape(-1)).sum()
    g = torch.autograd.grad(L, (theta0, alpha, beta))
    with torch.no_grad():
        return {"theta": e.s["th"].detach(), "qv": e.s["qv"].detach(), "qc": e.s["qc"].detach(), "xyz": xyz.detach(),
                "dtheta0": g[0], "dalpha": float(g[1]), "dbeta": float(g[2])}
