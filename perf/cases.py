"""Timed cases of the engine: what its users have it do, through the Python mirror of the C ABI.

A case is a dict of plain values:

  system   what is simulated: "liquid" (Warren MDPD liquid at density 6), "fluid" (plain DPD fluid
           at density 3), "membrane" (stacked 1H+3T bilayers, contracted into ribbons as they are
           after equilibration), "mixed" (a membrane patch with solvent), "reaction" (a membrane with
           10 % single precursor beads that convert to heads), "replicas" (independent liquids of
           uneven size in one handle)
  entry    how it is driven: "step" (K steps per call, state read back into device buffers),
           "observe" (the same with the macro observables every few steps), "host" (the host keeps
           pos / vel / acc and hands them over every step), "passes" (the fine-grained passes of the
           reference's driver loop with their write-back), "walks" (FDPS interaction groups)
  n        particles (replicas: of the largest one)
  steps    steps per pass
  skin     kept-list skin; 0 leaves the engine's default tuning
  lanes, blocks, dens_lanes   launch shape given to set_tuning with a skin

Every handle that steps has taken two steps before the first pass, as in a running program.
"""
import math

import numpy as np
import torch

from implicit_dpd_gb300 import abi, configs
from implicit_dpd_gb300.engine import WALK_DTYPES, Engine, derive_params

HYPHIL, HYPHOB, SOLVENT, NONE = abi.HYPHIL, abi.HYPHOB, abi.SOLVENT, abi.NONE32
AREA_PER_LIPID = 0.333  # over the whole box, as the stacked-bilayer workload has it
RIBBON_AREA = 0.075     # per lipid inside the ribbons of an equilibrated bilayer
LAYER = 4.8             # distance of stacked bilayers
WARM_STEPS = 2
CONVERT_P, CONVERT_SEED = 1e-4, 2024
OBSERVE_EVERY = 10
DT, DT_FLUID = 0.005, 0.01
SIGMA, CF_S, CF_B, VBB, CHI, KAPPA, RHO_CO = 3.0, 50.0, 10.0, 0.1, 30.0, 100.0, 40.0
WARREN_B, WARREN_RD = 25.0, 0.75


def _case(name, system, entry, n, steps, skin=0.0, lanes=16, blocks=1, dens_lanes=32, **more):
    return dict(name=name, system=system, entry=entry, n=n, steps=steps, skin=skin, lanes=lanes,
                blocks=blocks, dens_lanes=dens_lanes, **more)


def listed():
    return [
        # a first small system at the engine's defaults: latency and launches
        _case("liquid_3k", "liquid", "step", 3072, 40),
        # a membrane patch of 2,000 lipids, the size of one simulation of the reference
        _case("membrane_8k", "membrane", "step", 8000, 40, 0.2, 16, 1, 16, layers=1),
        # the plain DPD fluid workload, 20^3 at density 3
        _case("fluid_24k", "fluid", "step", 24000, 40, 0.3, 4, 1, 4),
        # every bead type, bonded and solvent rows in no spatial order, default tuning, odd size
        _case("mixed_31k", "mixed", "step", 31415, 20, layers=1),
        # membrane with precursors and their conversion
        _case("reaction_110k", "reaction", "step", 110000, 20, 0.15, 16, 1, 8, layers=1),
        # the headline membrane: ten stacked bilayers in 64 x 64 x 48
        _case("membrane_984k", "membrane", "step", 984040, 10, 0.15, 16, 1, 8, layers=10),
        # the 10^6-particle MDPD liquid at its tuned shape
        _case("liquid_998k", "liquid", "step", 998250, 20, 0.3, 4, 2, 4),
        # a sweep over parameters: independent liquids of 2k to 60k particles in one handle
        _case("replicas_24", "replicas", "step", 60000, 20, 0.25, 4, 2, 4, replicas=24),
        # a host program that keeps the particles and calls for one step at a time
        _case("host_131k", "membrane", "host", 131072, 4, 0.15, 16, 1, 8, layers=2),
        # the reference's own driver loop, pass by pass, with the write-back of every field
        _case("passes_21k", "mixed", "passes", 20999, 1, layers=1),
        # FDPS's multi-walk hook: both passes over its interaction groups
        _case("walks_13k", "mixed", "walks", 13001, 1, layers=1),
        # a production run that records temperature, pressure and diffusion
        _case("observe_62k", "membrane", "observe", 62000, 20, 0.2, 16, 1, 8, layers=1),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["step"] * 6 + ["observe", "host", "passes", "walks"])
    if entry in ("passes", "walks"):
        n = log(6000, 60000 if entry == "passes" else 20000) | 1
        c = _case("", "mixed", entry, n, 1, layers=1)
    else:
        system = rng.choice(["liquid", "liquid", "membrane", "membrane", "fluid", "mixed", "reaction",
                             "replicas"] if entry == "step" else ["liquid", "membrane"])
        skin = rng.choice([0.0, 0.1, 0.15, 0.2, 0.25, 0.3, 0.35])
        shape = (rng.choice([4, 8, 16, 32]), rng.choice([1, 2]), rng.choice([4, 8, 16, 32]))
        if system == "replicas":
            n, more = log(8000, 60000), {"replicas": rng.randint(2, 32)}
        elif system in ("membrane", "reaction", "mixed"):
            n = log(5000, 400000 if system == "membrane" else 120000)
            more = {"layers": rng.randint(1, 4) if n > 60000 else 1}
        else:
            n, more = log(2500, 600000), {}
        steps = 4 if entry == "host" else rng.choice([10, 20, 40])
        while n * steps > 6000000 and steps > 4:
            steps //= 2
        c = _case("", system, entry, n, steps, skin, *shape, **more)
    del c["name"]
    return c


# ----------------------------------------------------------------- systems
def _maxwell(rng, n):
    v = rng.normal(0.0, 1.0, (n, 3))
    return v - v.mean(axis=0)


def _rows(pos, prop, amp_id, unit, rng):
    n = len(pos)
    return {"pos": np.ascontiguousarray(pos), "vel": _maxwell(rng, n),
            "acc": rng.normal(0.0, 20.0, (n, 3)), "id": np.arange(n, dtype=np.uint32),
            "prop": np.asarray(prop, np.uint32), "amp_id": np.asarray(amp_id, np.uint32),
            "unit": np.asarray(unit, np.uint32)}


def _uniform(n, rho, rng):
    """A liquid: a jittered lattice, which has neither its start's overlaps nor its order."""
    side = (n / rho) ** (1.0 / 3.0)
    k = int(math.ceil(n ** (1.0 / 3.0)))
    cells = np.sort(rng.permutation(k ** 3)[:n])
    pos = np.stack([cells % k, cells // k % k, cells // (k * k)], axis=1).astype(np.float64)
    pos = (pos + 0.5 + rng.normal(0.0, 0.25, pos.shape)) * (side / k)
    pos -= np.floor(pos / side) * side
    none = np.full(n, NONE, np.uint32)
    return np.array([side] * 3), _rows(pos, np.full(n, SOLVENT), none, none, rng)


def _membrane(n_amp, layers, rng, height=None):
    """Bilayers contracted into ribbons along x, with the lateral density, thickness and bond
    lengths that the stacked-bilayer workload has after its equilibration."""
    area = AREA_PER_LIPID * n_amp / (2 * layers)
    side = max(math.sqrt(area), 8.0)
    box = np.array([side, side, height or max(LAYER * layers, 9.6)])
    ribbons = max(1, int(round(side / 12.0)))
    width = RIBBON_AREA * n_amp / (2 * layers) / (side * ribbons)
    m = np.arange(n_amp)
    sign = np.where(m % 2 == 0, 1.0, -1.0)
    mid = ((m // 2) % layers + 0.5) * box[2] / layers
    base = rng.random((n_amp, 3))
    p = np.stack([base[:, 0] * side,
                  (np.floor(rng.random(n_amp) * ribbons) + 0.5) * side / ribbons
                  + (base[:, 1] - 0.5) * width, mid + 1.15 * sign], axis=1)
    p += rng.normal(0.0, 0.25, p.shape)
    pos = np.empty((4 * n_amp, 3))
    for u in range(4):
        pos[u::4] = p
        p = p + rng.normal(0.0, 0.22, p.shape)
        p[:, 2] -= 0.4 * sign
    pos -= np.floor(pos / box) * box
    unit = np.tile(np.arange(4, dtype=np.uint32), n_amp)
    amp = np.repeat(np.arange(n_amp, dtype=np.uint32), 4)
    return box, _rows(pos, np.where(unit == 0, HYPHIL, HYPHOB), amp, unit, rng)


def _add_solvent(box, st, n, rng):
    none = np.full(n, NONE, np.uint32)
    st = {k: np.concatenate([v, e]) for (k, v), e in
          zip(st.items(), _rows(rng.random((n, 3)) * box, np.full(n, SOLVENT), none, none, rng).values())}
    st["id"] = np.arange(len(st["pos"]), dtype=np.uint32)
    return st


def _replica_sizes(case):
    """n and down to 2,000, evenly over the logarithm."""
    return [int(round(case["n"] * (2000.0 / case["n"]) ** (r / max(case["replicas"] - 1, 1))))
            for r in range(case["replicas"])]


def _systems(case, seed):
    """The case's systems: a list of (box, state, molecules, Warren A or None)."""
    rng = np.random.default_rng([seed, 77])
    kind, n = case["system"], case["n"]
    if kind == "replicas":
        out = []
        for m in _replica_sizes(case):
            box, st = _uniform(m, rng.uniform(5.0, 7.0), rng)
            out.append((box, st, 0, float(rng.uniform(-50.0, -30.0))))
        return out
    if kind in ("liquid", "fluid"):
        box, st = _uniform(n, 6.0 if kind == "liquid" else 3.0, rng)
        return [(box, st, 0, -40.0)]
    if kind == "membrane":
        box, st = _membrane(n // 4, case["layers"], rng)
        return [(box, st, n // 4, None)]
    share = 0.5 if kind == "mixed" else 1.0 / 1.1
    n_amp = int(n * share) // 4
    box, st = _membrane(n_amp, case["layers"], rng)
    st = _add_solvent(box, st, n - 4 * n_amp, rng)
    if kind == "mixed":  # rows in no spatial order
        order = rng.permutation(n)
        st = {k: np.ascontiguousarray(v[order]) for k, v in st.items()}
        st["id"] = np.arange(n, dtype=np.uint32)
    return [(box, st, n_amp, None)]


def _form(case):
    if case["system"] in ("liquid", "replicas"):
        return abi.FORM_WARREN
    return abi.FORM_PAIRWISE if case["system"] == "fluid" else abi.FORM_MDPD


def _dt(case):
    return abi.f32(DT_FLUID if case["system"] == "fluid" else DT)


def _params(case, box, warren_a, seed):
    p = derive_params(configs.run_param(box, dt=_dt(case), cf_r=SIGMA, cf_s=CF_S, cf_b=CF_B, vbb=VBB,
                                        chi=CHI, kappa=KAPPA, rho_co=RHO_CO))
    for k in range(3):
        p.box[k] = box[k]
    p.seed, p.time, p.form = (seed * 7919 + 13) & 0x7fffffff, 1, _form(case)
    p.warren_a, p.warren_b, p.warren_rd = warren_a or 0.0, WARREN_B, WARREN_RD
    return p


def prepare(case, seed):
    systems = _systems(case, seed)
    e = Engine(n_replicas=len(systems))
    for r, (box, st, n_amp, a) in enumerate(systems):
        e.set_params(_params(case, box, a, seed + r), r)
        if case["entry"] != "walks":
            e.upload(st, r)
            if n_amp:
                e.build_topology(n_amp, replica=r)
    state = {"case": case, "e": e}
    if case["entry"] == "walks":
        state.update(_walks(*systems[0][:2]))
        return state
    if case["skin"] > 0:
        e.set_tuning(1, case["skin"], lanes=case["lanes"], blocks=case["blocks"],
                     dens_lanes=case["dens_lanes"])
    if case["system"] == "reaction":
        e.set_precursor(SOLVENT, HYPHOB, HYPHIL, abi.precursor_threshold(CONVERT_P), CONVERT_SEED)
    if case["entry"] == "observe":
        e.set_observe(OBSERVE_EVERY, 64)
    sizes = [len(s[1]["pos"]) for s in systems]
    host = case["entry"] == "host"
    state["out"] = [torch.empty((sum(sizes), 3), dtype=torch.float64, pin_memory=host,
                                device="cpu" if host else "cuda") for _ in range(3)]
    state["rows"] = [slice(sum(sizes[:r]), sum(sizes[:r + 1])) for r in range(len(sizes))]
    torch.cuda.synchronize()
    if case["entry"] == "passes":
        return state
    e.step(WARM_STEPS)
    if host:
        e.download_dynamics(*state["out"])
    return state


def run(state):
    case, e = state["case"], state["e"]
    if case["entry"] == "walks":
        return _run_walks(state)
    names = ("pos", "vel", "acc")
    if case["entry"] == "host":
        for _ in range(case["steps"]):
            e.step_host(*state["out"])
        return dict(zip(names, state["out"]))
    got = {}
    if case["entry"] == "passes":
        e.drift()
        e.density()
        e.force()
        got["virial"] = e.bonded()
        e.kick()
        got.update(e.download_aux(density=True, press=True, nei_cm=True))
    else:
        e.step(case["steps"])
    if case["entry"] == "observe":
        seen = e.observations(64)
        for k in ("kin_temp", "pressure", "diffusion", "pair_virial", "bonded_virial"):
            got[k] = np.array([o[k] for o in seen])
    if case["system"] == "reaction":
        got["converted"] = e.precursor_count()
    for r, rows in enumerate(state["rows"]):
        e.download_dynamics(*(t[rows] for t in state["out"]), replica=r)
    got.update(zip(names, state["out"]))
    return got


# ------------------------------------------------------------------- walks
def _walks(box, st):
    """Interaction groups as FDPS's short-range tree makes them: the i particles of one cell of side
    >= 1.2, and the particles of the 27 cells around it, image-shifted. All walks lie one after the
    other in one record array per kind and side; a walk is a slice of it."""
    nc = np.floor(box / 1.2).astype(int)
    c = np.minimum((st["pos"] / box * nc).astype(int), nc - 1)
    cell = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    order = np.argsort(cell, kind="stable")
    start = np.searchsorted(cell[order], np.arange(nc.prod() + 1))
    off = np.array([(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)])
    ii, jj, shift = [], [], []
    for k in np.unique(cell):
        q = np.array([k % nc[0], k // nc[0] % nc[1], k // (nc[0] * nc[1])]) + off
        s = np.floor_divide(q, nc)
        q = q - s * nc
        at = (q[:, 2] * nc[1] + q[:, 1]) * nc[0] + q[:, 0]
        ii.append(order[start[k]:start[k + 1]])
        members = [order[start[a]:start[a + 1]] for a in at]
        jj.append(np.concatenate(members))
        shift.append(np.repeat(s * box, [len(m) for m in members], axis=0))
    ni, nj = np.cumsum([0] + [len(x) for x in ii]), np.cumsum([0] + [len(x) for x in jj])
    ii, jj, shift = np.concatenate(ii), np.concatenate(jj), np.concatenate(shift)
    rec = {}
    for kind in (0, 1):
        ti, tj, _ = WALK_DTYPES[kind]
        i, j = np.zeros(len(ii), ti), np.zeros(len(jj), tj)
        i["prop"], i["pos"] = st["prop"][ii], st["pos"][ii]
        j["prop"], j["pos"] = st["prop"][jj], st["pos"][jj] + shift
        if kind:
            i["id"], i["vel"], j["id"], j["vel"] = st["id"][ii], st["vel"][ii], st["id"][jj], st["vel"][jj]
            j["amp_id"], j["unit"] = st["amp_id"][jj], st["unit"][jj]
        rec[kind] = (i, j)
    return {"rec": rec, "ii": ii, "jj": jj,
            "walk": {k: ([rec[k][0][a:b] for a, b in zip(ni[:-1], ni[1:])],
                         [rec[k][1][a:b] for a, b in zip(nj[:-1], nj[1:])]) for k in (0, 1)}}


def _run_walks(state):
    e, (i, j) = state["e"], state["rec"][1]
    e.dispatch_walks(0, *state["walk"][0])
    den = np.concatenate(e.retrieve_walks(0))
    dens = np.empty((len(i), 3))
    dens[state["ii"]] = den["dens"]  # the write-back to the particles, and FDPS's copy into the groups
    i["dens"], j["dens"] = dens[state["ii"]], dens[state["jj"]]
    e.dispatch_walks(1, *state["walk"][1])
    frc = np.concatenate(e.retrieve_walks(1))
    got = {"dens": dens}
    for name, field in (("nei_pos_sum", den["nei_pos_sum"]), ("nei_cnt", den["nei_cnt"].astype(np.int64)),
                        ("acc", frc["acc"]), ("press", frc["press"])):
        got[name] = np.empty_like(field)
        got[name][state["ii"]] = field
    return got


# -------------------------------------------------------------------- work
def work(case):
    """State read and written once per pass (144 B of pos, vel, acc and 16 B of ids a particle), and
    the arithmetic of every pair within the cutoff taken once (density ~13, force ~134 operations)."""
    n = case["n"]
    if case["system"] == "replicas":
        n = sum(_replica_sizes(case))
    pairs = {"liquid": 12.5, "replicas": 12.5, "fluid": 6.3, "membrane": 65.0, "reaction": 60.0,
             "mixed": 30.0}[case["system"]]
    return {"bytes": 160.0 * n, "flops": float(case["steps"]) * n * pairs * 147.0}


# ------------------------------------------------- the same in 64 bits
M32 = 0xffffffff


def _i32(x, s):
    return (((x ^ 0x80000000) - 0x80000000) >> s) & M32  # arithmetic shift of a 32-bit word


class _Saru:
    """Saru(a, b, c) (saruprng.hpp:239-255, 322-333) on int64 tensors that hold 32-bit words."""

    def __init__(self, a, b, c):
        c = c ^ ((a << 7) & M32) ^ (b >> 6)
        b = (b + ((a >> 4) ^ (c >> 15))) & M32
        a = a ^ (((b << 9) + (c << 8)) & M32)
        c = c ^ (0xA5366B4D * ((b >> 11) ^ ((a << 1) & M32)) & M32)
        b = (b + 0x72BE1579 * (((a << 4) & M32) ^ (c >> 16))) & M32
        a = a ^ (0x3F38A6ED * ((c >> 5) ^ _i32(b, 22)) & M32)
        b = (b + a * c) & M32
        a = (a + (c ^ (b >> 2))) & M32
        b = b ^ _i32(b, 17)
        lcg = 0x79dedea3 * (a ^ _i32(a, 14)) & M32
        weyl = ((lcg + b) & M32) ^ _i32(lcg, 8)
        self.lcg = (lcg + weyl * (weyl ^ 0xdddf97f5)) & M32
        self.weyl = (0xABCB96F7 + (weyl >> 1)) & M32

    def u32(self):
        self.lcg = (0x4beb5d59 * self.lcg + 0x2600e1f7) & M32
        self.weyl = (self.weyl + 0x8009d14b + (_i32(self.weyl, 31) & 0xda879add)) & M32
        v = ((self.lcg ^ (self.lcg >> 26)) + self.weyl) & M32
        return ((v ^ (v >> 20)) * 0x6957f5a7) & M32

    def normal(self):
        u, v = (((self.u32() >> 1).double() + 0.5) / 2147483648.0 for _ in range(2))
        return torch.sqrt(-2.0 * torch.log(u)) * torch.cos(2.0 * math.pi * v)


def _tables():
    """CalcInterCoef (parameter.hpp:138-186) of the constants above."""
    f = lambda x: float(np.float32(x))  # noqa: E731
    reo, arc, unit = 1.4, 0.9, 4
    c = np.empty((3, 3))
    c[1, 1] = -2.0 * (f(KAPPA) + 3.0) / f(RHO_CO)
    c[0, 0] = c[2, 2] = c[0, 2] = c[2, 0] = f(VBB)
    c[0, 1] = c[1, 0] = c[2, 1] = c[1, 2] = f(CHI) / f(RHO_CO) + 0.5 * (c[0, 0] + c[1, 1])
    m = np.full((3, 3, 3), 1.5 * (f(KAPPA) + 2.0) / f(RHO_CO) ** 2)
    m[0, 0, 0] = m[2, 2, 2] = 0.0
    mol = reo ** 3 / unit ** 2
    c *= mol * -45.0 / ((arc ** 5 * (2.0 * arc - 3.0) + (3.0 * arc - 2.0)) * math.pi)
    m *= mol * (2.0 / 3.0) * (15.0 / math.pi) * (reo ** 3 * 15.0 / (2.0 * math.pi * unit))
    return c, m


class _System:
    """The step of the engine in 64 bits, with plain torch."""

    def __init__(self, case, box, st, n_amp, warren_a, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda k, d=torch.float64: torch.as_tensor(st[k].astype(np.int64) if d == torch.int64  # noqa: E731
                                                       else st[k], dtype=d, device=dev)
        self.case, self.dev, self.n = case, dev, len(st["pos"])
        self.x, self.v, self.a = t("pos"), t("vel"), t("acc")
        self.id, self.prop = t("id", torch.int64), t("prop", torch.int64)
        self.box = torch.as_tensor(box, dtype=torch.float64, device=dev)
        self.moved = torch.zeros_like(self.x)
        self.seed, self.time, self.dt, self.wa = (seed * 7919 + 13) & 0x7fffffff, 1, _dt(case), warren_a
        self.c, self.m = (torch.as_tensor(v, device=dev) for v in _tables())
        self.amp = None
        if n_amp:
            mol = np.empty((n_amp, 4), np.int64)
            own = st["amp_id"] != NONE
            mol[st["amp_id"][own], st["unit"][own]] = np.nonzero(own)[0]
            self.amp = torch.as_tensor(mol, device=dev)

    def drift(self):
        self.v = self.v + 0.5 * self.dt * self.a
        d = self.dt * self.v
        self.moved = self.moved + d
        x = self.x + d
        self.x = x - torch.floor(x / self.box) * self.box

    def pairs(self, rc):
        """Pairs (i, j) closer than rc, once each, and x_i - x_j at the nearest image."""
        nc = torch.floor(self.box / rc).long()
        c = torch.minimum((self.x / self.box * nc).long(), nc - 1)
        cell = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
        key, order = torch.sort(cell)
        start = torch.searchsorted(key, torch.arange(int(nc.prod()) + 1, device=self.dev))
        half = [(0, 0, 0)] + [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)
                              if (z, y, x) > (0, 0, 0)]
        out = []
        for lo in range(0, self.n, 1 << 17):
            hi = min(lo + (1 << 17), self.n)
            rows = order[lo:hi]
            for o in half:
                q = (c[rows] + torch.tensor(o, device=self.dev)) % nc
                other = (q[:, 2] * nc[1] + q[:, 1]) * nc[0] + q[:, 0]
                first, end = start[other], start[other + 1]
                if o == (0, 0, 0):
                    first = torch.arange(lo + 1, hi + 1, device=self.dev)
                count = (end - first).clamp(min=0)
                which = torch.repeat_interleave(torch.arange(hi - lo, device=self.dev), count)
                if which.numel() == 0:
                    continue
                within = torch.arange(which.numel(), device=self.dev) - (torch.cumsum(count, 0) - count)[which]
                i, j = rows[which], order[first[which] + within]
                d = self.x[i] - self.x[j]
                d = d - torch.round(d / self.box) * self.box
                ok = (d * d).sum(1) < rc * rc
                out.append((i[ok], j[ok], d[ok]))
        return tuple(torch.cat(v) for v in zip(*out))

    def density(self, i, j, r):
        if self.case["system"] in ("liquid", "replicas"):
            u = (1.0 - r / WARREN_RD).clamp(min=0.0)
            w = 15.0 / (2.0 * math.pi * WARREN_RD ** 3) * u * u
        else:
            w = (1.0 - r) ** 2
        d = torch.zeros(3 * self.n, dtype=torch.float64, device=self.dev)
        d.index_add_(0, 3 * i + self.prop[j], w)
        d.index_add_(0, 3 * j + self.prop[i], w)
        return d.view(-1, 3)

    def pair_force(self):
        """Acceleration and virial (per particle) of the pair force; the density and the pairs."""
        i, j, e = self.pairs(1.0)
        r = torch.sqrt((e * e).sum(1))
        self.dens = rho = self.density(i, j, r)
        w = 1.0 - r
        if self.case["system"] == "fluid":
            cons = 25.0 * w
        elif self.case["system"] in ("liquid", "replicas"):
            wb = (1.0 - r / WARREN_RD).clamp(min=0.0)
            cons = self.wa * w + WARREN_B * (rho[i] + rho[j]).sum(1) * wb
        else:
            pi, pj = self.prop[i], self.prop[j]
            cons = (self.c[pi, pj] * (r - 0.9) * (r >= 0.9) + (self.m[pi, pj] * (rho[i] + rho[j])).sum(1)) * w
        a, b = self.id[i], self.id[j]
        z = _Saru(torch.minimum(a, b), torch.maximum(a, b),
                  torch.full_like(a, (self.seed + self.time) & M32)).normal()
        cf_r, cf_g = SIGMA / math.sqrt(self.dt), 0.5 * SIGMA * SIGMA
        f = (cons + cf_r * torch.sqrt(w) * z - cf_g * w * (e * (self.v[i] - self.v[j])).sum(1) / r) / r
        g = f[:, None] * e
        acc, vir = torch.zeros_like(self.x), torch.zeros_like(self.x)
        acc.index_add_(0, i, g).index_add_(0, j, -g)
        vir.index_add_(0, i, g * e).index_add_(0, j, g * e)
        return acc, vir, (i, j)

    def bonded(self, acc):
        """Adds bond and bend forces (bdf_calculator.hpp:95-220); returns their virial."""
        vir = torch.zeros(3, dtype=torch.float64, device=self.dev)
        if self.amp is None:
            return vir
        prev = None
        for u in range(1, 4):
            lo, hi = self.amp[:, u - 1], self.amp[:, u]
            d = self.x[hi] - self.x[lo]
            d = d - torch.round(d / self.box) * self.box
            inv = 1.0 / torch.sqrt((d * d).sum(1, keepdim=True))
            f = CF_S * (inv - 2.0) * d
            acc.index_add_(0, hi, f).index_add_(0, lo, -f)
            vir += 2.0 * (d * f).sum(0)
            if prev is not None:
                b, ib = prev
                dot, cf = (b * d).sum(1, keepdim=True), CF_B * ib * inv
                t0, t1 = cf * (d - dot * ib * ib * b), cf * (b - dot * inv * inv * d)
                acc.index_add_(0, self.amp[:, u - 2], -t0).index_add_(0, lo, t0 - t1).index_add_(0, hi, t1)
                vir += 2.0 * (b * t0 + d * t1).sum(0)
            prev = (d, inv)
        return vir

    def step(self):
        self.drift()
        self.a, self.press, (i, j) = self.pair_force()
        converted = 0
        if self.case["system"] == "reaction":
            near = torch.zeros(self.n, dtype=torch.bool, device=self.dev)
            near[i[self.prop[j] == HYPHOB]] = True
            near[j[self.prop[i] == HYPHOB]] = True
            turn = near & (self.prop == SOLVENT)
            t = torch.full_like(self.id, self.time)
            turn &= _Saru(self.id, t, torch.full_like(t, CONVERT_SEED)).u32() < abi.precursor_threshold(CONVERT_P)
            converted = int(turn.sum())
            self.next_prop = torch.where(turn, torch.full_like(self.prop, HYPHIL), self.prop)
        self.bonded_virial = self.bonded(self.a)
        self.v = self.v + 0.5 * self.dt * self.a
        if self.time % 100 == 0:
            self.v = self.v - self.v.mean(0)
        if self.case["system"] == "reaction":
            self.prop = self.next_prop
        return converted

    def observation(self):
        n, k = self.n, 0 if self.amp is None else len(self.amp)
        t = (self.v * self.v).mean(0)
        pair = self.press.sum(0)
        msd = (self.moved * self.moved).sum(1)
        lipid = (self.moved[:4 * k].view(-1, 4, 3).mean(1) ** 2).sum(1).mean() if k else torch.zeros(())
        sol = n - 4 * k
        return {"kin_temp": torch.cat([t, t.mean()[None]]), "pair_virial": pair,
                "pressure": (0.5 * pair + t * n + 0.5 * self.bonded_virial) / self.box.prod(),
                "diffusion": torch.stack([msd.mean(), lipid.to(msd), msd[k:].sum() / sol if sol
                                          else torch.zeros((), device=self.dev).to(msd)]),
                "bonded_virial": self.bonded_virial}

    def neighbour_sums(self):
        """Position sums and counts of the neighbours (nbdf_calculator.hpp:22-55): hydrophilic within
        1 and the particle itself, hydrophobic within 1.2."""
        i, j, d = self.pairs(1.2)
        r2 = (d * d).sum(1)
        total = torch.zeros((self.n, 2, 3), dtype=torch.float64, device=self.dev)
        count = torch.zeros((self.n, 2), dtype=torch.int64, device=self.dev)
        total[:, 0] = self.x
        count[:, 0] = 1
        for a, b, s in ((i, j, -1.0), (j, i, 1.0)):
            for k, prop, rc in ((0, HYPHIL, 1.0), (1, HYPHOB, 1.2)):
                ok = (self.prop[b] == prop) & (r2 < rc * rc)
                total[:, k] = total[:, k].index_add(0, a[ok], self.x[a[ok]] + s * d[ok])
                count[:, k] = count[:, k].index_add(0, a[ok], torch.ones_like(a[ok]))
        return total, count


def exact(case, seed):
    systems = [_System(case, box, st, n_amp, a, seed + r)
               for r, (box, st, n_amp, a) in enumerate(_systems(case, seed))]
    s = systems[0]
    out = {}
    if case["entry"] in ("passes", "walks"):
        if case["entry"] == "passes":
            s.drift()
        total, count = s.neighbour_sums()
        acc, press, _ = s.pair_force()
        out.update(dens=s.dens, press=press)
        if case["entry"] == "walks":
            out.update(nei_pos_sum=total, nei_cnt=count, acc=acc)
        else:
            out.update(nei_cm=(total / count[:, :, None]).view(-1, 6), virial=s.bonded(acc)[None, :])
            out.update(pos=s.x, vel=s.v + 0.5 * s.dt * acc, acc=acc)
        return {k: v.cpu() for k, v in out.items()}
    seen, converted = [], 0
    for k in range(WARM_STEPS + case["steps"]):
        for one in systems:
            converted += one.step()
            if case["entry"] == "observe" and one.time % OBSERVE_EVERY == 0:
                seen.append(one.observation())
            one.time += 1
    if seen:
        out.update({k: torch.stack([o[k].cpu() for o in seen]) for k in seen[0]})
    if case["system"] == "reaction":
        out["converted"] = converted
    for name, field in (("pos", "x"), ("vel", "v"), ("acc", "a")):
        out[name] = torch.cat([getattr(one, field) for one in systems]).cpu()
    return out
