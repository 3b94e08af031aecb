"""Performance cases of the IS-SPA engine: what a user of the framework has it do.

Every case goes through the public entry points (`isspa_gb300.Engine`,
`isspa_force_noalloc`), on systems of this repository's own kinds: chains of
atoms in a periodic box at the density of the benchmark's systems, IS-SPA
tables on the fixtures' radial grid, and the ADI2 dimer read from its Amber
files.  Kinds:

  host_step   one MD step with page-locked host buffers (positions and
              velocities in; positions, velocities and forces out): a driver
              that owns the state, the engine behind it
  trajectory  a stretch of MD steps, then the coordinates for the trajectory
              file: the inner loop of the drop-in executable between outputs
  forces      the per-term force calls in the reference's order, then the
              force: an output step, or an integrator of the caller's own
  noalloc     the IS-SPA force on the caller's device arrays and stream
  adjoint     the mean COM-axis force of umbrella windows and its gradient in
              the force-field tables, for one frame

`exact` restates the model in 64 bits with torch alone: values in double,
the branch decisions (minimum image, inside-rmax, table bins, rejection of
Monte Carlo points) in the float arithmetic that defines them.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "isspa-force-cuda_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "isspa-force-cuda_gb300"))

import isspa_gb300 as ig  # noqa: E402
from isspa_gb300 import abi, synth  # noqa: E402

# atoms per cubic Angstrom of the benchmark's 1100-atom system in its 60 A box
DENSITY = 1100 / 60.0 ** 3


def _box(atoms):
    return max(40.0, (atoms / DENSITY) ** (1.0 / 3.0))


def _case(kind, chains, length, box, n_mc, steps=1, windows=1, us=False, solvent=True, cutoff=0.0, tuned=False, adi2=False):
    return dict(kind=kind, chains=chains, length=length, box=float(box), n_mc=n_mc, steps=steps, windows=windows, us=us,
                solvent=solvent, cutoff=float(cutoff), tuned=tuned, adi2=adi2)


def listed():
    return [
        # the smallest system of the benchmark, one step per call
        dict(_case("host_step", 2, 22, 40.0, 20, tuned=True), name="host step 44"),
        # the reference's published run: the ADI2 dimer under its umbrella restraint
        dict(_case("trajectory", 2, 22, 200.0, 100, steps=32, us=True, tuned=True, adi2=True), name="trajectory ADI2 44"),
        # an output step of a mid-size window, engine as created
        dict(_case("forces", 12, 22, 40.0, 20), name="forces 264"),
        # odd and ragged: 741 atoms, 37 points per atom, a box that is no round number
        dict(_case("trajectory", 57, 13, 53.7, 37, steps=8), name="trajectory 741 ragged"),
        # the benchmark's flagship, end to end and back to back
        dict(_case("host_step", 50, 22, 60.0, 50, tuned=True), name="host step 1100"),
        dict(_case("trajectory", 50, 22, 60.0, 50, steps=8, tuned=True), name="trajectory 1100"),
        # umbrella windows of 44 to 1100 atoms in one engine
        dict(_case("trajectory", 50, 22, 60.0, 50, steps=2, windows=12, us=True, tuned=True), name="windows 12"),
        # a large solvated system, one step per call, engine as created
        dict(_case("host_step", 400, 22, 120.0, 100), name="host step 8800"),
        # the IS-SPA force inside a caller's own stream and memory pool
        dict(_case("noalloc", 50, 22, 60.0, 50), name="noalloc 1100"),
        # the benchmark's differentiation workload: 16 windows of 550 atoms
        dict(_case("adjoint", 25, 22, 50.0, 50, windows=16, us=True), name="adjoint 16x550"),
        # without the solvent pass (energy-conservation runs): every pair, and the cutoff mode
        dict(_case("trajectory", 200, 22, 95.0, 50, steps=16, solvent=False), name="vacuum 4400 all pairs"),
        dict(_case("trajectory", 400, 22, 120.0, 50, steps=16, solvent=False, cutoff=12.0), name="vacuum 8800 cutoff"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host_step", "trajectory", "trajectory", "forces", "noalloc", "adjoint", "windows", "vacuum"])
    length = rng.randint(9, 25)
    n_mc = _log(rng, 10, 100)
    slack = rng.uniform(1.0, 1.25)
    tuned = rng.random() < 0.5
    if kind == "adjoint":
        atoms = _log(rng, 60, 600)
        chains = max(2, atoms // length)
        return _case("adjoint", chains, length, round(_box(chains * length) * slack, 2), min(n_mc, 50),
                     windows=rng.randint(1, 16), us=True)
    if kind == "windows":
        chains = max(2, _log(rng, 60, 1100) // length)
        return _case("trajectory", chains, length, round(_box(chains * length) * slack, 2), min(n_mc, 50), steps=2,
                     windows=rng.randint(2, 12), us=True, tuned=tuned)
    if kind == "vacuum":
        chains = max(2, _log(rng, 500, 8800) // length)
        cutoff = rng.choice([0.0, rng.uniform(9.0, 14.0)])
        return _case("trajectory", chains, length, round(_box(chains * length) * slack, 2), n_mc, steps=16, solvent=False,
                     cutoff=round(cutoff, 2))
    atoms = _log(rng, 44, 2200 if kind == "noalloc" else 4400)
    chains = max(2, atoms // length)
    if kind == "noalloc":
        n_mc = min(n_mc, 150000 // (chains * length))  # what its fixed buffer takes
    n_mc = max(10, n_mc)
    steps = 1 if kind != "trajectory" else 32 if atoms < 300 else 8
    return _case(kind, chains, length, round(_box(chains * length) * slack, 2), n_mc, steps=steps, tuned=tuned and kind != "noalloc")


# ------------------------------------------------------------------- systems
def _seeded_adi2(n_mc, seed):
    """The ADI2 dimer of the repository's input files: its coordinates with
    thermal noise, velocities and run seed from `seed`, restrained as in the
    reference's published umbrella run (k 20, x0 10 A)."""
    s = ig.System.from_config(os.path.join(ROOT, "tests", "golden", "adi2_config.txt"))
    rng = np.random.default_rng(seed)
    n = s.n_atoms
    s.n_mc = n_mc
    s.seed = int(seed) + 1
    s.pos[:, :3] += rng.normal(0.0, 0.01, (n, 3)).astype(np.float32)
    s.vel[:, :3] = rng.normal(size=(n, 3)) * np.sqrt(s.kT / s.vel[:, 3])[:, None]
    s.us_on = 1
    s.bias_list = np.array([(a, a // 22) for a in range(n)], np.int32)
    s.us_k, s.us_x0 = 20.0, 10.0
    return s


def _systems(case, seed):
    """The windows of a case: window w has its own chains, charges, types and velocities."""
    if case["adi2"]:
        return [_seeded_adi2(case["n_mc"], seed)]
    ff = synth.forcefield(n_mc=case["n_mc"])
    out = []
    W = case["windows"]
    for w in range(W):
        chains = case["chains"]
        if case["kind"] != "adjoint" and W > 1:  # windows from two chains up to the case's size
            chains = 2 + round((chains - 2) * w / (W - 1))
        us = (10.0, 4.0 + 12.0 * w / max(1, W - 1)) if case["us"] else None
        out.append(synth.make_system(chains, case["length"], case["box"], case["n_mc"], 1000 * int(seed) + w, ff=ff, us=us,
                                     run_seed=int(seed) + 12345))
    return out


def _start_step(seed):
    return 100 + int(seed) % 1000  # the MC points' Philox step key of the first pass


# ----------------------------------------------------------- prepare and run
class _NoAlloc:
    """Device arrays of one system, as a caller of isspa_force_noalloc holds them."""

    def __init__(self, s, step):
        def dev(a, dtype):
            return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")

        self.keep = [dev(s.pos, torch.float32), dev(s.isspa_type, torch.int32), dev(s.rmax, torch.float32)]
        self.keep += [dev(t, torch.float32) for t in (s.g_table, s.e_table, s.f_table)]
        self.out = torch.empty((s.n_atoms, 4), dtype=torch.float32, device="cuda")
        a = abi.NoallocInputs()
        a.n_atoms, a.n_mc, a.n_isspa_types = s.n_atoms, s.n_mc, len(s.rmax)
        a.pos, a.isspa_type, a.rmax, a.g_table, a.e_table, a.f_table = (t.data_ptr() for t in self.keep)
        a.n_g, a.n_e, a.n_f = s.g_table.shape[1], s.e_table.shape[1], s.f_table.shape[1]
        a.g_r0, a.g_dr, a.e_r0, a.e_dr, a.f_r0, a.f_dr = s.g_r0, s.g_dr, s.e_r0, s.e_dr, s.f_r0, s.f_dr
        a.box, a.seed, a.step = s.box, s.seed, step
        self.inputs = a

    def force(self):
        stream = torch.cuda.current_stream().cuda_stream
        abi.check(abi.lib().isspa_force_noalloc(ctypes.byref(self.inputs), ctypes.c_void_p(self.out.data_ptr()),
                                                ctypes.c_void_p(stream)), "isspa_force_noalloc")
        return self.out


def prepare(case, seed):
    systems = _systems(case, seed)
    kind = case["kind"]
    step = _start_step(seed)
    if kind == "noalloc":
        return {"kind": kind, "call": _NoAlloc(systems[0], step)}
    eng = ig.Engine(systems, isspa_terms=7 if case["solvent"] else abi.TERMS_NONE, nonbond_cutoff=case["cutoff"])
    if case["tuned"]:  # as a production run does once
        eng.autotune()
    eng.set_step(step)
    st = {"kind": kind, "eng": eng, "steps": case["steps"], "next": step}
    if kind == "host_step":
        st["bufs"] = [ig.host_array((eng.n_atoms, 4)) for _ in range(5)]
        st["bufs"][0][:] = np.concatenate([s.pos for s in systems])
        st["bufs"][1][:] = np.concatenate([s.vel for s in systems])
    return st


def run(st):
    kind = st["kind"]
    if kind == "noalloc":
        return [st["call"].force()]
    eng = st["eng"]
    if kind == "host_step":
        eng.step_host(*st["bufs"])
        return [st["bufs"][2], st["bufs"][3], st["bufs"][4]]
    if kind == "trajectory":
        eng.step(st["steps"])
        return [eng.positions()]
    if kind == "forces":
        return [eng.compute_forces()]
    # a fitting step of the float tables: value and gradient in the tables' own type
    grads = eng.adjoint_mean_force([st["next"]])
    st["next"] += 1
    return [g.astype(np.float32) for g in grads]


def _sizes(case):
    if case["adi2"]:
        return [44]
    W = case["windows"]
    if case["kind"] == "adjoint" or W == 1:
        return [case["chains"] * case["length"]] * W
    return [(2 + round((case["chains"] - 2) * w / (W - 1))) * case["length"] for w in range(W)]


def work(case):
    """One pass, with the benchmark's counting (FMA = 2): 38 flop per point-atom
    pair of the field, 88 per atom-point pair of the force, 30 per point, 32 per
    ordered atom pair.  Bytes: the state, forces and tables in and out."""
    flops, nbytes = 0.0, 8.0 * 3 * 5 * 120
    for n in _sizes(case):
        f = 0.0
        points = n * case["n_mc"]
        if case["solvent"]:
            f += n * points * (38 + 88) + 30 * points
        if case["kind"] != "noalloc":
            partners = n - 1
            if case["cutoff"] > 0:
                partners = min(partners, n / case["box"] ** 3 * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3)
            f += 32.0 * n * partners + 300.0 * n
        if case["kind"] == "adjoint":  # the points' adjoint on the restrained atoms, and the density's
            f += points * (2 * case["length"] * 120 + n * 15)
        flops += f * case["steps"]
        nbytes += n * 16.0 * (2 if case["kind"] in ("noalloc", "forces", "adjoint") else 5)
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------- exact
D = torch.float64
EP, RHO, P0, Q0, O0, PI = (float(np.float32(v)) for v in (2.3473, 0.0075, 4.173705894203977, 1.6899960102882601,
                                                          9.3658298730779350, 3.1415926535))


def _e0():
    f = np.float32
    return float(f(3) / (f(4) * f(PI) * f(RHO) * f(P0)) * (f(1) - f(1) / f(EP)))


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=D):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev()).to(dtype)


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al. 2011) on arrays of counters."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.broadcast_to(np.asarray(v, np.uint64), np.broadcast_shapes(*(np.shape(q) for q in (c0, c1, c2, c3)))).copy()
         for v in (c0, c1, c2, c3)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0 = c[0] * np.uint64(0xD2511F53)
        p1 = c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0 = (k0 + 0x9E3779B9) & 0xFFFFFFFF
        k1 = (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _u01(x):
    return (x >> np.uint64(8)).astype(np.float64) * 2.0 ** -24


def _u01_open0(x):
    return ((x >> np.uint64(8)).astype(np.float64) + 1.0) * 2.0 ** -24


def _f32(x):
    return x.to(torch.float32).to(D)


def _d2_float(r):
    """Squared length as the engine decides on it: three float roundings (fused multiply-adds)."""
    q = _f32(r[0] * r[0])
    q = _f32(r[1] * r[1] + q)
    return _f32(r[2] * r[2] + q)


def _image(a, b, L):
    """Components of a - b at the nearest image (one box at most): the float
    ones that decide, and the double ones that count."""
    dec, val = [], []
    h = 0.5 * L
    for k in range(3):
        d = a[..., k] - b[..., k]
        f = _f32(_f32(a[..., k]) - _f32(b[..., k]))
        shift = torch.where(f.abs() > h, torch.copysign(torch.full_like(f, L), f), torch.zeros_like(f))
        dec.append(_f32(f - shift))
        val.append(d - shift)
    return dec, val


def _points(s, x, step, window):
    """Monte Carlo points [N n_mc, 3]: uniform in the ball r^2 < 0.99 of each owner, by rejection."""
    n_points = s.n_atoms * s.n_mc
    m = np.zeros((n_points, 3))
    m[:, 0] = 0.5
    todo = np.arange(n_points)
    for attempt in range(64):
        o = _philox(todo.astype(np.uint64), attempt, step, window << 8, s.seed)
        u = np.stack([2.0 * _u01(o[k]) - 1.0 for k in range(3)], 1)
        f32 = lambda v: v.astype(np.float32).astype(np.float64)  # noqa: E731
        d2 = f32(u[:, 2] ** 2 + f32(u[:, 1] ** 2 + f32(u[:, 0] ** 2)))
        ok = d2 < float(np.float32(0.99))
        m[todo[ok]] = u[ok]
        todo = todo[~ok]
        if not len(todo):
            break
    owner = np.repeat(np.arange(s.n_atoms), s.n_mc)
    rm = s.rmax.astype(np.float64)[s.isspa_type[owner]]
    xo = x[torch.as_tensor(owner, device=x.device)]
    return _f32(_t(m) * _t(rm)[:, None] + xo), torch.as_tensor(owner, device=x.device)


def _langevin(x):
    small = torch.clamp(x, max=5.0)
    r = torch.zeros_like(x)
    r2 = r3 = r
    for k in range(28, 0, -1):
        r = small / ((2 * k + 1) + small * r)
        r3 = r if k == 3 else r3
        r2 = r if k == 2 else r2
    big = torch.clamp(x, min=5.0)
    c, i = 1.0 / torch.tanh(big), 1.0 / big
    lo = x < 5.0
    return (torch.where(lo, r, c - i), torch.where(lo, r * r2, 1 + 3 * i * i - 3 * c * i),
            torch.where(lo, r * r2 * r3, (1 + 15 * i * i) * c - 6 * i - 15 * i ** 3))


class _Tables:
    def __init__(self, s):
        pad = max(s.g_table.shape[1], s.e_table.shape[1], s.f_table.shape[1]) + 1
        flat = lambda t: torch.cat([_t(t).reshape(-1), torch.zeros(pad, dtype=D, device=_dev())])  # noqa: E731
        self.g, self.e, self.f = flat(s.g_table), flat(s.e_table), flat(s.f_table)
        lj = _t(s.lj_ab)
        self.A, self.B = lj[:, 0].clone(), lj[:, 1].clone()

    def leaves(self):
        return [t.requires_grad_() for t in (self.f, self.g, self.A, self.B)]


def _bin(v):
    return torch.trunc(v).to(torch.int64)


def _inv(dr):
    return float(np.float32(1.0) / np.float32(dr))


def _isspa_chunk(s, T, x, q, points, owner, atoms):
    """IS-SPA force on `atoms` from `points` (their field from every atom)."""
    L = float(np.float32(s.box))
    rmax = _t(s.rmax)
    types = torch.as_tensor(s.isspa_type.astype(np.int64), device=x.device)
    dec, r = _image(points[:, None, :], x[None, :, :], L)
    d2f = _d2_float(dec)
    d2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
    d = torch.sqrt(d2)
    rm2 = _f32(rmax[types[owner]] ** 2)[:, None]
    inside = d2f <= rm2
    n = inside.sum(1).to(D)
    n_g, n_e, n_f = s.g_table.shape[1], s.e_table.shape[1], s.f_table.shape[1]
    dist = _f32(torch.sqrt(d2f))
    b = _bin(_f32(_f32(dist - float(np.float32(s.g_r0))) * _inv(s.g_dr)))
    look = inside & (b >= 0) & (b < n_g - 1)
    bc = torch.clamp(b, 0, n_g - 2)
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    gi, ei = types[None, :] * n_g + bc, types[None, :] * n_e + bc
    fr = (d - (f32(s.g_r0) + bc * f32(s.g_dr))) / f32(s.g_dr)
    one = torch.ones_like(d)
    g = torch.where(look, T.g[gi] * (1 - fr) + T.g[gi + 1] * fr, one)
    w = torch.where(inside & (b < 0), torch.zeros_like(d), g).prod(1)
    fe = (d - (f32(s.e_r0) + bc * f32(s.e_dr))) / f32(s.e_dr)
    et = torch.where(look, (T.e[ei] * (1 - fe) + T.e[ei + 1] * fe) / d, torch.zeros_like(d))
    c = _e0() * q[None, :] / (d2 * d)
    far = torch.where(inside, torch.zeros_like(c), c)
    E = torch.stack([((et - c) * r[k]).sum(1) for k in range(3)], 1)
    E0 = torch.stack([-(far * r[k]).sum(1) for k in range(3)], 1)
    mag = E.norm(dim=1)
    eh = torch.where(mag[:, None] > 0, E / mag[:, None], torch.zeros_like(E))
    p1, p2, p3 = _langevin(mag)
    # the force, on the chosen atoms
    if len(atoms) != s.n_atoms:
        r, d2, d, d2f, dist = [v[:, atoms] for v in r], d2[:, atoms], d[:, atoms], d2f[:, atoms], dist[:, atoms]
    ta = types[atoms]
    vt = 4.0 / 3.0 * PI * _t(s.rmax) ** 3 * 0.0074 / f32(s.n_mc)
    vt = _f32(vt)[ta][None, :]
    qi = q[atoms][None, :]
    sden = (w / n)[:, None]
    R = sum(eh[:, k, None] * r[k] for k in range(3)) / d
    dp1, dp2, dp3 = 3 * R, 7.5 * R * R - 1.5, (17.5 * R * R - 7.5) * R
    t1, t2, t3 = P0 * p1[:, None] / (d2 * d), Q0 * p2[:, None] / (d2 * d2), O0 * p3[:, None] / (d2 * d2 * d)
    inside = d2f <= _f32(rmax[ta] ** 2)[None, :]
    bf = _bin(_f32(_f32(dist - f32(s.f_r0)) * _inv(s.f_dr) + 0.5))
    look = inside & (bf >= 0) & (bf < n_f)
    bc = torch.clamp(bf, 0, n_f - 1)
    fi = ta[None, :] * n_f + bc
    ff = (d - (f32(s.f_r0) + bc * f32(s.f_dr))) / f32(s.f_dr)
    lj = torch.where(look, (T.f[fi] * (1 - ff) + T.f[fi + 1] * ff) / d, torch.zeros_like(d))
    cdd = torch.where(inside, torch.zeros_like(d), P0 / (3 * n[:, None] * d2 * d))
    pdr = 3 * sum(E0[:, k, None] * r[k] for k in range(3)) / d2
    radial = (t1 * dp1 + t2 * dp2 + t3 * dp3) / d
    axial = t1 + t2 * dp1 + t3 * dp2
    F = [(-vt * (qi * (sden * (radial * r[k] - axial * eh[:, k, None]) + cdd * (pdr * r[k] - E0[:, k, None])) +
                 sden * lj * r[k])).sum(0) for k in range(3)]
    return torch.stack(F, 1)


def _chunks(n, per_row, budget=24_000_000):
    step = max(1, budget // max(1, per_row))
    return [slice(k, min(n, k + step)) for k in range(0, n, step)]


def _isspa(s, T, x, q, step, window):
    points, owner = _points(s, x, step, window)
    F = torch.zeros((s.n_atoms, 3), dtype=D, device=x.device)
    every = torch.arange(s.n_atoms, device=x.device)
    for c in _chunks(len(points), s.n_atoms):
        F += _isspa_chunk(s, T, x, q, points[c], owner[c], every)
    return F


def _exclusions(s):
    """Excluded pairs by the reference's scan: ascending entries above the atom."""
    rows, cols = [], []
    start = 0
    for a, stop in enumerate(s.n_excl_cum):
        top = -(1 << 31)
        for e in s.excl_list[start:stop]:
            if e > a and e < s.n_atoms and e >= top:
                rows += [a, e]
                cols += [e, a]
            top = max(top, e)
        start = stop
    return rows, cols


def _nonbond(s, T, x, q, atoms, cutoff=0.0):
    dev = x.device
    ljt = torch.as_tensor(s.lj_type.astype(np.int64), device=dev)
    nbp = torch.as_tensor(np.asarray(s.nb_parm_index).astype(np.int64).reshape(s.n_lj_types, s.n_lj_types), device=dev)
    rm = _t(s.rmax)[torch.as_tensor(s.isspa_type.astype(np.int64), device=dev)][None, :]
    rows, cols = _exclusions(s)
    rows, cols = (torch.as_tensor(np.asarray(v, np.int64), device=dev) for v in (rows, cols))
    slot = torch.full((s.n_atoms,), -1, dtype=torch.int64, device=dev)
    epf = 1.0 - 1.0 / EP
    L = float(np.float32(s.box))
    out = []
    for c in _chunks(len(atoms), s.n_atoms):
        at = atoms[c]
        dec, r = _image(x[at][:, None, :], x[None, :, :], L)
        own = at[:, None] == torch.arange(s.n_atoms, device=dev)[None, :]
        d2 = torch.where(own, torch.ones_like(r[0]), r[0] ** 2 + r[1] ** 2 + r[2] ** 2)
        d = torch.sqrt(d2)
        qq = q[at][:, None] * q[None, :]
        d2f = _d2_float(dec)
        two = _f32(2 * rm) ** 2
        fs = torch.where(d2f > _f32(two), -2 * qq * epf / (3 * d2 * d), -qq * epf * (8 * rm - 3 * d) / (24 * rm ** 4))
        k = nbp[ljt[at]][:, ljt]
        i6 = 1.0 / d2 ** 3
        pair = i6 * (12 * T.A[k] * i6 - 6 * T.B[k]) / d2 + qq / (d2 * d)
        slot.fill_(-1)
        slot[at] = torch.arange(len(at), device=dev)
        keep = slot[rows] >= 0
        ex = torch.zeros_like(own)
        ex[slot[rows[keep]], cols[keep]] = True
        fs = fs + torch.where(ex, torch.zeros_like(pair), pair)
        drop = own
        if cutoff > 0:
            rc = np.float32(cutoff)
            drop = own | ~(d2f < float(rc * rc))
        fs = torch.where(drop, torch.zeros_like(fs), fs)
        out.append(torch.stack([(fs * r[m]).sum(1) for m in range(3)], 1))
    return torch.cat(out)


def _bonded_energy(s, T, x, q):
    L = float(np.float32(s.box))
    dev = x.device
    idx = lambda a: torch.as_tensor(np.asarray(a).astype(np.int64), device=dev)  # noqa: E731
    vec = lambda a, b: torch.stack(_image(x[a], x[b], L)[1], -1)  # noqa: E731
    U = torch.zeros((), dtype=D, device=dev)
    if len(s.bond_atoms):
        b = idx(s.bond_atoms)
        p = _t(s.bond_params)[b[:, 2]]
        U = U + (0.5 * p[:, 0] * (vec(b[:, 0], b[:, 1]).norm(dim=1) - p[:, 1]) ** 2).sum()
    if len(s.angle_atoms):
        a = idx(s.angle_atoms)
        p = _t(s.angle_params)[a[:, 3]]
        u, v = vec(a[:, 0], a[:, 1]), vec(a[:, 2], a[:, 1])
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
        U = U + (0.5 * p[:, 0] * (th - p[:, 1]) ** 2).sum()
    if len(s.dih_atoms):
        raw, t = idx(s.dih_atoms), idx(s.dih_types)
        d = raw.abs()
        p, sc = _t(s.dih_params)[t], _t(s.scaled14)[t]
        b1, b2, b3 = vec(d[:, 0], d[:, 1]), vec(d[:, 1], d[:, 2]), vec(d[:, 2], d[:, 3])
        m, n = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        phi = torch.atan2(torch.linalg.cross(m, n).norm(dim=1), (m * n).sum(1))
        U = U + (p[:, 1] * (1 + torch.cos(p[:, 0] * phi - p[:, 2]))).sum()
        one4 = (raw[:, 2] > 0) & (raw[:, 3] > 0)
        d, sc = d[one4], sc[one4]
        ljt = idx(s.lj_type)
        nbp = idx(np.asarray(s.nb_parm_index)).reshape(s.n_lj_types, s.n_lj_types)
        k = nbp[ljt[d[:, 0]], ljt[d[:, 3]]]
        r2 = (vec(d[:, 0], d[:, 3]) ** 2).sum(1)
        i6 = 1.0 / r2 ** 3
        U = U + (i6 * (T.A[k] * i6 - T.B[k]) / sc[:, 1] + q[d[:, 0]] * q[d[:, 3]] / (torch.sqrt(r2) * sc[:, 0])).sum()
    return U


def _bonded(s, T, x, q, create_graph=False):
    y = x.detach().clone().requires_grad_()
    U = _bonded_energy(s, T, y, q)
    return -torch.autograd.grad(U, y, create_graph=create_graph)[0] if U.requires_grad else torch.zeros_like(x)


def _axis(s, x):
    """Weights of the restrained groups' centres, and the vector between them."""
    bl = torch.as_tensor(np.asarray(s.bias_list).astype(np.int64), device=x.device)
    m = _t(s.bias_mass_fraction())
    com = [(m[bl[:, 1] == g, None] * x[bl[bl[:, 1] == g, 0]]).sum(0) for g in (0, 1)]
    r = com[0] - com[1]
    L = float(np.float32(s.box))
    return bl, m, r - L * (r > 0.5 * L).to(D) + L * (r < -0.5 * L).to(D)


def _umbrella(s, x):
    F = torch.zeros_like(x)
    if s.us_on:
        bl, m, r = _axis(s, x)
        d = r.norm()
        sign = torch.where(bl[:, 1] == 0, -1.0, 1.0).to(D)
        F.index_add_(0, bl[:, 0], (sign * float(np.float32(s.us_k)) * (d - float(np.float32(s.us_x0))) / d * m)[:, None] * r[None, :])
    return F


def _leapfrog(s, x, v, F, step, window):
    mass = _t(s.vel[:, 3])[:, None]
    dt, kT, L = (float(np.float32(u)) for u in (s.dt, s.kT, s.box))
    i = np.arange(s.n_atoms, dtype=np.uint64)
    hit = _u01(_philox(i, 0, step, (window << 8) | 1, s.seed)[0]) < float(np.float32(s.pnu))
    o = [_u01_open0(u) for u in _philox(i, 1, step, (window << 8) | 1, s.seed)]
    ra, rb = np.sqrt(-2 * np.log(o[0])), np.sqrt(-2 * np.log(o[2]))
    g = np.stack([ra * np.cos(2 * np.pi * o[1]), ra * np.sin(2 * np.pi * o[1]), rb * np.cos(2 * np.pi * o[3])], 1)
    v = torch.where(_t(hit, torch.bool)[:, None], _t(g) * torch.sqrt(kT / mass) + F * dt / (2 * mass), v + F * dt / mass)
    x = x + v * dt
    return torch.where(x > L, x - L, torch.where(x < 0, x + L, x)), v


def _exact_forces(case, s, T, x, q, step, window):
    every = torch.arange(s.n_atoms, device=x.device)
    F = _bonded(s, T, x, q) + _nonbond(s, T, x, q, every, case["cutoff"]) + _umbrella(s, x)
    return F + _isspa(s, T, x, q, step, window) if case["solvent"] else F


def _exact_adjoint(case, systems, step):
    out = [[], [], [], [], []]
    for w, s in enumerate(systems):
        x, q = _t(s.pos[:, :3]), _t(s.pos[:, 3])
        T = _Tables(s)
        leaves = T.leaves()
        bl, _, r = _axis(s, x)
        n = r / r.norm()
        c = torch.zeros_like(x)
        c.index_add_(0, bl[:, 0], torch.where(bl[:, 1] == 0, 0.5, -0.5).to(D)[:, None] * n[None, :])
        atoms = torch.unique(bl[:, 0])
        rest = (_bonded(s, T, x, q, create_graph=True) * c).sum() + (_nonbond(s, T, x, q, atoms) * c[atoms]).sum()
        J = float(rest.detach())
        grads = [torch.zeros_like(t) if g is None else g
                 for t, g in zip(leaves, torch.autograd.grad(rest, leaves, allow_unused=True))]
        points, owner = _points(s, x, step, w)
        for k in _chunks(len(points), s.n_atoms, 6_000_000):
            part = (_isspa_chunk(s, T, x, q, points[k], owner[k], atoms) * c[atoms]).sum()
            J += float(part.detach())
            for a, g in zip(grads, torch.autograd.grad(part, leaves, allow_unused=True)):
                if g is not None:
                    a += g
        nf, ng = s.f_table.size, s.g_table.size
        got = [J, grads[0][:nf].reshape(s.f_table.shape), grads[1][:ng].reshape(s.g_table.shape), grads[2], grads[3]]
        for o, g in zip(out, got):
            o.append(g if isinstance(g, float) else g.detach().cpu().numpy())
    return [np.asarray(o, np.float64) for o in out]


def exact(case, seed):
    pairs = sum(n * n * case["n_mc"] for n in _sizes(case)) * case["steps"] if case["solvent"] else 0
    if pairs > 2.5e9:  # over 20 seconds in 64 bits
        return None
    systems = _systems(case, seed)
    step = _start_step(seed)
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, systems, step)
    out = []
    for w, s in enumerate(systems):
        T = _Tables(s)
        x, q, v = _t(s.pos[:, :3]), _t(s.pos[:, 3]), _t(s.vel[:, :3])
        if kind == "noalloc":
            out.append([torch.cat([_isspa(s, T, x, q, step, 0), torch.zeros_like(q)[:, None]], 1)])
            continue
        if kind == "forces":
            out.append([_exact_forces(case, s, T, x, q, step, w)])
            continue
        for k in range(case["steps"]):
            F = _exact_forces(case, s, T, x, q, step + k, w)
            x, v = _leapfrog(s, x, v, F, step + k, w)
        mass, zero = _t(s.vel[:, 3])[:, None], torch.zeros_like(q)[:, None]
        one = [torch.cat([x, q[:, None]], 1), torch.cat([v, mass], 1), torch.cat([F, zero], 1)]
        out.append(one if kind == "host_step" else one[:1])
    return [torch.cat([o[k] for o in out]).cpu().numpy() for k in range(len(out[0]))]
