"""What users run with this framework, as cases that can be timed.

Two kinds of program use the public API (heddle_b200.api):

  * a simulation advances a system by many steps and reads a frame now and
    then: Integrator.step_exchange / Batch.step, with the thermostat,
    barostat and constraints of the run ("md", "batch");
  * a program with its own driver hands over positions and reads forces and
    energies back: System.set_state_f32, ForceField.step, System.state_f32
    ("frames"), or relaxes a start structure: Minimizer ("minimize").

The systems are those of the repository's configurations (SPC water, LJ
argon, rock-salt ions, a bonded chain in water), from a few hundred atoms,
where a step is a chain of short kernels, to 196,608 atoms.
"""

import math

import numpy as np
import torch

import heddle_b200 as hb
from heddle_b200 import systems as S
from heddle_b200 import units as U


def listed():
    return [
        # one force call of a small solvation box driven from outside (a
        # path-integral or hybrid driver): launch and copy latency
        dict(name="frames_water_300", kind="frames", system="water", n=300, r_cut=9.0, order=4,
             tilt=False, frames=1, scalars=False),
        # stored frames of a trajectory evaluated again with energies in a
        # tilted cell at a higher spline order; every frame needs its own list
        dict(name="frames_water_729_tilted_order6", kind="frames", system="water", n=729, r_cut=9.0,
             order=6, tilt=True, frames=2, scalars=True),
        # the same on a large orthorhombic box
        dict(name="frames_water_21952", kind="frames", system="water", n=21952, r_cut=9.0, order=4,
             tilt=False, frames=2, scalars=True),
        # a small NVT box, the size of a free-energy window: step latency
        dict(name="md_water_343_nvt", kind="md", system="water", n=343, r_cut=9.0, order=4, steps=20,
             ensemble="langevin"),
        # NPT with CSVR and stochastic cell rescaling: virial and pressure on
        # every step
        dict(name="md_water_1237_csvr_crescale", kind="md", system="water", n=1237, r_cut=9.0,
             order=4, steps=20, ensemble="csvr-c-rescale"),
        # a solvated chain: bonded terms, scaled 1-4 pairs, SHAKE and SETTLE
        dict(name="md_chain_1900_nvt", kind="md", system="chain", n=1900, r_cut=9.0, order=4, steps=20,
             ensemble="langevin"),
        # LJ argon, NVE: the pair path alone
        dict(name="md_argon_10000_nve", kind="md", system="argon", n=10000, r_cut=8.5, order=4,
             steps=20, ensemble="nve"),
        # bit-reversible dynamics of ions (exact pair forces, SPME)
        dict(name="md_ions_13824_lossless", kind="md", system="ions", n=13824, r_cut=9.0, order=4,
             steps=10, ensemble="lossless"),
        # the 8,192-molecule NVT box
        dict(name="md_water_8192_nvt", kind="md", system="water", n=8192, r_cut=9.0, order=4, steps=20,
             ensemble="langevin"),
        # the 65,536-molecule NPT box, one Monte-Carlo volume move per frame
        dict(name="md_water_65536_npt", kind="md", system="water", n=65536, r_cut=9.0, order=4,
             steps=25, ensemble="langevin-mc"),
        # an uneven batch of replicas advanced together
        dict(name="batch_12_replicas", kind="batch", system="water", n=12, lo=256, hi=2048, steps=10),
        # relaxing a start structure before dynamics
        dict(name="minimize_water_2000", kind="minimize", system="water", n=2000, r_cut=9.0, order=4,
             iterations=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames", "frames", "md", "md", "md", "md", "batch", "minimize"])
    if kind == "batch":
        return dict(kind="batch", system="water", n=rng.randint(3, 16), lo=rng.randint(256, 400),
                    hi=rng.randint(1000, 3000), steps=rng.randint(4, 20))
    if kind == "minimize":
        return dict(kind="minimize", system="water", n=_log_int(rng, 500, 8000), r_cut=9.0, order=4,
                    iterations=rng.randint(8, 24))
    if kind == "frames":
        n = _log_int(rng, 300, 30000)
        return dict(kind="frames", system="water", n=n, r_cut=rng.choice([8.0, 9.0]) if n < 1000 else
                    rng.choice([8.0, 9.0, 10.0]), order=rng.choice([4, 4, 5, 6, 8]),
                    tilt=n > 500 and rng.random() < 0.4, frames=rng.randint(1, 2),
                    scalars=rng.random() < 0.6)
    system = rng.choice(["water", "water", "water", "argon", "ions", "chain"])
    if system == "water":
        n = _log_int(rng, 300, 50000)
        return dict(kind="md", system=system, n=n, r_cut=rng.choice([8.0, 9.0]) if n < 1000 else
                    rng.choice([8.0, 9.0, 10.0]), order=rng.choice([4, 4, 4, 6]),
                    steps=rng.randint(8, 25),
                    ensemble=rng.choice(["langevin", "langevin", "langevin-mc", "csvr-c-rescale"]))
    if system == "argon":
        return dict(kind="md", system=system, n=_log_int(rng, 3000, 60000), r_cut=8.5, order=4,
                    steps=rng.randint(8, 25), ensemble="nve")
    if system == "ions":
        side = 2 * rng.randint(5, 16)
        return dict(kind="md", system=system, n=side ** 3, r_cut=9.0, order=4,
                    steps=rng.randint(5, 12), ensemble=rng.choice(["nve", "lossless"]))
    return dict(kind="md", system=system, n=rng.choice([1500, 1650, 1800, 1900, 2200, 2500, 2900, 3300]), r_cut=9.0, order=4,
                steps=rng.randint(8, 25), ensemble="langevin")


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------
TILT = (0.10, -0.06, 0.08)  # xy, xz, yz of the tilted cells, in units of the edge


def _cap_skin(spec, width, r_cut_A, skin_A):
    """The default skin, or what the cell's smallest width leaves for it."""
    room = 0.5 * width * (1.0 - 2e-4) - U.angstrom_au(r_cut_A + 0.01)
    spec.r_skin = min(U.angstrom_au(skin_A), room)
    return spec


def _spec(case, seed):
    system, n, rc = case["system"], case["n"], case["r_cut"]
    if system == "water":
        spec = S.spc_water(n, seed=seed, velocity_seed=seed + 1, r_cut_A=rc, order=case["order"])
        width = spec.box[0]
        if case.get("tilt"):
            L = spec.box[0]
            spec.box = np.array([L, L, L, TILT[0] * L, TILT[1] * L, TILT[2] * L])
            s = spec.positions / L
            spec.positions = np.stack([L * s[:, 0] + spec.box[3] * s[:, 1] + spec.box[4] * s[:, 2],
                                       L * s[:, 1] + spec.box[5] * s[:, 2], L * s[:, 2]], axis=1)
            # the waters keep their shape under the shear: move whole molecules
            rigid = S.spc_water(n, seed=seed, r_cut_A=rc).positions.reshape(-1, 3, 3)
            mol = spec.positions.reshape(-1, 3, 3)
            mol[:, 1:] = mol[:, :1] + (rigid[:, 1:] - rigid[:, :1])
            spec.positions = mol.reshape(-1, 3)
            h = np.array([[L, spec.box[3], spec.box[4]], [0, L, spec.box[5]], [0, 0, L]])
            width = 1.0 / np.linalg.norm(np.linalg.inv(h), axis=1).max()
        return _cap_skin(spec, width, rc, 0.3 * rc)
    if system == "argon":
        side = max(1, math.ceil((n * 1.065) ** (1.0 / 3.0)))
        return S.lj_argon(seed=seed, velocity_seed=seed + 1, n_atoms=n, n_side=side,
                          box_m=7.84e-9 * side / 22.0)
    if system == "ions":
        spec = S.ionic_lattice(n_side=round(n ** (1.0 / 3.0)), r_cut_A=rc, seed=seed,
                               velocity_seed=seed + 1)
        return _cap_skin(spec, spec.box[0], rc, 1.0)
    return S.peptide_in_water(n_water=n, box_A=38.6 * (n / 1900.0) ** (1.0 / 3.0), seed=5,
                              velocity_seed=seed + 1)


class _State:
    """Objects of one program; the device objects are given back in order."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for o in self.__dict__.pop("own", []):
            o.close()


def _frame_buffers(n):
    return tuple(torch.empty((n, 3), dtype=d, pin_memory=True).numpy()
                 for d in (torch.float32, torch.float32, torch.int32, torch.float32))


# (fs, 1/ps, steps) of strongly damped steps that take the first heat out of
# a start structure: waters turned at random on a lattice, a chain among them
HEAT_BATH = {"water": ((0.5, 200.0, 60), (2.0, 100.0, 20)),
             "chain": ((0.25, 200.0, 160), (1.0, 100.0, 40)), "argon": (), "ions": ()}


def _damped(ctx, spec, system_kind, seed):
    """System, force field and constraints of a run ready to start."""
    system = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(system, spec)
    cons = None
    if spec.group_offsets is not None:
        cons = hb.Constraints.from_spec(system, spec)
        cons.after_kick(0.0)
    for dt_fs, friction_per_ps, steps in HEAT_BATH[system_kind]:
        bath = hb.Integrator(system, "langevin-baoab", U.time_au_fs(dt_fs),
                             friction=friction_per_ps / (1.0e-12 / U.AUT_S),
                             temperature=spec.temperature, seed=seed)
        bath.step_graph(ff, cons, n_steps=steps)
        bath.close()
    return system, ff, cons


def prepare(case, seed):
    if case["kind"] == "batch":
        specs = S.replica_batch(seed=2025, n_boxes=case["n"], lo=case["lo"], hi=case["hi"])
        master = hb.Context(0)
        own, members, systems = [], [], []
        for k, spec in enumerate(specs):
            rng = np.random.default_rng(seed * 1000 + k)
            spec.velocities = spec.velocities * rng.choice([-1.0, 1.0], size=3)
            ctx = hb.Context(0)
            system, ff, cons = _damped(ctx, spec, "water", seed + k)
            it = hb.Integrator(system, "langevin-baoab", spec.dt, friction=spec.friction,
                               temperature=spec.temperature, seed=seed + 500 + k)
            members.append((it, ff, cons))
            systems.append(system)
            own += [it, ff, cons, system, ctx]
        batch = hb.Batch(master, members)
        return _State(own=[batch] + own + [master], case=case, batch=batch, systems=systems,
                      out=[_frame_buffers(s.n) for s in systems])
    ctx = hb.Context(0)
    spec = _spec(case, seed)
    if case["kind"] == "frames":
        system = hb.System.from_spec(ctx, spec)
        ff = hb.ForceField.from_spec(system, spec)
        frames = [torch.from_numpy(f).pin_memory().numpy() for f in _frames(case, seed, spec)]
        return _State(own=[ff, system, ctx], case=case, system=system, ff=ff, frames=frames,
                      out=[_frame_buffers(spec.n) for _ in frames])
    if case["kind"] == "minimize":
        system = hb.System.from_spec(ctx, spec)
        ff = hb.ForceField.from_spec(system, spec)
        cons = hb.Constraints.from_spec(system, spec)
        mini = hb.Minimizer(ff, cons)
        return _State(own=[mini, cons, ff, system, ctx], case=case, system=system, mini=mini,
                      start=spec.positions.astype(np.float32), out=_frame_buffers(spec.n))
    ens = case["ensemble"]
    system, ff, cons = _damped(ctx, spec, case["system"], seed)
    coupling = []
    if ens in ("langevin", "langevin-mc"):
        it = hb.Integrator(system, "langevin-baoab", spec.dt, friction=spec.friction,
                           temperature=spec.temperature, seed=seed + 7)
        if ens == "langevin-mc":
            baro = hb.Barostat(system, U.pressure_au_bar(1.0), spec.temperature, seed=seed + 8,
                               frequency=25, molecules=(spec.mol_offsets, spec.mol_atoms))
            it.set_barostat(baro)
            coupling = [baro]
    elif ens == "lossless":
        # exact pair forces: a force field of its own
        ff.close()
        ff = hb.ForceField.from_spec(system, spec, exact_pairs=True)
        it = hb.Integrator(system, "velocity-verlet-lossless", spec.dt)
    else:
        it = hb.Integrator(system, "velocity-verlet", spec.dt)
        if ens == "csvr-c-rescale":
            thermo = hb.Thermostat(system, "csvr", spec.temperature, seed=seed + 8,
                                   tau=U.time_au_fs(100.0), n_constraints=spec.n_constraints)
            it.set_thermostat(thermo)
            pc = hb.PressureCoupling(system, "c_rescale", U.pressure_au_bar(1.0), U.time_au_fs(1000.0),
                                     4.5e-10 * U.PRESSURE_PA, temperature=spec.temperature,
                                     seed=seed + 9)
            it.set_barostat(pc)
            coupling = [thermo, pc]
    own = [it] + coupling + ([cons] if cons else []) + [ff, system, ctx]
    return _State(own=own, case=case, system=system, ff=ff, cons=cons, it=it,
                  out=_frame_buffers(spec.n))


def _frames(case, seed, spec):
    """The stored positions: the first structure and others of the same cell
    (every molecule turned anew about its oxygen)."""
    out = [spec.positions.astype(np.float32)]
    for k in range(1, case["frames"]):
        out.append(_spec(case, seed + 7919 * k).positions.astype(np.float32))
    return out


SCALARS = ("lj", "coulomb_real", "recip", "potential", "virial")


def run(state):
    case = state.case
    if case["kind"] == "md":
        pos, vel, img, frc = state.it.step_exchange(state.ff, state.cons, case["steps"], out=state.out)
        return {"positions": pos, "velocities": vel, "images": img, "forces": frc}
    if case["kind"] == "batch":
        state.batch.step(case["steps"])
        return [dict(zip(("positions", "velocities", "images", "forces"), s.state_f32(o)))
                for s, o in zip(state.systems, state.out)]
    if case["kind"] == "minimize":
        state.system.set_state_f32(state.start)
        rows = [state.mini.begin()] + state.mini.iterate(case["iterations"])
        state.system.state_f32(state.out)
        return {"energy": np.array([r["energy"] for r in rows]),
                "max_force": np.array([r["max_force"] for r in rows]),
                "accepted": np.array([int(r["accepted"]) for r in rows]),
                "positions": state.out[0], "forces": state.out[3]}
    got = []
    for frame, out in zip(state.frames, state.out):
        state.system.set_state_f32(frame)
        state.ff.step(scalars=case["scalars"])
        state.system.state_f32(out)
        res = {"forces": out[3]}
        if case["scalars"]:
            sc = state.ff.scalars()
            res["scalars"] = np.array([sc[k] for k in SCALARS])
        got.append(res)
    return got


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _evaluation(case):
    """(bytes, flops) of one force evaluation / step: positions read and
    forces written, charge grid written and read once by the transforms; the
    pairs within the cut-off, the splines and the transforms."""
    n = case["n"]
    atoms = {"water": 3 * n, "argon": n, "ions": n, "chain": 3 * n + 166}[case["system"]]
    per_A3 = {"water": 0.09998, "argon": 0.0207, "ions": 0.0278, "chain": 0.102}[case["system"]]
    rc = case.get("r_cut", 9.0)
    pairs = 0.5 * atoms * per_A3 * 4.0 / 3.0 * math.pi * rc ** 3
    flops = pairs * (25.0 if case["system"] == "argon" else 50.0)
    bytes_ = 100.0 * atoms
    if case["system"] != "argon":
        m = S.fft_friendly(math.ceil((atoms / per_A3) ** (1.0 / 3.0))) ** 3
        bytes_ += 24.0 * m
        flops += 5.0 * m * math.log2(m) + atoms * 8.0 * case.get("order", 4) ** 3
    return bytes_, flops


def work(case):
    if case["kind"] == "batch":
        specs = S.replica_batch(seed=2025, n_boxes=case["n"], lo=case["lo"], hi=case["hi"])
        per = [_evaluation(dict(system="water", n=s.n // 3)) for s in specs]
        b, f = sum(p[0] for p in per), sum(p[1] for p in per)
        times = case["steps"]
    else:
        b, f = _evaluation(case)
        times = {"md": case.get("steps"), "minimize": case.get("iterations", 0) + 1,
                 "frames": case.get("frames")}[case["kind"]]
    return {"bytes": b * times, "flops": f * times}


def tolerance(case):
    """About four times what a change of the start positions by half a unit
    in their last place makes of the same outputs three passes later."""
    if case["kind"] == "frames":
        # one evaluation in single precision: each side is within 1e-5 of
        # the 64-bit forces on the largest boxes
        return {"rel": 3e-5, "max": 3e-3}
    if case["kind"] == "minimize":
        return {"rel": 5e-5, "max": 2e-3}
    if case["system"] in ("argon", "ions"):
        return {"rel": 2e-4, "max": 2e-2, "differ": 1e-5}
    # liquid water parts faster: the velocities of its hydrogens show it first
    return {"rel": 1.3e-2, "max": 0.95, "differ": 1e-4}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "frames":
        return None
    spec = _spec(case, seed)
    return [_exact_frame(spec, f.astype(np.float64), case["scalars"]) for f in _frames(case, seed, spec)]


def _exact_frame(spec, pos, scalars):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = dict(dtype=torch.float64, device=dev)
    x = torch.tensor(pos, **t64)
    q = torch.tensor(np.asarray(spec.charges, dtype=np.float32).astype(np.float64), **t64)
    lx, ly, lz, xy, xz, yz = (float(v) for v in spec.box)
    h = torch.tensor([[lx, xy, xz], [0.0, ly, yz], [0.0, 0.0, lz]], **t64)  # columns: cell vectors
    hinv = torch.linalg.inv(h)
    e_lj, e_c, w_pair, f = _exact_pairs(spec, x, q, h, hinv, dev)
    e_rec, w_rec, f_rec = _exact_recip(spec, x, q, h, hinv, dev)
    res = {"forces": (f + f_rec).cpu().numpy()}
    if scalars:
        e_self = float(spec.alpha / math.sqrt(math.pi) * (q * q).sum())
        res["scalars"] = np.array([e_lj, e_c, e_rec, e_lj + e_c + e_rec - e_self, w_pair + w_rec])
    return res


def _exact_pairs(spec, x, q, h, hinv, dev):
    """Lennard-Jones with the switch and erfc-screened Coulomb over all pairs
    within the cut-off, each pair seen from both atoms; atoms in slabs along
    the third axis, so that a chunk meets only the slabs near it."""
    n = x.shape[0]
    rc = float(max(spec.lj_cutoff.max(), spec.r_cut_coul))
    s = (x @ hinv.T)
    s = s - torch.floor(s + 0.5)
    order = torch.argsort(s[:, 2])
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device=dev)
    xs, ss, qs = x[order], s[order], q[order]
    typ = torch.tensor(spec.types.astype(np.int64), device=dev)[order]
    tab = [torch.tensor(np.asarray(a, dtype=np.float64), device=dev)
           for a in (spec.lj_sigma, spec.lj_epsilon, spec.lj_cutoff, spec.lj_switch)]
    off = torch.tensor(spec.excl_offsets.astype(np.int64), device=dev)
    part = torch.tensor(spec.excl_partners.astype(np.int64), device=dev)
    owner = torch.repeat_interleave(torch.arange(n, device=dev), off[1:] - off[:-1])
    ex_i, ex_j = rank[owner], rank[part]
    reach = rc / float(h[2, 2]) + 1e-9
    c = ss[:, 2]
    f = torch.zeros_like(xs)
    e_lj = e_c = w = 0.0
    a = float(spec.alpha)
    step = max(1, min(n, 1024))
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        lo, hi = float(c[i0]) - reach, float(c[i1 - 1]) + reach
        near = torch.zeros(n, dtype=torch.bool, device=dev)
        for sh in (-1.0, 0.0, 1.0):
            near |= (c + sh >= lo) & (c + sh <= hi)
        js = torch.nonzero(near).reshape(-1)
        d = ss[i0:i1, None, :] - ss[None, js, :]
        d = d - torch.round(d)
        d = d @ h.T
        r2 = (d * d).sum(-1)
        ii = torch.arange(i0, i1, device=dev)
        ok = (r2 < rc * rc) & (ii[:, None] != js[None, :])
        col = torch.full((n,), -1, dtype=torch.int64, device=dev)
        col[js] = torch.arange(js.numel(), device=dev)
        sel = (ex_i >= i0) & (ex_i < i1) & (col[ex_j] >= 0)
        ok[ex_i[sel] - i0, col[ex_j[sel]]] = False
        a_i, a_j = torch.nonzero(ok, as_tuple=True)
        dv, r2 = d[a_i, a_j], r2[a_i, a_j]
        ti, tj = typ[i0:i1][a_i], typ[js][a_j]
        sig, eps, cut, sw = (t[ti, tj] for t in tab)
        inv2 = 1.0 / r2
        sr6 = (sig * sig * inv2) ** 3
        u = 4.0 * eps * (sr6 * sr6 - sr6)
        fac = 24.0 * eps * inv2 * (2.0 * sr6 * sr6 - sr6)
        width = torch.clamp(cut * cut - sw * sw, min=1e-30)
        tau = (r2 - sw * sw) / width
        omt = 1.0 - tau
        smooth = omt * omt * (1.0 + 2.0 * tau)
        chain = 12.0 * tau * omt / width
        switched = (r2 > sw * sw) & (cut > sw)
        fac = torch.where(switched, smooth * fac + chain * u, fac)
        u = torch.where(switched, smooth * u, u)
        inside = r2 <= cut * cut
        fac, u = torch.where(inside, fac, 0.0), torch.where(inside, u, 0.0)
        r = torch.sqrt(r2)
        qq = torch.where(r2 <= spec.r_cut_coul ** 2, qs[i0:i1][a_i] * qs[js][a_j], 0.0)
        ec = qq * torch.erfc(a * r) / r
        fac = fac + inv2 * (ec + qq * 2.0 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2))
        f.index_add_(0, ii[a_i], fac[:, None] * dv)
        e_lj += 0.5 * float(u.sum())
        e_c += 0.5 * float(ec.sum())
        w += 0.5 * float((fac * r2).sum())
    return e_lj, e_c, w, f[rank]


def _bspline(p, t):
    """Weights M_p(d + t) and derivatives M_p'(d + t), d = 0 .. p - 1."""
    def m(k, u):
        if k == 1:
            return ((u >= 0.0) & (u < 1.0)).to(u.dtype)
        return (u * m(k - 1, u) + (k - u) * m(k - 1, u - 1.0)) / (k - 1)
    u = t[..., None] + torch.arange(p, device=t.device, dtype=t.dtype)
    return m(p, u), m(p - 1, u) - m(p - 1, u - 1.0)


def _exact_recip(spec, x, q, h, hinv, dev):
    """Smooth particle-mesh Ewald reciprocal part on the case's grid."""
    n, p = x.shape[0], int(spec.order)
    K = [int(g) for g in spec.grid]
    s = x @ hinv.T
    s = s - torch.floor(s + 0.5)
    idx, wt, dwt = [], [], []
    for ax in range(3):
        u = (s[:, ax] + 0.5) * K[ax]
        b = torch.floor(u)
        w, dw = _bspline(p, u - b)
        idx.append((b.long()[:, None] - torch.arange(p, device=dev)) % K[ax])
        wt.append(w)
        dwt.append(dw * K[ax])
    flat = ((idx[0][:, :, None, None] * K[1] + idx[1][:, None, :, None]) * K[2]
            + idx[2][:, None, None, :]).reshape(n, -1)
    W = torch.einsum("na,nb,nc->nabc", wt[0], wt[1], wt[2]).reshape(n, -1)
    rho = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=dev)
    rho.index_add_(0, flat.reshape(-1), (q[:, None] * W).reshape(-1))
    hat = torch.fft.fftn(rho.reshape(K))
    mods, freq = [], []
    node = _bspline(p, torch.zeros(1, dtype=torch.float64, device=dev))[0][0]  # M_p(0 .. p - 1)
    for ax in range(3):
        k = torch.arange(K[ax], dtype=torch.float64, device=dev)
        ph = torch.exp(2j * math.pi * k[:, None] * torch.arange(p - 1, device=dev) / K[ax])
        mod = (node[1:p].to(ph.dtype) * ph).sum(-1).abs() ** 2
        bad = mod < 1e-7
        mod = torch.where(bad, 0.5 * (torch.roll(mod, 1) + torch.roll(mod, -1)), mod)
        mods.append(1.0 / mod)
        freq.append(torch.where(k <= K[ax] // 2, k, k - K[ax]))
    B = mods[0][:, None, None] * mods[1][None, :, None] * mods[2][None, None, :]
    m = torch.stack(torch.meshgrid(*freq, indexing="ij"), dim=-1)
    k2 = ((2.0 * math.pi * (m @ hinv)) ** 2).sum(-1)
    vol = float(torch.linalg.det(h))
    k2s = torch.where(k2 > 0, k2, 1.0)
    G = torch.where(k2 > 0, 4.0 * math.pi / vol / k2s * torch.exp(-k2 / (4.0 * spec.alpha ** 2)) * B, 0.0)
    power = G * hat.abs() ** 2
    e = 0.5 * float(power.sum())
    w = 0.5 * float((power * (1.0 - k2 / (2.0 * spec.alpha ** 2))).sum())
    V = (torch.fft.ifftn(G * hat).real * (K[0] * K[1] * K[2])).reshape(-1)
    Vn = V[flat].reshape(n, p, p, p)
    grad = torch.stack([torch.einsum("nabc,na,nb,nc->n", Vn, *[(dwt if ax == d else wt)[ax] for ax in range(3)])
                        for d in range(3)], dim=-1)
    return e, w, -(q[:, None] * grad) @ hinv
