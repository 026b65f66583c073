"""Timed cases of the framework: what a user of it has it do, each through the
public entry points of ``protomol_b200``.

Kinds of work (the sizes and options come from the configurations the
benchmark and the tests name):

* ``call``: one force line evaluated as ProtoMol calls a force,
  ``SystemForce.evaluate(positions, forces, energies)`` on host arrays.
* ``request``: a single energy and force evaluation of a water box with PME
  (the served form's evaluation): positions in, energies and forces out.
* ``segment``: an MD segment of a water box (the served form's other
  request, and the plain single-system form): positions and velocities in,
  the steps on the device, positions, velocities and energies out.
* ``ensemble``: uneven small boxes advanced together, a segment per pass.
* ``polymer_segment``, ``polymer_call``: implicit solvent (GB) with LJ,
  Coulomb and bonded terms over all pairs, as a Langevin segment and as the
  force lines of one evaluation.
* ``gb_device``: GB forces on device arrays the caller owns.
* ``scpism``: the SCPISM implicit-solvent force lines of one evaluation.

Systems in mixed precision compute pair forces in FP32, and their results
are taken as FP32 arrays (what a DCD trajectory or an FP32 host program
keeps); systems in double precision return FP64.
"""
import ctypes
import math
from types import SimpleNamespace

import numpy as np
import torch

from protomol_b200 import (Context, ForceFactory, GpuSystem, LangevinLeapfrogIntegrator,
                           LeapfrogIntegrator, ScalarStructure, _lib, systems)
from protomol_b200.engine import SystemEnsemble
from protomol_b200.serve import ALPHA, LJ_SWITCHON, ORDER, RC, WATER_DENSITY, fft_size

COULOMB, LJ, BOND, ANGLE, DIHEDRAL = range(5)
SOLUTE, SOLVENT = 1.0, 78.5
OBC = (1.0, 0.8, 4.85)
SWITCHES = {
    # the water test systems' LJ C2 + Coulomb C1 and C2 + C2, and Cn
    "c2c1": ("C2 -switchon {on:g} -cutoff {rc:g}", "C1 -cutoff {rc:g}"),
    "c2c2": ("C2 -switchon {on:g} -cutoff {rc:g}", "C2 -switchon {on:g} -cutoff {rc:g}"),
    "cncn": ("Cn -n 4 -switchon {on:g} -cutoff {rc:g}", "Cn -n 4 -switchon {on:g} -cutoff {rc:g}"),
}


def listed():
    return [
        # ProtoMol's own use of a cutoff force line on the small water box
        dict(name="call_648", kind="call", waters=216, algorithm="NonbondedCutoff",
             switches="c2c1", on=7.0, rc=8.0, precision="mixed", virial=False),
        # a solvated box with the Cn switch and the virial (pressure output)
        dict(name="call_12000_cn", kind="call", waters=4000, algorithm="NonbondedCutoff",
             switches="cncn", on=8.0, rc=10.0, precision="mixed", virial=True),
        # the small plain configuration: FP64, 0.5 fs leapfrog
        dict(name="segment_648_double", kind="segment", waters=216, terms="cutoff",
             precision="double", integrator="leapfrog", dt=0.5, steps=50),
        # the served stream's smallest and largest evaluation
        dict(name="request_501", kind="request", waters=167, precision="mixed", virial=False),
        dict(name="request_49998", kind="request", waters=16666, precision="mixed", virial=False),
        # the solvated single system with PME, leapfrog 1 fs
        dict(name="segment_23550", kind="segment", waters=7850, terms="pme", precision="mixed",
             integrator="leapfrog", dt=1.0, steps=50),
        # a middling Langevin segment of the served stream
        dict(name="segment_5001", kind="segment", waters=1667, terms="pme", precision="mixed",
             integrator="langevin", dt=1.0, steps=50),
        # the batched ensemble's boxes (100 to 1,000 waters), 20 steps a pass
        dict(name="ensemble_24", kind="ensemble", boxes=24, least=100, most=1000, steps=20),
        # the implicit-solvent polymer, Langevin 1 fs
        dict(name="polymer_segment_2000", kind="polymer_segment", atoms=2000, steps=50),
        # a protein-sized molecule, FP64, GB + ACE + LJ + Coulomb + bonded
        dict(name="polymer_call_544_double", kind="polymer_call", atoms=544, precision="double"),
        # GB forces of a large molecule for a host that owns its buffers
        dict(name="gb_device_8191", kind="gb_device", atoms=8191, precision="mixed"),
        # the WW-domain sized SCPISM force lines
        dict(name="scpism_547", kind="scpism", atoms=547, precision="double"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "call", "request", "request", "segment", "segment", "ensemble",
                       "polymer_segment", "polymer_call", "gb_device", "scpism"])
    if kind == "call":
        return dict(kind=kind, waters=size(216, 8000),
                    algorithm=rng.choice(["NonbondedCutoff", "NonbondedCutoff", "NonbondedFull"]),
                    switches=rng.choice(sorted(SWITCHES)), on=round(rng.uniform(6.0, 7.0), 2),
                    rc=round(rng.uniform(7.5, 8.5), 2),
                    precision=rng.choice(["mixed", "mixed", "double"]),
                    virial=rng.random() < 0.5)
    if kind == "request":
        return dict(kind=kind, waters=size(167, 16000), precision="mixed",
                    virial=rng.random() < 0.3)
    if kind == "segment":
        pme = rng.random() < 0.7
        return dict(kind=kind, waters=size(216, 7000 if pme else 1500),
                    terms="pme" if pme else "cutoff",
                    precision="mixed" if pme else "double",
                    integrator=rng.choice(["leapfrog", "langevin"]),
                    dt=rng.choice([0.5, 1.0]), steps=rng.randint(20, 50))
    if kind == "ensemble":
        return dict(kind=kind, boxes=rng.randint(4, 24), least=100, most=size(300, 1000),
                    steps=rng.randint(8, 20))
    if kind == "polymer_segment":
        return dict(kind=kind, atoms=size(100, 2400), steps=rng.randint(20, 50))
    if kind == "polymer_call":
        return dict(kind=kind, atoms=size(50, 1200), precision=rng.choice(["mixed", "double"]))
    if kind == "gb_device":
        mixed = rng.random() < 0.7
        return dict(kind=kind, atoms=size(500, 10000 if mixed else 4000),
                    precision="mixed" if mixed else "double")
    return dict(kind=kind, atoms=size(60, 1500), precision="double")


# ------------------------------------------------------------------ inputs
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def _box(waters, seed):
    """The seeded TIP3P box the served stream and the ensembles use, its bonds
    and angles off their rest values by about kT."""
    s = systems.water_box_for_density(waters, WATER_DENSITY, seed, jitter=0.2)
    s.pos += np.random.default_rng([seed, 2]).normal(0.0, 0.03, s.pos.shape)
    return s


def _water_grid(waters):
    return fft_size(int(math.ceil((waters / WATER_DENSITY) ** (1.0 / 3.0))))


def _pme_lines(waters):
    g = _water_grid(waters)
    return ["Bond", "Angle",
            f"LennardJones -algorithm NonbondedCutoff -switchingFunction C2 "
            f"-switchon {LJ_SWITCHON} -cutoff {RC} -cutoff {RC}",
            f"Coulomb -algorithm PMEwald -alpha {ALPHA} -cutoff {RC} -order {ORDER} "
            f"-gridsize {g} {g} {g}"]


def _cutoff_line(case):
    lj, co = (t.format(on=case["on"], rc=case["rc"]) for t in SWITCHES[case["switches"]])
    return (f"LennardJones Coulomb -algorithm {case['algorithm']} -switchingFunction {lj} "
            f"-switchingFunction {co} -cutoff {case['rc']:g}")


#: The small plain configuration's force line (C2 switches, 7 to 8 A).
SMALL = dict(algorithm="NonbondedCutoff", switches="c2c2", on=7.0, rc=8.0)


def _polymer(atoms, seed, kinds=40):
    """A linear heteropolymer as ``systems.gb_polymer`` makes it (bond 1.53 A,
    109.5 degree angles, contacts beyond 3 A, the same charge, LJ and radius
    distributions), with the LJ parameters of a force field's tens of atom
    types."""
    rng = np.random.default_rng(seed)
    n, b, bend = atoms, 1.53, math.radians(180.0 - 109.5)
    pos = np.zeros((n, 3))
    pos[1] = [b, 0, 0]
    pos[2] = pos[1] + b * np.array([math.cos(bend), math.sin(bend), 0.0])
    for i in range(3, n):
        u = (pos[i - 1] - pos[i - 2]) / b
        for _ in range(40):
            t = rng.normal(size=(8, 3))
            t -= (t @ u)[:, None] * u
            t /= np.linalg.norm(t, axis=1, keepdims=True)
            cand = pos[i - 1] + b * (math.cos(bend) * u + math.sin(bend) * t)
            if i < 4:
                ok = np.ones(8, bool)
            else:
                ok = ((pos[None, :i - 3] - cand[:, None]) ** 2).sum(-1).min(1) > 9.0
            if ok.any():
                break
        pos[i] = cand[int(np.argmax(ok))]
    pos += rng.normal(0.0, 0.03, pos.shape) - pos.mean(0)
    q = rng.uniform(-0.5, 0.5, n)
    q -= q.mean()
    mass = np.array([12.011, 14.007, 15.999, 1.008, 32.06])[np.arange(n) % 5]
    k = np.arange(n)
    ex = np.concatenate([np.stack([k[:-d], k[d:], np.full(n - d, c)], 1)
                         for d, c in ((1, 2), (2, 2), (3, 1))])
    kinds = min(kinds, n)
    eps, half = rng.uniform(0.05, 0.2, kinds), rng.uniform(3.0, 3.8, kinds) * 2 ** (1 / 6) / 2
    sysm = SimpleNamespace(
        pos=pos, vel=systems.mb_velocities(mass, 300.0, rng),
        charge=q * systems.SQRTCOULOMBCONSTANT, mass=mass,
        type=rng.integers(0, kinds, n).astype(np.int32), molecule=np.zeros(n, np.int32),
        lj=systems.charmm_lj_table(eps, half), exclusions=ex.astype(np.int32),
        bonds=np.stack([k[:-1], k[1:]], 1).astype(np.int32),
        bond_params=np.tile([300.0, b], (n - 1, 1)),
        angles=np.stack([k[:-2], k[1:-1], k[2:]], 1).astype(np.int32),
        angle_params=np.tile([50.0, math.radians(109.5), 0.0, 0.0], (n - 2, 1)),
        dihedrals=np.stack([k[:-3], k[1:-2], k[2:-1], k[3:]], 1).astype(np.int32),
        dihedral_params=np.tile([0.2, 3.0, 0.0], (n - 3, 1)),
        periodic=False, box=np.zeros(12), coulomb_scaling=1.0, water=np.zeros(n, np.int32),
        gb_vdwr=rng.uniform(1.2, 1.9, n),
        gb_scale=np.array([0.72, 0.79, 0.85, 0.85, 0.96])[np.arange(n) % 5],
        gb_offset=np.full(n, 0.09), gb_obc=OBC)
    return sysm


def _scpism_polymer(atoms, seed):
    """The polymer with SCPISM parameters in the ranges of a protein's."""
    s = _polymer(atoms, seed)
    rng = np.random.default_rng([seed, 1])
    n = atoms
    hb = np.where(np.arange(n) % 12 == 4, 1, np.where(np.arange(n) % 12 == 9, 2, 0))
    root = rng.uniform(0.674, 0.775, n)
    s.scpism = dict(scp_sqrtalpha=root, scp_alpha=root * root,
                    scp_zeta=rng.uniform(1.4, 2.0, n), scp_eta=rng.uniform(0.023, 0.067, n),
                    scp_c=rng.uniform(0.22, 0.8, n),
                    scp_g=np.where(hb > 0, rng.uniform(0.47, 1.4, n), 0.47),
                    scp_hbond=hb.astype(np.int32), scp_residue=(np.arange(n) // 16).astype(np.int32),
                    scp_name=np.where(np.arange(n) % 48 == 4, 1,
                                      np.where(hb == 2, 2, 0)).astype(np.int32))
    return s


GB_LINES = ["GBBornRadii -algorithm NonbondedSimpleFull", "GBPartialSum -algorithm NonbondedSimpleFull",
            f"GBForce -algorithm NonbondedSimpleFull -soluteDielec {SOLUTE} -solventDielec {SOLVENT}"]
ALL_PAIRS = ["LennardJones -algorithm NonbondedSimpleFull", "Coulomb -algorithm NonbondedSimpleFull"]
BONDED = ["Bond", "Angle", "Dihedral"]
SCPISM_LINES = [
    "LennardJones CoulombSCPISM -algorithm NonbondedCutoff -switchingFunction Cn -n 4 "
    "-switchon 8.0 -cutoff 20.0 -switchingFunction Cn -n 4 -switchon 8.0 -cutoff 20.0 -cutoff 20.0",
    "BornRadii -algorithm NonbondedCutoff -switchingFunction Cutoff -bornswitch 3 -cutoff 5 -cutoff 5",
    "BornSelf -algorithm NonbondedCutoff -switchingFunction Cutoff -bornswitch 3 -cutoff 5 -cutoff 5"]


def _system(case, seed):
    if case["kind"] in ("polymer_segment", "polymer_call", "gb_device"):
        return _polymer(case["atoms"], seed) if case["kind"] != "gb_device" else None
    if case["kind"] == "scpism":
        return _scpism_polymer(case["atoms"], seed)
    return _box(case["waters"], seed)


def _globule(atoms, seed):
    """Positions, charges and GB parameters of a compact molecule: a random
    subset of a jittered 2.4 A lattice in a ball."""
    rng = np.random.default_rng(seed)
    m = int(math.ceil((atoms * 2.2) ** (1.0 / 3.0))) + 2
    g = np.arange(m, dtype=np.float64) - 0.5 * (m - 1)
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    sites = sites[np.argsort((sites ** 2).sum(1) + 1e-9 * rng.random(len(sites)))[:atoms]]
    pos = 2.4 * sites[rng.permutation(atoms)] + rng.uniform(-0.3, 0.3, (atoms, 3))
    q = rng.uniform(-0.5, 0.5, atoms)
    q -= q.mean()
    return SimpleNamespace(pos=pos, charge=q * systems.SQRTCOULOMBCONSTANT,
                           gb_vdwr=rng.uniform(1.2, 1.9, atoms),
                           gb_scale=rng.choice([0.72, 0.79, 0.85, 0.96], atoms),
                           gb_offset=np.full(atoms, 0.09), gb_obc=OBC)


def _ensemble_waters(case, seed):
    """Water counts log-uniform in [least, most], the ends among them."""
    rng = np.random.default_rng(12345)  # the mix belongs to the case, the boxes to the seed
    w = np.exp(rng.uniform(math.log(case["least"]), math.log(case["most"]), case["boxes"]))
    w = np.round(w).astype(int)
    w[0], w[-1] = case["least"], case["most"]
    return [int(x) for x in w]


def _integrator(case, seed):
    if case.get("integrator", "langevin") == "leapfrog":
        return LeapfrogIntegrator(case["dt"])
    return LangevinLeapfrogIntegrator(case.get("dt", 1.0), temperature=300.0, gamma=5.0, seed=seed)


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    st = SimpleNamespace(case=case, kind=kind)
    if kind == "ensemble":
        members, st.integrator = [], _integrator(case, seed)
        for k, w in enumerate(_ensemble_waters(case, seed)):
            gs = GpuSystem(ctx, _box(w, seed * 1000 + k), "mixed")
            ff = ForceFactory(gs, RC)
            for line in _pme_lines(w):
                ff.make(line)
            st.integrator.run(gs, 5)  # every box on its own first, then together
            members.append(gs)
        st.ensemble = SystemEnsemble(members)
        st.ensemble.run(st.integrator, 66)  # off the lattice; the passes carry on from here
        return st
    if kind == "gb_device":
        s = _globule(case["atoms"], seed)
        st.n = case["atoms"]
        st.arrays = [torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda")
                     for a in (s.pos, s.charge, s.gb_vdwr, s.gb_scale, s.gb_offset)]
        st.forces = torch.zeros(3 * st.n, dtype=torch.float64, device="cuda")
        st.energy = torch.zeros(1, dtype=torch.float64, device="cuda")
        st.obc = (ctypes.c_double * 3)(*s.gb_obc)
        st.precision = _lib.PREC_MIXED if case["precision"] == "mixed" else _lib.PREC_DOUBLE
        return st
    sysm = _system(case, seed)
    precision = case.get("precision", "mixed")
    st.real = np.float32 if precision == "mixed" else np.float64
    st.pos, st.vel = np.ascontiguousarray(sysm.pos), np.ascontiguousarray(sysm.vel)
    st.gs = GpuSystem(ctx, sysm, precision)
    ff = ForceFactory(st.gs, RC)
    if kind == "call":
        lines = [_cutoff_line(case)]
    elif kind == "request" or (kind == "segment" and case["terms"] == "pme"):
        lines = _pme_lines(case["waters"])
    elif kind == "segment":
        lines = ["Bond", "Angle", _cutoff_line(SMALL)]
    elif kind == "polymer_segment":
        lines = GB_LINES + ALL_PAIRS + BONDED
    elif kind == "polymer_call":
        lines = GB_LINES + ["GBACEForce -algorithm NonbondedSimpleFull"] + ALL_PAIRS + BONDED
    else:
        lines = SCPISM_LINES
    st.force = [ff.make(line) for line in lines]
    st.integrator = _integrator(case, seed) if "steps" in case else None
    return st


# -------------------------------------------------------------------- run
def run(st):
    if st.kind == "ensemble":
        st.ensemble.run(st.integrator, st.case["steps"])
        return {"positions": [m.positions().astype(np.float32) for m in st.ensemble.members],
                "energies": np.array([m.energies()[0][:4] for m in st.ensemble.members],
                                     np.float32)}
    if st.kind == "gb_device":
        a = st.arrays
        _lib.check(_lib.load().pmgpu_gb_forces_noalloc(
            st.n, a[0].data_ptr(), a[1].data_ptr(), a[2].data_ptr(), a[3].data_ptr(),
            a[4].data_ptr(), None, st.obc, SOLUTE, SOLVENT, st.precision, st.forces.data_ptr(),
            st.energy.data_ptr(), torch.cuda.current_stream().cuda_stream))
        if st.precision == _lib.PREC_MIXED:
            return {"forces": st.forces.float().view(-1, 3), "energy": st.energy.float()}
        return {"forces": st.forces.view(-1, 3), "energy": st.energy}
    if st.kind in ("segment", "polymer_segment"):
        gs = st.gs
        gs.set_positions(st.pos)
        gs.set_velocities(st.vel)
        gs.set_step(0)
        st.integrator.run(gs, st.case["steps"])
        return {"positions": gs.positions().astype(st.real, copy=False),
                "velocities": gs.velocities().astype(st.real, copy=False),
                "energies": gs.energies()[0][:5].astype(st.real)}
    if st.kind == "request":
        gs = st.gs
        gs.set_positions(st.pos)
        e, v = gs.evaluate(virial=st.case["virial"])
        out = {"forces": gs.forces_total().astype(st.real, copy=False),
               "energies": e[:5].astype(st.real)}
        if v is not None:
            out["virial"] = v.astype(st.real, copy=False)
        return out
    # ProtoMol's evaluation of the force lines one after another
    forces, energies = np.zeros(st.pos.shape, st.real), ScalarStructure()
    virial = bool(st.case.get("virial"))
    for f in st.force:
        f.evaluate(st.pos, forces, energies, virial=virial)
    out = {"forces": forces, "energies": energies[:5].astype(st.real)}
    if virial:
        out["virial"] = energies[7:16].reshape(3, 3).astype(st.real)
    return out


# ------------------------------------------------------------------- work
def _water_work(waters, rc, steps, grid):
    n = 3 * waters
    pairs = n * 3 * WATER_DENSITY * 4.18879 * rc ** 3 / 2
    flops = 55.0 * pairs + 100.0 * n
    if grid:
        G = grid ** 3
        flops += n * ORDER ** 3 * 16.0 + 2 * 2.5 * G * math.log2(G) + 3.0 * G
    return 24.0 * n * 2, steps * flops


def work(case):
    kind = case["kind"]
    if kind in ("call", "request", "segment"):
        pme = kind == "request" or case.get("terms") == "pme"
        rc = RC if pme else case.get("rc", 8.0)
        b, f = _water_work(case["waters"], rc, case.get("steps", 1),
                           _water_grid(case["waters"]) if pme else 0)
        return {"bytes": b * (2 if kind == "segment" else 1), "flops": f}
    if kind == "ensemble":
        w = [_water_work(x, RC, case["steps"], _water_grid(x))
             for x in _ensemble_waters(case, 0)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    n = case["atoms"]
    pairs = n * (n - 1) / 2.0
    per = {"gb_device": 170.0, "scpism": 60.0}.get(kind, 225.0)
    return {"bytes": 24.0 * n * (4 if kind == "polymer_segment" else 2),
            "flops": case.get("steps", 1) * per * pairs}


# ------------------------------------------------------------------ exact
# The same quantities in 64 bits with plain torch: pair sums over every pair
# within the cutoff, smooth PME, bonded terms, GB by differentiation.
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, kind=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=kind, device=DEV)


class _Sum:
    """Forces, energies and virial being added up."""

    def __init__(self, n):
        self.f = torch.zeros(n, 3, dtype=torch.float64, device=DEV)
        self.e = torch.zeros(5, dtype=torch.float64, device=DEV)
        self.v = torch.zeros(3, 3, dtype=torch.float64, device=DEV)

    def pairs(self, i, j, d, f):
        """Pair force f over the distance: F_j += d f, F_i -= d f."""
        fd = d * f[:, None]
        self.f.index_add_(0, j, fd)
        self.f.index_add_(0, i, -fd)
        self.v += d.T @ fd

    def by_gradient(self, slot, i, j, d, energy):
        """Forces of an energy of the vectors d = x_j - x_i."""
        d = [x.detach().requires_grad_(True) for x in d]
        e = energy(*d)
        for a, b, x, g in zip(i, j, d, torch.autograd.grad(e, d)):
            self.f.index_add_(0, b, -g)
            self.f.index_add_(0, a, g)
            self.v -= x.detach().T @ g
        self.e[slot] += e.detach()


def _near(d, L):
    return d - L * torch.round(d / L) if L else d


def _pair_list(x, L, reach, images):
    """(i, j, whole-box shifts) of every i < j within reach, with every image
    when asked (box edges between the reach and twice it)."""
    n = x.shape[0]
    shifts = [(a, b, c) for a in (0, -1, 1) for b in (0, -1, 1) for c in (0, -1, 1)] \
        if images else [(0, 0, 0)]
    out = [[], [], []]
    rows = max(1, 30_000_000 // n)
    for r0 in range(0, n, rows):
        r1 = min(n, r0 + rows)
        d = x[None, :, :] - x[r0:r1, None, :]
        base = -torch.round(d / L) if L else torch.zeros_like(d)
        upper = torch.arange(n, device=DEV)[None, :] > torch.arange(r0, r1, device=DEV)[:, None]
        for s in shifts:
            w = base + torch.tensor(s, dtype=torch.float64, device=DEV)
            r2 = ((d + (L or 0.0) * w) ** 2).sum(-1)
            a, b = torch.nonzero(upper & (r2 < reach * reach), as_tuple=True)
            out[0].append(a + r0)
            out[1].append(b)
            out[2].append(w[a, b])
    return [torch.cat(o) for o in out]


def _switch(kind, r, on, rc):
    """Value and derivative over the distance."""
    one = torch.ones_like(r)
    if kind == "C2":
        t = (rc * rc - on * on) ** 3
        c = rc * rc - r * r
        w = rc * rc - 3 * on * on + 2 * r * r
        v, dv = c * c * w / t, 4 * (c * c - c * w) / t
        v, dv = torch.where(r < on, one, v), torch.where(r < on, 0 * one, dv)
    elif kind == "C1":
        v, dv = 1 - 1.5 * r / rc + 0.5 * (r / rc) ** 3, (-1.5 / rc + 1.5 * r * r / rc ** 3) / r
    else:  # Cn, n = 4
        t = (r - rc) / (on - rc)
        co = (126.0, -420.0, 540.0, -315.0, 70.0)
        v = sum(c * t ** (5 + k) for k, c in enumerate(co))
        dv = sum((5 + k) * c * t ** (4 + k) for k, c in enumerate(co)) / (on - rc) / r
        v, dv = torch.where(r < on, one, v), torch.where(r < on, 0 * one, dv)
    return torch.where(r > rc, 0 * one, v), torch.where(r > rc, 0 * one, dv)


class _Exact:
    """Force and energy sums of one molecular system at given positions."""

    def __init__(self, s):
        self.s, self.n = s, len(s.charge)
        self.q, self.m = _t(s.charge), _t(s.mass)
        self.L = float(s.box[0]) if s.periodic else 0.0
        ex = np.asarray(s.exclusions)
        self.full = _t(np.sort(ex[ex[:, 2] == 2][:, :2] @ [self.n, 1]), torch.int64)
        self.ex = [_t(ex[ex[:, 2] == 2][:, k], torch.int64) for k in (0, 1)]
        lj = np.asarray(s.lj)
        self.A, self.B, self.type = _t(lj[..., 0]), _t(lj[..., 1]), _t(s.type, torch.int64)
        self.list, self.at = None, 0

    def pairs(self, x, rc, images):
        """The pairs within rc: from a list with a margin, remade now and then."""
        margin = 3.0 if self.n > 3000 else 0.0
        if self.list is None or not margin or self.at % 15 == 0:
            i, j, w = _pair_list(x, self.L, rc + margin, images)
            k = torch.searchsorted(self.full, i * self.n + j).clamp_(max=max(0, len(self.full) - 1))
            minimal = (w == -torch.round((x[j] - x[i]) / self.L)).all(1) if self.L else None
            excluded = (self.full[k] == i * self.n + j) if len(self.full) else torch.zeros_like(i, dtype=torch.bool)
            if minimal is None:
                minimal = torch.ones_like(i, dtype=torch.bool)
            keep = ~(excluded & minimal)
            self.list = i[keep], j[keep], w[keep], minimal[keep]
        self.at += 1
        i, j, w, minimal = self.list
        d = x[j] - x[i] + self.L * w
        r = d.norm(dim=1)
        k = r <= rc
        return i[k], j[k], d[k], r[k], minimal[k]

    def lennard_jones(self, i, j, r):
        A, B = self.A[self.type[i], self.type[j]], self.B[self.type[i], self.type[j]]
        r6 = r ** -6
        return A * r6 * r6 - B * r6, (12 * A * r6 * r6 - 6 * B * r6) / (r * r)

    def switched(self, out, x, lj, co, on, rc, images):
        i, j, d, r, _ = self.pairs(x, rc, images)
        for slot, kind in ((LJ, lj), (COULOMB, co)):
            if slot == LJ:
                e, f = self.lennard_jones(i, j, r)
            else:
                e = self.q[i] * self.q[j] / r
                f = e / (r * r)
            v, dv = _switch(kind, r, on, rc)
            out.e[slot] += (e * v).sum()
            out.pairs(i, j, d, f * v - e * dv)

    def pme(self, out, x, grid):
        small = self.L < 2 * (RC + (3.0 if self.n > 3000 else 0.0))
        i, j, d, r, minimal = self.pairs(x, RC, small)
        e, f = self.lennard_jones(i, j, r)
        v, dv = _switch("C2", r, LJ_SWITCHON, RC)
        on = minimal.to(torch.float64)
        out.e[LJ] += (on * e * v).sum()
        f = on * (f * v - e * dv)
        # real space with the Abramowitz-Stegun 7.1.26 erfc of the reference
        t = 1 / (1 + 0.3275911 * ALPHA * r)
        ee = self.q[i] * self.q[j] * torch.exp(-(ALPHA * r) ** 2)
        e = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (
            -1.453152027 + t * 1.061405429)))) * ee / r
        out.e[COULOMB] += e.sum()
        out.pairs(i, j, d, f + (e + 2 * ALPHA / math.sqrt(math.pi) * ee) / (r * r))
        # excluded pairs and the self energy
        a, b = self.ex
        d = _near(x[b] - x[a], self.L)
        r = d.norm(dim=1)
        qq = self.q[a] * self.q[b]
        ee = torch.erf(ALPHA * r) / r
        out.e[COULOMB] -= (qq * ee).sum() + ALPHA / math.sqrt(math.pi) * (self.q ** 2).sum()
        out.pairs(a, b, d, qq * (2 * ALPHA / math.sqrt(math.pi) * torch.exp(-(ALPHA * r) ** 2)
                                 - ee) / (r * r))
        self.reciprocal(out, x, grid)

    def reciprocal(self, out, x, K):
        L, p = self.L, ORDER
        u = (x / L + 0.5) % 1.0 * K
        lo = torch.floor(u)
        fr = u - lo

        def spline(fr):
            m = [fr, 1 - fr]
            for o in range(3, p + 1):
                dm = [m[0]] + [m[k] - m[k - 1] for k in range(1, o - 1)] + [-m[-1]]
                m = [((fr + k) * (m[k] if k < o - 1 else 0)
                      + (o - fr - k) * (m[k - 1] if k else 0)) / (o - 1) for k in range(o)]
            return torch.stack(m, -1), torch.stack(dm, -1)

        th, dth = spline(fr)  # n, 3, p
        g = (lo.long()[..., None] - torch.arange(p, device=DEV)) % K
        at = ((g[:, 0, :, None, None] * K + g[:, 1, None, :, None]) * K + g[:, 2, None, None, :])
        w = torch.einsum("n,na,nb,nc->nabc", self.q, th[:, 0], th[:, 1], th[:, 2])
        Q = torch.zeros(K ** 3, dtype=torch.float64, device=DEV).index_add_(
            0, at.reshape(-1), w.reshape(-1)).view(K, K, K)
        mk = spline(torch.zeros(1, dtype=torch.float64, device=DEV))[0][0]
        k = torch.arange(K, dtype=torch.float64, device=DEV)
        arg = 2 * math.pi * k[:, None] * torch.arange(p - 1, device=DEV) / K
        mod = (mk[1:] * torch.cos(arg)).sum(1) ** 2 + (mk[1:] * torch.sin(arg)).sum(1) ** 2
        mod = torch.where(mod < 1e-7, 0.5 * (mod.roll(1) + mod.roll(-1)), mod)
        h = torch.where(k <= K // 2, k, k - K) / L
        hx, hy, hz = h[:, None, None], h[None, :, None], h[None, None, :]
        h2 = hx * hx + hy * hy + hz * hz
        h2[0, 0, 0] = 1.0
        G = torch.exp(-math.pi ** 2 * h2 / ALPHA ** 2) / (math.pi * L ** 3 * h2) / (
            mod[:, None, None] * mod[None, :, None] * mod[None, None, :])
        G[0, 0, 0] = 0.0
        S = torch.fft.fftn(Q)
        mode = 0.5 * G * (S.real ** 2 + S.imag ** 2)
        out.e[COULOMB] += mode.sum()
        c = 2 * (1 / h2 + math.pi ** 2 / ALPHA ** 2)
        hs = (hx, hy, hz)
        for a in range(3):
            out.v[a, a] += mode.sum()
            for b in range(3):
                out.v[a, b] -= (mode * c * hs[a] * hs[b]).sum()
        phi = torch.fft.ifftn(G * S).real.reshape(-1)[at] * float(K ** 3)
        for a in range(3):
            t = [dth[:, k] if k == a else th[:, k] for k in range(3)]
            out.f[:, a] -= self.q * K / L * torch.einsum("na,nb,nc,nabc->n", *t, phi)

    def bonded(self, out, x):
        s = self.s

        def vec(a, b):
            return _near(x[b] - x[a], self.L)

        b, p = _t(s.bonds, torch.int64), _t(s.bond_params)
        out.by_gradient(BOND, [b[:, 0]], [b[:, 1]], [vec(b[:, 0], b[:, 1])],
                        lambda d: (p[:, 0] * (d.norm(dim=1) - p[:, 1]) ** 2).sum())
        a, pa = _t(s.angles, torch.int64), _t(s.angle_params)

        def angle(u, w):
            th = torch.atan2(torch.linalg.cross(u, w).norm(dim=1), (u * w).sum(1))
            return (pa[:, 0] * (th - pa[:, 1]) ** 2).sum()

        out.by_gradient(ANGLE, [a[:, 1], a[:, 1]], [a[:, 0], a[:, 2]],
                        [vec(a[:, 1], a[:, 0]), vec(a[:, 1], a[:, 2])], angle)
        if getattr(s, "dihedrals", None) is None:
            return
        t, pt = _t(s.dihedrals, torch.int64), _t(s.dihedral_params)

        def torsion(u, v, w):
            m, k = torch.linalg.cross(u, v), torch.linalg.cross(v, w)
            phi = torch.atan2((torch.linalg.cross(m, k) * v).sum(1) / v.norm(dim=1),
                              (m * k).sum(1))
            return (pt[:, 0] * (1 + torch.cos(pt[:, 1] * phi + pt[:, 2]))).sum()

        out.by_gradient(DIHEDRAL, [t[:, 0], t[:, 1], t[:, 2]], [t[:, 1], t[:, 2], t[:, 3]],
                        [vec(t[:, k], t[:, k + 1]) for k in range(3)], torsion)

    def all_pairs(self, out, x):
        i, j, d, r, _ = self.pairs(x, 1e9, False)
        e, f = self.lennard_jones(i, j, r)
        c = self.q[i] * self.q[j] / r
        out.e[LJ] += e.sum()
        out.e[COULOMB] += c.sum()
        out.pairs(i, j, d, f + c / (r * r))

    def scpism(self, out, x):
        z, D = self.s.scpism, 80.0
        i, j, d, r, _ = self.pairs(x, 20.0, False)
        e, f = self.lennard_jones(i, j, r)
        v, dv = _switch("Cn", r, 8.0, 20.0)
        out.e[LJ] += (e * v).sum()
        out.pairs(i, j, d, f * v - e * dv)
        root = _t(z["scp_sqrtalpha"])
        aij, k = root[i] * root[j], (D - 1) / 2
        di = (1 + D) / (1 + k * torch.exp(-aij * r)) - 1
        e = self.q[i] * self.q[j] / (r * di)
        f = (aij * (1 + di) * (D - di) / (1 + D) / di + 1 / r) * e / r
        out.e[COULOMB] += (e * v).sum()
        out.pairs(i, j, d, f * v - e * dv)
        # Born radii and self energies of the pairs within 5 A
        near = r <= 5.0
        i, j, d = i[near], j[near], d[near]
        eta, C, g = _t(z["scp_eta"]), _t(z["scp_c"]), _t(z["scp_g"])
        hb, res = _t(z["scp_hbond"], torch.int64), _t(z["scp_residue"], torch.int64)
        name = _t(z["scp_name"], torch.int64)
        alpha, zeta = _t(z["scp_alpha"]), _t(z["scp_zeta"])

        def energy(d):
            r = d.norm(dim=1)
            fs = (1 - .0016 * r ** 4) ** 4
            R = zeta.clone()
            for a, b in ((i, j), (j, i)):
                polar = (hb[a] == 1) & (hb[b] == 2) & (res[a] != res[b])
                gp = torch.where((name[a] == 1) & (name[b] == 2), torch.full_like(r, -0.378), g[a])
                R = R.index_add(0, a, eta[a] * fs * torch.exp(-C[a] * r)
                                + torch.where(polar, gp * g[b] * fs * torch.exp(-0.8 * r), 0 * r))
            Ds = (1 + D) / (1 + k * torch.exp(-alpha * R)) - 1
            return (0.5 * self.q ** 2 / R * (1 / Ds - 1)).sum()

        out.by_gradient(COULOMB, [i], [j], [d], energy)

    def gb(self, out, x, ace):
        gb_sum(out, x, self.q, self.s, ace)


def gb_sum(out, x, q, s, ace, rows=None):
    """OBC generalized Born (and the ACE term) by differentiating the energy,
    a block of rows at a time."""
    n = len(q)
    rho, oi = _t(s.gb_vdwr), _t(s.gb_vdwr - s.gb_offset)
    so = _t(s.gb_scale) * oi
    rows = rows or max(1, 6_000_000 // n)
    blocks = [torch.arange(a, min(n, a + rows), device=DEV) for a in range(0, n, rows)]
    every = torch.arange(n, device=DEV)

    def distance(x, b):
        d = x[None] - x[b][:, None]
        return torch.sqrt((d * d).sum(-1) + (every[None] == b[:, None]))

    def burial(x, b):
        r, o, sj = distance(x, b), oi[b][:, None], so[None]
        a = (r - sj).abs()
        out_ = o >= r + sj
        Lo, U = torch.where(o > a, o.expand_as(a), a), r + sj
        Lo, U = torch.where(out_, torch.ones_like(r), Lo), torch.where(out_, torch.ones_like(r), U)
        term = 1 / Lo - 1 / U + r / 4 * (1 / U ** 2 - 1 / Lo ** 2) + torch.log(Lo / U) / (2 * r) \
            + sj * sj / (4 * r) * (1 / Lo ** 2 - 1 / U ** 2)
        term = term + torch.where(o < sj - r, 2 * (1 / o - 1 / Lo), 0 * r)
        return (term * (every[None] != b[:, None])).sum(1)

    with torch.no_grad():
        I = torch.cat([burial(x, b) for b in blocks])
    I.requires_grad_(True)
    psi = 0.5 * I * oi
    R = 1 / (1 / oi - torch.tanh(OBC[0] * psi - OBC[1] * psi ** 2 + OBC[2] * psi ** 3) / rho)
    tau = 1 / SOLUTE - 1 / SOLVENT
    own = (-0.5 * q * q / R * tau).sum()
    if ace:
        own = own + (4 * 3.14169 * (2.26 / 418.4) * (rho + 1.4) ** 2 * (rho / R) ** 6).sum()
    Rf = R.detach().requires_grad_(True)
    xf = x.detach().requires_grad_(True)
    e = own.detach().clone()
    for b in blocks:
        r2 = distance(xf, b) ** 2
        bb = Rf[b][:, None] * Rf[None]
        eb = (-0.5 * tau * q[b][:, None] * q[None] / torch.sqrt(r2 + bb * torch.exp(-r2 / (4 * bb)))
              * (every[None] != b[:, None])).sum()
        eb.backward()
        e += eb.detach()
    gI = torch.autograd.grad(own + (R * Rf.grad).sum(), I)[0]
    for b in blocks:
        (burial(xf, b) * gI[b]).sum().backward()
    out.f -= xf.grad
    out.e[COULOMB] += e


def _evaluate(case, ex, x, lines):
    out = _Sum(ex.n)
    if lines == "pme":
        ex.bonded(out, x)
        ex.pme(out, x, _water_grid(case["waters"]))
    elif lines == "cutoff":
        if case["kind"] != "call":
            ex.bonded(out, x)
            case = SMALL
        lj, co = (k.split()[0] for k in SWITCHES[case["switches"]])
        ex.switched(out, x, lj, co, case["on"], case["rc"],
                    case["algorithm"] == "NonbondedFull" and ex.L < 2 * (case["rc"] + 3.0))
    elif lines == "scpism":
        ex.scpism(out, x)
    else:
        ex.bonded(out, x)
        ex.all_pairs(out, x)
        ex.gb(out, x, lines == "gbace")
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "polymer_segment") or case.get("integrator") == "langevin":
        return None  # the noise is the framework's own sequence of random numbers
    if kind == "gb_device":
        s, out = _globule(case["atoms"], seed), _Sum(case["atoms"])
        gb_sum(out, _t(s.pos), _t(s.charge), s, False)
        return {"forces": out.f, "energy": out.e[COULOMB:COULOMB + 1]}
    s = _system(case, seed)
    if kind == "segment" and case["steps"] * len(s.charge) > 400_000 and DEV == "cpu":
        return None
    ex, x = _Exact(s), _t(s.pos)
    lines = "pme" if kind == "request" else case.get("terms") or {
        "call": "cutoff", "scpism": "scpism", "polymer_call": "gbace"}[kind]
    if kind == "segment":
        # leapfrog: half a kick, then drifts and kicks, half a kick
        h, v = case["dt"] * 0.02045482828087295, _t(s.vel)
        out = _evaluate(case, ex, x, lines)
        for k in range(case["steps"]):
            v = v + out.f * ((0.5 if k == 0 else 1.0) * h) / ex.m[:, None]
            x = x + h * v
            out = _evaluate(case, ex, x, lines)
        v = v + out.f * (0.5 * h) / ex.m[:, None]
        return {"positions": x, "velocities": v, "energies": out.e}
    out = _evaluate(case, ex, x, lines)
    got = {"forces": out.f, "energies": out.e}
    if case.get("virial"):
        got["virial"] = out.v
    return got
