"""Every FP64 all-pairs pass with a warp (or several) per atom, through its
force line, at sizes around a warp and the split rule's steps and with idle
warps in the last block: plain and switched LJ and Coulomb, SCPISM, the Born
lines and the ACE term, forces, energies and virial against the FP64 oracle
(tolerances of the repository's double-precision tests: 1e-8 relative, or
four units of the 2^-32 force resolution).  The pair forces are internal, so
the virial also has to be the first moment of the forces."""
import numpy as np
import pytest

import fixtures as F
import oracle
from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

pytestmark = pytest.mark.gpu

TOL, UNIT = 1e-8, 2.0 ** -32
C2 = ("-switchingFunction C2 -switchon 15 -cutoff 25", oracle.Switch("C2", 25.0, 15.0))
CN = ("-switchingFunction Cn -n 4 -switchon 8 -cutoff 20",
      oracle.Switch("Cn", 20.0, 8.0, 0.0, 4.0))
C1 = ("-switchingFunction C1 -cutoff 30", oracle.Switch("C1", 30.0))
LJ, COUL = "LennardJones", "Coulomb"


def _polymer(n):
    s = systems.gb_polymer(n, seed=n + 1)
    rng = np.random.default_rng([n, 1])
    hb = np.where(np.arange(n) % 12 == 4, 1, np.where(np.arange(n) % 12 == 9, 2, 0))
    root = rng.uniform(0.674, 0.775, n)
    s.scpism = dict(scp_sqrtalpha=root, scp_alpha=root * root,
                    scp_zeta=rng.uniform(1.4, 2.0, n), scp_eta=rng.uniform(0.023, 0.067, n),
                    scp_c=rng.uniform(0.22, 0.8, n),
                    scp_g=np.where(hb > 0, rng.uniform(0.47, 1.4, n), 0.47),
                    scp_hbond=hb.astype(np.int32),
                    scp_residue=(np.arange(n) // 16).astype(np.int32),
                    scp_name=np.where(np.arange(n) % 48 == 4, 1,
                                      np.where(hb == 2, 2, 0)).astype(np.int32))
    o = oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                      excl=s.exclusions, periodic=False, box=s.box, water=s.water,
                      gb_vdwr=s.gb_vdwr, gb_scale=s.gb_scale, gb_offset=s.gb_offset,
                      gb_obc=s.gb_obc, scpism=s.scpism)
    return s, o


def _pairs(o, terms):
    f, e, v = oracle.simplefull_force_n(o, terms)
    return f, e, v


def _plain(o, names):
    parts = [oracle.simplefull_force(o, name) for name in names]
    return (sum(p[0] for p in parts),
            {k: sum(p[1][k] for p in parts) for k in ("coulomb", "lj")}, sum(p[2] for p in parts))


def _born(o):
    f, e, _ = oracle.born_force(o, 3, 5.0, 3, 5.0)
    return f, {"coulomb": e, "lj": 0.0}, None


def _gb(o):
    f, e, _ = oracle.gb_force(o, 1.0, 78.5)
    return f, {"coulomb": e, "lj": 0.0}, None


def _ace(o):
    f, e = oracle.gbace_force(o)
    return f, {"coulomb": e, "lj": 0.0}, None


SIMPLE = "-algorithm NonbondedSimpleFull"
SCP = "-algorithm NonbondedCutoff"
LINES = {
    "lj": ([f"{LJ} {SIMPLE}"], lambda o: _plain(o, [LJ])),
    "coulomb": ([f"{COUL} {SIMPLE}"], lambda o: _plain(o, [COUL])),
    "lj+coulomb": ([f"{LJ} {COUL} {SIMPLE}"], lambda o: _plain(o, [LJ, COUL])),
    "switched": ([f"{LJ} {COUL} {SIMPLE} {C2[0]} {C1[0]}"],
                 lambda o: _pairs(o, [(LJ, C2[1]), (COUL, C1[1])])),
    "one switch": ([f"{LJ} {COUL} {SIMPLE} {CN[0]} {CN[0]}"],
                   lambda o: _pairs(o, [(LJ, CN[1]), (COUL, CN[1])])),
    "scpism": ([f"{LJ} CoulombSCPISM {SCP} {CN[0]} {CN[0]} -cutoff 20"],
               lambda o: oracle.scpism_pair_force(o, [(LJ, CN[1]), ("CoulombSCPISM", CN[1])])),
    "born": ([f"{name} {SCP} -switchingFunction Cutoff -bornswitch 3 -cutoff 5 -cutoff 5"
              for name in ("BornRadii", "BornSelf")], _born),
    "gb": ([f"GBForce {SIMPLE} -soluteDielec 1.0 -solventDielec 78.5"], _gb),
    "ace": ([f"GBACEForce {SIMPLE}"], _ace),
}


@pytest.mark.parametrize("line", sorted(LINES))
@pytest.mark.parametrize("n", [2, 5, 31, 33, 64, 149, 297, 593, 1185, 2400])
def test_row_line(ctx, n, line):
    s, o = _polymer(n)
    text, reference = LINES[line]
    fo, eo, vo = reference(o)
    gs = GpuSystem(ctx, s, "double")
    ff = ForceFactory(gs)
    force = [ff.make(t) for t in text][-1]
    f, e = np.zeros_like(s.pos), ScalarStructure()
    force.evaluate(s.pos, f, e, virial=line not in ("gb", "ace"))  # (GB has none)
    f2, e2 = np.zeros_like(s.pos), ScalarStructure()
    force.evaluate(s.pos, f2, e2)  # without the virial: the same launches otherwise
    f3 = np.zeros_like(s.pos)
    force.evaluate(s.pos, f3, None)
    gs.close()
    assert np.array_equal(f, f2) and np.array_equal(f, f3)
    assert np.array_equal(e[:7], e2[:7])
    assert F.rms_rel(f, fo) <= TOL or np.abs(f - fo).max() <= 4 * UNIT
    assert abs(e[0] - eo["coulomb"]) <= TOL * max(1.0, abs(eo["coulomb"]))
    assert abs(e[1] - eo["lj"]) <= TOL * max(1.0, abs(eo["lj"]))
    if line in ("gb", "ace"):
        return
    v = np.asarray(e[7:16]).reshape(3, 3)
    moment = s.pos.T @ fo
    scale = max(1.0, np.abs(moment).max())
    assert np.abs(v - moment).max() <= TOL * scale
    if vo is not None:
        assert np.abs(v - vo).max() <= TOL * scale
