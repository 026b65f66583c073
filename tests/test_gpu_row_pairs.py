"""The FP64 all-pairs passes with a warp (or several) per atom: sizes around
the warp and the split rule's steps, double-precision GB + ACE + all-pairs
LJ / Coulomb on polymers, against the FP64 oracle.  Tolerance 1e-8 RMS
relative on the forces, the repository's bound of its double-precision
tests (fixed-point force resolution)."""
import numpy as np
import pytest

import fixtures as F
import oracle
from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 31, 33, 64, 149, 297, 593, 1185])
def test_double_all_pairs_vs_oracle(ctx, n):
    s = systems.gb_polymer(n, seed=3)
    gs = GpuSystem(ctx, s, "double")
    ff = ForceFactory(gs)
    o = oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                      excl=s.exclusions, periodic=False, box=s.box)
    o.gb_vdwr, o.gb_scale, o.gb_offset, o.gb_obc = s.gb_vdwr, s.gb_scale, s.gb_offset, s.gb_obc
    o.water = s.water
    gb = oracle.gb_force(o, 1.0, 78.5)
    cases = [("GBForce -algorithm NonbondedSimpleFull -soluteDielec 1.0 -solventDielec 78.5",
              gb[0], gb[1], 0),
             ("LennardJones -algorithm NonbondedSimpleFull",
              oracle.simplefull_force(o, "LennardJones")[0], None, 1),
             ("Coulomb -algorithm NonbondedSimpleFull", oracle.simplefull_force(o, "Coulomb")[0],
              None, 0)]
    for line, fo, eo, slot in cases:
        force = ff.make(line)
        f, e = np.zeros_like(s.pos), ScalarStructure()
        force.evaluate(s.pos, f, e)
        assert F.rms_rel(f, fo) <= 1e-8 or np.abs(f - fo).max() <= 4 * 2.0 ** -32, (line, n)
        if eo is not None:
            assert abs(e[slot] - eo) <= 1e-8 * max(1.0, abs(eo))
        force.set_enabled(False)
    gs.close()
