"""How a cluster's tiles are divided over warps must not be seen in results.
Batched launches give a warp several of the shares a box alone has a warp
each for, and still leave the same bits (boxes below twice the cutoff take
the tile kernel); in double precision the division follows the system's size
and only rounds differently."""
import numpy as np
import pytest

import fixtures as F
import oracle
from protomol_b200 import ForceFactory, GpuSystem, LeapfrogIntegrator, ScalarStructure, systems
from protomol_b200.engine import SystemEnsemble

pytestmark = pytest.mark.gpu

CUT = ("LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon 7 "
       "-cutoff 8 -switchingFunction C1 -cutoff 8 -cutoff 8")


def _box(ctx, waters, seed):
    s = systems.water_box_for_density(waters, 0.0334, seed, jitter=0.2)
    gs = GpuSystem(ctx, s, "mixed")
    ff = ForceFactory(gs, 9.0)
    for line in ["Bond", "Angle", "LennardJones -algorithm NonbondedCutoff -switchingFunction C2 "
                 "-switchon 8 -cutoff 9 -cutoff 9", "Coulomb -algorithm PMEwald -alpha 0.35 "
                 "-cutoff 9 -order 4 -gridsize 16 16 16"]:
        ff.make(line)
    return gs


@pytest.mark.parametrize("count", [12, 40, 110])
def test_members_of_a_batch_as_alone(ctx, count):
    """12, 40 and 110 boxes of 60 to 100 waters: groups of two, four and
    eight shares a warp."""
    waters = [60 + 10 * (k % 5) for k in range(count)]
    it = LeapfrogIntegrator(1.0)
    members = [_box(ctx, w, k) for k, w in enumerate(waters)]
    ens = SystemEnsemble(members)
    for n in (5, 7):
        ens.run(it, n)
    got = [(gs.positions(), gs.velocities(), gs.energies()[0]) for gs in members]
    ens.close()
    for gs in members:
        gs.close()
    for k in (0, 1, 4, count - 1):
        gs = _box(ctx, waters[k], k)
        one = SystemEnsemble([gs])
        for n in (5, 7):
            one.run(it, n)
        for a, b in zip((gs.positions(), gs.velocities(), gs.energies()[0]), got[k]):
            assert np.array_equal(a, b)
        one.close()
        gs.close()


@pytest.mark.parametrize("waters", [1, 30, 216, 400, 700, 1300, 2600, 6000])
def test_double_at_every_division(ctx, waters):
    s = systems.water_box_for_density(max(waters, 150), 0.0334, 7, jitter=0.2)
    if waters < 150:  # a few molecules in a box that holds twice the cutoff
        s = systems.tip3p_box(waters, 17.0, seed=7, jitter=0.2)
    gs = GpuSystem(ctx, s, "double")
    force = ForceFactory(gs, 8.0).make(CUT)
    f, e = np.zeros_like(s.pos), ScalarStructure()
    force.evaluate(s.pos, f, e, virial=True)
    gs.close()
    o = oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                      excl=s.exclusions, periodic=True, box=s.box)
    fo, eo, vo = oracle.cutoff_force(o, 8.0, 8.0, [
        ("LennardJones", oracle.Switch("C2", 8.0, 7.0)), ("Coulomb", oracle.Switch("C1", 8.0))])
    assert F.rms_rel(f, fo) <= 1e-8 or np.abs(f - fo).max() <= 4 * 2.0 ** -32
    assert abs(e[0] - eo["coulomb"]) <= 1e-8 * max(1.0, abs(eo["coulomb"]))
    assert abs(e[1] - eo["lj"]) <= 1e-8 * max(1.0, abs(eo["lj"]))
    assert np.abs(e[7:16] - np.ravel(vo)).max() <= 1e-8 * max(1.0, np.abs(vo).max())


@pytest.mark.parametrize("waters,rc,splits", [(600, 9.0, 6), (1667, 9.0, 3), (1667, 12.0, 6),
                                              (2600, 9.0, 2), (2600, 12.0, 4), (5000, 12.0, 2)])
def test_force_kernel_at_long_cutoffs(ctx, waters, rc, splits):
    """The force-only kernel's division grows with the cutoff; FP32 forces
    against the oracle (1e-5 relative, the repository's mixed-precision bound)."""
    s = systems.water_box_for_density(waters, 0.0334, 7, jitter=0.2)
    gs = GpuSystem(ctx, s, "mixed")
    force = ForceFactory(gs, rc).make(
        f"LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon "
        f"{rc - 1} -cutoff {rc} -switchingFunction C1 -cutoff {rc} -cutoff {rc}")
    f = np.zeros_like(s.pos)
    force.evaluate(s.pos, f, None)
    one = SystemEnsemble([gs])
    assert one.member(0)[1] == splits
    one.close()
    gs.close()
    o = oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                      excl=s.exclusions, periodic=True, box=s.box)
    fo, _, _ = oracle.cutoff_force(o, rc, rc, [
        ("LennardJones", oracle.Switch("C2", rc, rc - 1)), ("Coulomb", oracle.Switch("C1", rc))])
    assert F.rms_rel(f, fo) <= 1e-5
