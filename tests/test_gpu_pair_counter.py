"""Counting accepted pairs must not change what is computed: the force-only
kernels (with an Ewald table or without, LJ parameters in shared memory or
read per pair) give the same bits with the counter on and off, a Langevin
run (whose steps take their two half kicks one by one) split into several
calls under counting gives the unsplit run's trajectory, and
the force-only count is the energy pass's count and the pair set's size."""
import numpy as np
import pytest

from protomol_b200 import ForceFactory, GpuSystem, LangevinLeapfrogIntegrator, systems

pytestmark = pytest.mark.gpu

LJ = "LennardJones -algorithm NonbondedCutoff -switchingFunction C2 -switchon 7 -cutoff 8 -cutoff 8"
PME = "Coulomb -algorithm PMEwald -alpha 0.35 -cutoff 8 -order 4 -gridsize 20 20 20"
CUT = ("LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon 7 "
       "-cutoff 8 -switchingFunction C1 -cutoff 8 -cutoff 8")


def _system(ctx, types, lines):
    s = systems.tip3p_box(216, 18.64, seed=5, jitter=0.2)
    if types > 2:  # as many LJ types, cut from the two of the water
        t = np.arange(types) % 2
        s.lj = np.ascontiguousarray(np.asarray(s.lj).reshape(2, 2, -1)[t][:, t])
        s.type = (s.type + 2 * (np.arange(len(s.type)) % (types // 2))).astype(np.int32)
    gs = GpuSystem(ctx, s, "mixed")
    ff = ForceFactory(gs, 8.0)
    return s, gs, [ff.make(line) for line in ["Bond", "Angle"] + lines][-1]


def _count(gs, on):
    assert gs.lib.pmgpu_set_count_pairs(gs.h, int(on)) == 0


@pytest.mark.parametrize("types", [2, 20])
@pytest.mark.parametrize("lines", [[LJ, PME], [CUT]], ids=["pme", "cutoff"])
def test_counting_leaves_the_forces(ctx, types, lines):
    s, gs, force = _system(ctx, types, lines)
    off = gs.evaluate_forces()
    _count(gs, True)
    on = gs.evaluate_forces()
    pairs = force.stats()["pairs_in_cutoff"]
    assert np.array_equal(on, off)
    gs.evaluate()  # energies and forces
    assert np.array_equal(gs.forces_total(), off)
    assert force.stats()["pairs_in_cutoff"] == pairs == len(force.pair_set(1 << 20))
    gs.close()


@pytest.mark.parametrize("types", [2, 20])
def test_split_run_under_counting(ctx, types):
    out = []
    for count, parts in ((0, (20,)), (1, (20,)), (1, (7, 13)), (1, (2, 5, 13))):
        s, gs, _ = _system(ctx, types, [LJ, PME])
        _count(gs, count)
        for n in parts:
            LangevinLeapfrogIntegrator(0.5, 300.0, 5.0, seed=3).run(gs, n)
        out.append((gs.positions(), gs.velocities(), gs.energies()[0]))
        gs.close()
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)
