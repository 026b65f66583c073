"""Runs whose every part is replayed: from the third run with an integrator
on, the first and the last step (energies, closing kick) come from captured
launches like the inner ones.  Each run must leave the bits of the eager
one (profiling on forces the eager path), for runs of 2 steps up to several
chunks, and follow what happens between runs: an evaluation, new positions,
another integrator, a list that grows, a force switched off."""
import numpy as np
import pytest

from protomol_b200 import (ForceFactory, GpuSystem, LangevinLeapfrogIntegrator,
                           LeapfrogIntegrator, ScalarStructure, systems)

pytestmark = pytest.mark.gpu

CUT = ("LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon 6 "
       "-cutoff 8 -switchingFunction C1 -cutoff 8 -cutoff 8")


def _system(ctx, kind, precision, eager):
    if kind == "polymer":
        s = systems.gb_polymer(150, seed=3)
        lines = ["Bond", "Angle", "LennardJones Coulomb -algorithm NonbondedSimpleFull",
                 "GBForce -algorithm NonbondedSimpleFull -soluteDielec 1.0 -solventDielec 78.5"]
    else:
        s = systems.tip3p_box(150, 18.0, seed=4, jitter=0.2)
        lines = ["Bond", "Angle", CUT]
    gs = GpuSystem(ctx, s, precision)
    ff = ForceFactory(gs, 8.0)
    forces = [ff.make(line) for line in lines]
    gs.profile(enable=eager)
    return s, gs, forces


def _state(gs):
    return gs.positions(), gs.velocities(), gs.energies()[0], gs.forces_total()


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("kind", ["water", "polymer"])
@pytest.mark.parametrize("langevin", [True, False])
def test_replayed_runs_equal_eager_runs(ctx, kind, precision, langevin):
    out = []
    for eager in (True, False):
        s, gs, forces = _system(ctx, kind, precision, eager)
        it = LangevinLeapfrogIntegrator(0.5, 300.0, 5.0, seed=3) if langevin else \
            LeapfrogIntegrator(0.5)
        got = []
        for n in (2, 2, 3, 2, 13, 1, 25, 2):
            it.run(gs, n)
            got.append(_state(gs))
        e = ScalarStructure()
        forces[2].evaluate(s.pos, np.zeros_like(s.pos), e)  # other positions, one force
        it.run(gs, 4)
        got.append(_state(gs))
        gs.set_positions(s.pos)
        for n in (3, 3):
            it.run(gs, n)
            got.append(_state(gs))
        LeapfrogIntegrator(0.25).run(gs, 12)
        it.run(gs, 12)
        got.append(_state(gs))
        if kind == "water":
            gs.set_list_capacity(1)  # overflows on the next build
        it.run(gs, 12)
        got.append(_state(gs))
        forces[2].set_enabled(False)
        for n in (2, 2, 2, 2):
            it.run(gs, n)
        got.append(_state(gs))
        out.append(got)
        gs.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
