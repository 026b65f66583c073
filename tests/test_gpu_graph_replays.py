"""That repeated work is replayed: graph launches rise from the third call of
a kind of evaluation and from the third run (the inner steps: the first), for
every kind of force, and stay at zero where the work is eager.  Without this
a capture that fails would leave the tests that compare replayed with eager
results comparing eager with eager."""
import numpy as np
import pytest

from protomol_b200 import (ForceFactory, GpuSystem, LangevinLeapfrogIntegrator, ScalarStructure,
                           systems)

pytestmark = pytest.mark.gpu

KINDS = {
    "cutoff": ["Bond", "Angle",
               "LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction Cn -n 4 "
               "-switchon 6 -cutoff 8 -switchingFunction C1 -cutoff 8 -cutoff 8"],
    "pme": ["LennardJones -algorithm NonbondedCutoff -switchingFunction C2 -switchon 6 -cutoff 8 "
            "-cutoff 8", "Coulomb -algorithm PMEwald -alpha 0.35 -cutoff 8 -order 4 "
            "-gridsize 20 20 20"],
    "pme_cufft": ["Coulomb -algorithm PMEwald -alpha 0.35 -cutoff 8 -order 4 "
                  "-gridsize 22 22 22"],
    "gb": ["LennardJones Coulomb -algorithm NonbondedSimpleFull",
           "GBForce -algorithm NonbondedSimpleFull -soluteDielec 1.0 -solventDielec 78.5",
           "GBACEForce -algorithm NonbondedSimpleFull"],
}


def _system(ctx, kind, precision):
    s = systems.gb_polymer(150, seed=3) if kind == "gb" else \
        systems.tip3p_box(216, 18.64, seed=4, jitter=0.2)
    gs = GpuSystem(ctx, s, precision)
    ff = ForceFactory(gs, 8.0)
    return s, gs, [ff.make(line) for line in KINDS[kind]]


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_evaluations_replay(ctx, kind, precision):
    s, gs, forces = _system(ctx, kind, precision)
    forces[-1].evaluate(s.pos, np.zeros_like(s.pos), None)  # the list of the force is built
    for call in (lambda: gs.evaluate(), lambda: gs.evaluate(virial=True), gs.evaluate_forces,
                 lambda: forces[-1].evaluate(s.pos, np.zeros_like(s.pos), ScalarStructure())):
        call()  # (builds the lists of the other forces, another kind)
        call()
        before = gs.graph_replays()
        for k in range(4):
            call()
        assert gs.graph_replays() - before >= 3
    gs.profile(enable=True)
    before = gs.graph_replays()
    for _ in range(4):
        gs.evaluate()
    assert gs.graph_replays() == before
    gs.close()


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_runs_replay(ctx, kind, precision):
    s, gs, _ = _system(ctx, kind, precision)
    it = LangevinLeapfrogIntegrator(0.5, 300.0, 5.0, seed=3)
    got = []
    for _ in range(4):
        before = gs.graph_replays()
        it.run(gs, 13)  # the first step, ten, one, the last
        got.append(gs.graph_replays() - before)
    assert got == [2, 2, 4, 4]
    gs.close()
    s, gs, _ = _system(ctx, kind, precision)
    gs.profile(enable=True)
    for _ in range(3):
        it.run(gs, 13)
    assert gs.graph_replays() == 0
    gs.close()
