"""Repeated evaluations: the third and later calls of a kind replay captured
launches.  Every one must return the bits of the first (eager) calls' sums
(fixed point, order independent), for other positions too, and everything
that changes what an evaluation does must reach it: new positions, a grown
list, forces switched off and on or added, and positions that are refused."""
import numpy as np
import pytest

from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

pytestmark = pytest.mark.gpu

CUT = ("LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon 6 "
       "-cutoff 8 -switchingFunction C1 -cutoff 8 -cutoff 8")
RADII = 8.0


def _make(ctx, kind, precision="mixed"):
    if kind == "polymer":
        s = systems.gb_polymer(150, seed=3)
        line = "Coulomb -algorithm NonbondedSimpleFull"
    else:
        s = systems.tip3p_box(150, 18.0, seed=4, jitter=0.2)
        line = CUT
    gs = GpuSystem(ctx, s, precision)
    return s, gs, ForceFactory(gs, RADII).make(line)


def _call(force, pos, mode):
    f = np.full(pos.shape, 0.25)
    e = None if mode == "forces" else ScalarStructure()
    force.evaluate(pos, f, e, virial=mode == "virial")
    return f, e


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("mode", ["forces", "energies", "virial"])
@pytest.mark.parametrize("kind", ["water", "polymer"])
def test_replayed_equals_eager(ctx, kind, mode, precision):
    s, gs, force = _make(ctx, kind, precision)
    rng = np.random.default_rng(5)
    there = s.pos + rng.normal(size=s.pos.shape) * 0.05
    eager = [_call(force, p, mode) for p in (s.pos, there)]  # the two eager calls
    if kind == "water" and mode == "forces":  # the other kinds' graphs live beside it
        for _ in range(4):
            _call(force, s.pos, "energies")
    for k in (0, 1, 1, 0, 1, 0):
        f, e = _call(force, (s.pos, there)[k], mode)
        assert np.array_equal(f, eager[k][0])
        assert e is None or np.array_equal(e, eager[k][1])
    gs.close()


def test_whole_system_follows_its_forces(ctx):
    s, gs, force = _make(ctx, "water")
    for _ in range(4):
        gs.evaluate()
    one = gs.forces_total().copy()
    force.set_enabled(False)
    for _ in range(4):
        gs.evaluate()
    assert not gs.forces_total().any()
    force.set_enabled(True)
    bonded = ForceFactory(gs).make("Bond")  # added to a system that replays
    for k in range(4):
        gs.evaluate()
        if k == 0:
            both = gs.forces_total().copy()
        assert np.array_equal(gs.forces_total(), both)
    bonded.set_enabled(False)
    for _ in range(4):
        gs.evaluate()
        assert np.array_equal(gs.forces_total(), one)
    # positions that went to the device by themselves
    gs.set_positions(s.pos + 0.01 * np.arange(3))
    gs.evaluate()
    moved = gs.forces_total()
    fresh = GpuSystem(ctx, s, "mixed")
    ForceFactory(fresh, RADII).make(CUT)
    fresh.evaluate()
    fresh.set_positions(s.pos + 0.01 * np.arange(3))
    fresh.evaluate()
    assert np.array_equal(moved, fresh.forces_total())
    fresh.close()
    gs.close()


def test_list_growth_after_capture(ctx):
    """Molecules moved together fill the list's rows beyond what the replayed
    calls' launches were made for; such a call runs again with larger ones."""
    s, gs, force = _make(ctx, "water")
    gs.set_list_capacity(4)
    for _ in range(4):
        want = _call(force, s.pos, "energies")
    centre = np.repeat(s.pos[::3], 3, axis=0)
    tight = s.pos - 0.2 * centre
    got = [_call(force, tight, "energies") for _ in range(4)]
    _, other_gs, other = _make(ctx, "water")
    ref = _call(other, tight, "energies")
    for f, e in got:
        assert np.array_equal(f, ref[0]) and np.array_equal(e, ref[1])
    back = _call(force, s.pos, "energies")
    assert np.array_equal(back[0], want[0]) and np.array_equal(back[1], want[1])
    other_gs.close()
    gs.close()


def test_refused_positions_after_capture(ctx):
    s, gs, force = _make(ctx, "water")
    for _ in range(4):
        want = _call(force, s.pos, "energies")
    bad = s.pos.copy()
    bad[7, 1] = np.nan
    with pytest.raises(Exception):
        _call(force, bad, "energies")
    got = _call(force, s.pos, "energies")
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    gs.close()
