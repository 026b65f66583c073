"""The list build's candidate groups: boxes whose rows end in partly filled
groups of eight candidates, molecules spread over clusters (exclusions and
scaled 1-4 pairs between them), boxes below twice the cutoff (image shells)
and long rows, as pair sets and forces against the FP64 oracle.  The pair set
must be exact; forces within the repository's mixed-precision bound 1e-5.
The chains' random positions nearly overlap: their forces reach 1e11, where
one pair's FP32 rounding is beyond that bound for any list, so a chain is
its pair set alone."""
import numpy as np
import pytest

import fixtures as F
import oracle
from protomol_b200 import ForceFactory, GpuSystem, LeapfrogIntegrator, systems

pytestmark = pytest.mark.gpu

LINE = ("LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C2 -switchon {on} "
        "-cutoff {rc} -switchingFunction C2 -switchon {on} -cutoff {rc} -cutoff {rc}")


def _chain_box(n, edge, seed):
    """A polymer wrapped into a periodic box: bonded neighbours in several
    clusters and images, full and modified exclusions."""
    s = systems.gb_polymer(n, seed)
    s.periodic = True
    s.box = np.array([edge, 0, 0, 0, edge, 0, 0, 0, edge, 0, 0, 0], float)
    s.pos = np.random.default_rng(seed).uniform(-0.5 * edge, 0.5 * edge, (n, 3))
    return s


@pytest.mark.parametrize("kind,n,edge,rc", [
    ("water", 1, 12.0, 8.0), ("water", 2, 12.0, 8.0), ("water", 11, 12.0, 8.0),
    ("water", 90, 13.9, 8.0), ("water", 333, 21.5, 9.0), ("water", 500, 24.6, 11.5),
    ("chain", 37, 14.0, 6.0), ("chain", 400, 20.0, 8.0), ("chain", 900, 26.0, 5.0)])
def test_pair_set_and_forces(ctx, kind, n, edge, rc):
    s = systems.tip3p_box(n, edge, seed=4, jitter=0.2) if kind == "water" else \
        _chain_box(n, edge, 4)
    gs = GpuSystem(ctx, s, "mixed")
    force = ForceFactory(gs, rc).make(LINE.format(on=rc - 1, rc=rc))
    o = oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                      excl=s.exclusions, periodic=True, box=s.box)
    got = {(int(a), int(b)) for a, b in force.pair_set(1 << 20)}
    # the minimal image within the cutoff, less the full exclusions
    d = s.pos[None] - s.pos[:, None]
    d -= edge * np.rint(d / edge)
    i, j = np.nonzero(np.triu((d ** 2).sum(-1) <= rc * rc, 1))
    full = {(min(a, b), max(a, b)) for a, b, c in s.exclusions if c == 2}
    assert got == {(int(a), int(b)) for a, b in zip(i, j)} - full
    if kind == "chain":
        gs.close()
        return
    sw = oracle.Switch("C2", rc, rc - 1)
    fo, _, _ = oracle.cutoff_force(o, rc, rc, [("LennardJones", sw), ("Coulomb", sw)])
    for energies in (None, np.zeros(36)):
        f = np.zeros_like(s.pos)
        force.evaluate(s.pos, f, energies)
        assert F.rms_rel(f, fo) <= 1e-5 or np.abs(f - fo).max() <= 4 * 2.0 ** -32
    gs.close()


def test_column_overflow_in_recycled_memory(ctx):
    """A first build that drops atoms (column buckets of 32) in memory another
    system left full of other values: the dropped atoms have no slot, and the
    repeated segment equals the one that never overflowed."""
    big = systems.tip3p_box(4000, 49.5, seed=5, jitter=0.2)
    out = []
    for cap in (None, 32, 32):
        other = GpuSystem(ctx, big, "mixed")
        ForceFactory(other, 8.0).make(LINE.format(on=7.0, rc=8.0))
        other.evaluate()
        other.close()
        s = systems.tip3p_box(216, 18.62, seed=5, jitter=0.2)
        gs = GpuSystem(ctx, s, "mixed")
        ForceFactory(gs, 8.0).make(LINE.format(on=7.0, rc=8.0))
        if cap:
            gs.set_column_capacity(cap)
        LeapfrogIntegrator(0.5).run(gs, 20)
        out.append((gs.positions(), gs.velocities()))
        gs.close()
    for got in out[1:]:
        assert np.array_equal(got[0], out[0][0]) and np.array_equal(got[1], out[0][1])
