"""The FP64 energy pass of the mixed-precision path (its own kernel beside
the force-only ones): energies, virial and pair count on systems whose lists
give it partly filled warp steps, leftover queues, several image shells and
unequal cutoffs, against the FP64 oracle.  Tolerance: 1e-10 relative on sums
of the magnitude of the pair energies (the kernel's terms carry a few
2^-53 each, its per-warp sums are rounded to 2^-32)."""
import numpy as np
import pytest

import oracle
from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

pytestmark = pytest.mark.gpu


def _oracle(s):
    return oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                         excl=s.exclusions, periodic=True, box=s.box)


@pytest.mark.parametrize("waters,edge", [(1, 19.0), (3, 19.0), (64, 19.0), (216, 18.62), (700, 27.6)])
@pytest.mark.parametrize("lj,coul", [
    ("C2 -switchon 6 -cutoff 8", "C2 -switchon 6 -cutoff 8"),
    ("C2 -switchon 6 -cutoff 8", "C1 -cutoff 8"),
    ("Cn -n 4 -switchon 6 -cutoff 8", "Cn -n 4 -switchon 6 -cutoff 8"),
    ("C2 -switchon 5 -cutoff 6.5", "C1 -cutoff 8"),
    ("C1 -cutoff 7", "Cn -n 2 -switchon 5 -cutoff 8")])
def test_cutoff_energies_and_virial(ctx, waters, edge, lj, coul):
    s = systems.tip3p_box(waters, edge, seed=5, jitter=0.2)
    gs = GpuSystem(ctx, s, "mixed")
    force = ForceFactory(gs, 8.0).make(
        f"LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction {lj} "
        f"-switchingFunction {coul} -cutoff 8")
    f, e = np.zeros_like(s.pos), ScalarStructure()
    force.evaluate(s.pos, f, e, virial=True)
    pairs = force.stats()["pairs_in_cutoff"]
    e1 = ScalarStructure()
    force.evaluate(s.pos, np.zeros_like(s.pos), e1)
    assert np.array_equal(e[:2], e1[:2])  # the virial form sums the same energies

    def switch(text):
        t = text.split()
        p = {t[k]: float(t[k + 1]) for k in range(1, len(t), 2)}
        return oracle.Switch(t[0], p["-cutoff"], p.get("-switchon", 0.0), 0.0, p.get("-n", 0.0))

    _, eo, vo = oracle.cutoff_force(_oracle(s), 8.0, 8.0,
                                    [("LennardJones", switch(lj)), ("Coulomb", switch(coul))])
    size = max(1.0, np.abs(vo).max(), abs(eo["coulomb"]), abs(eo["lj"]))
    # the oracle sums pair by pair over energies of up to a few hundred each
    size = max(size, 300.0 * waters)
    assert abs(e[0] - eo["coulomb"]) <= 1e-10 * size
    assert abs(e[1] - eo["lj"]) <= 1e-10 * size
    assert np.abs(e[7:16] - np.asarray(vo).ravel()).max() <= 1e-10 * 10 * size
    assert pairs == len(force.pair_set(1 << 20))
    gs.close()
