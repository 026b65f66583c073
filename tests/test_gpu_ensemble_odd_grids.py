"""Ensembles whose PME grids have an odd number of points and need cuFFT (a
dimension with a factor 7): the members' grids are slices of one buffer, and
each member's own plan must take its slice as well (the forces of members
that have none yet are evaluated one by one)."""
import numpy as np
import pytest

from protomol_b200 import ForceFactory, GpuSystem, LeapfrogIntegrator, systems
from protomol_b200.engine import SystemEnsemble

pytestmark = pytest.mark.gpu


def _members(ctx):
    out = []
    # three boxes on 21^3, one on a grid the library's own transform takes
    for seed, k in ((1, 21), (2, 21), (3, 21), (4, 20)):
        s = systems.tip3p_box(216, 18.64, seed=seed, jitter=0.2)
        gs = GpuSystem(ctx, s, "mixed")
        ff = ForceFactory(gs, 8.0)
        for line in ["Bond", "Angle", "LennardJones -algorithm NonbondedCutoff -switchingFunction "
                     "C2 -switchon 7 -cutoff 8 -cutoff 8", "Coulomb -algorithm PMEwald -alpha 0.35 "
                     f"-cutoff 8 -order 4 -gridsize {k} {k} {k}"]:
            ff.make(line)
        out.append(gs)
    return out


def test_members_without_forces(ctx):
    it = LeapfrogIntegrator(0.5)
    members = _members(ctx)
    ens = SystemEnsemble(members)
    ens.run(it, 10)
    ens.run(it, 10)
    batched = [(gs.positions(), gs.energies()[0]) for gs in members]
    # a member evaluated by itself while it belongs to the ensemble
    alone = [gs.evaluate()[0] for gs in members]
    ens.close()
    for gs in members:
        gs.close()
    members = _members(ctx)
    for gs, (x, e), e1 in zip(members, batched, alone):
        for _ in range(2):
            it.run(gs, 10)
        # as tests/test_gpu_ensemble.py: the FFT's FP32 rounding
        assert np.abs(gs.positions() - x).max() <= 1e-6
        assert np.abs(gs.energies()[0] - e).max() <= 1e-6 * np.abs(e).max()
        assert np.abs(gs.evaluate()[0] - e1).max() <= 1e-6 * np.abs(e1).max()
        gs.close()
