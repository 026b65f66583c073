"""Which transform a PME grid takes: the library's three FFT kernels (five
launches a reciprocal term) or cuFFT (four of the library's own), on both
sides of every line of the rule, and the largest plane the kernels take
against the FP64 SPME restatement (tolerance of the repository's PME tests)."""
import numpy as np
import pytest

import fixtures as F
from oracle import spme
from protomol_b200 import GpuSystem, PMEwaldSystemForce, ScalarStructure, systems

pytestmark = pytest.mark.gpu


def _force(ctx, topo, grid):
    gs = GpuSystem(ctx, topo, "mixed")
    return gs, PMEwaldSystemForce(gs, 0.35, 0.0, order=4, grid=grid, real=False, reciprocal=True,
                                  correction=False)


@pytest.mark.parametrize("grid,own", [
    # planes beyond one wave: one plane an SM, two planes an SM
    ((144, 128, 128), True), ((150, 128, 128), False), ((160, 160, 160), False),
    ((200, 100, 100), True), ((300, 100, 100), False),
    # few large planes
    ((48, 128, 128), True), ((45, 128, 128), False), ((32, 125, 128), True),
    # long columns, 16 and 8 of them a block
    ((256, 64, 64), True), ((270, 64, 64), False), ((512, 16, 16), True), ((540, 16, 16), False),
    # sizes the kernels do not take
    ((21, 20, 20), False), ((60, 180, 180), False)])
def test_path_of_a_grid(ctx, grid, own):
    s = systems.tip3p_box(64, 19.0, seed=3, jitter=0.2)
    gs, rec = _force(ctx, s, grid)
    before = gs.kernel_count()
    gs.evaluate_forces()
    assert gs.kernel_count() - before == (5 if own else 4)
    gs.close()


@pytest.mark.parametrize("grid", [(48, 162, 162), (160, 128, 128), (270, 16, 64)])
def test_reciprocal_at_the_lines(ctx, grid):
    topo = F.topology(F.load("water423"))
    gs, rec = _force(ctx, topo, grid)
    fo, eo = spme.reciprocal(topo.pos, topo.charge, topo.box, 0.35, 4, grid)
    f, e = np.zeros_like(topo.pos), ScalarStructure()
    rec.evaluate(topo.pos, f, e)
    assert F.rms_rel(f, fo) <= 1e-5
    assert abs(e[0] - eo) <= 1e-5 * abs(eo)
    gs.close()
