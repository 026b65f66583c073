"""PME reciprocal term on grids of every transform the library has: the
own FFT kernels (dimensions that are products of 2, 3 and 5: odd and even,
unequal, one to four passes a dimension, the largest plane) and cuFFT
(another prime, a plane beyond the kernels' shared memory), against the
FP64 SPME restatement at the same grid, order and alpha.  Tolerance: the
RMS and energy bound of the repository's other PME test, 1e-5 (FP32
splines and FFT: about 1e-7 per operation, under 100 operations deep)."""
import numpy as np
import pytest

import fixtures as F
from oracle import spme
from protomol_b200 import GpuSystem, PMEwaldSystemForce, ScalarStructure

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,grid", [
    (4, (4, 5, 6)), (4, (18, 15, 27)), (4, (16, 25, 20)), (6, (30, 9, 8)), (5, (45, 32, 24)),
    (4, (54, 50, 64)), (4, (81, 80, 90)), (4, (16, 162, 162)),
    (4, (128, 18, 4)), (4, (21, 20, 18)), (4, (16, 20, 49)), (4, (8, 180, 180))])
def test_reciprocal_on_grid(ctx, order, grid):
    z = F.load("water423")
    topo = F.topology(z)
    gs = GpuSystem(ctx, topo, "mixed")
    rec = PMEwaldSystemForce(gs, 0.35, 0.0, order=order, grid=grid, real=False, reciprocal=True,
                             correction=False)
    fo, eo = spme.reciprocal(topo.pos, topo.charge, topo.box, 0.35, order, grid)
    for _ in range(2):  # twice: the charge grid is clear again after a pass
        f, e = np.zeros_like(topo.pos), ScalarStructure()
        rec.evaluate(topo.pos, f, e, virial=True)
        assert F.rms_rel(f, fo) <= 1e-5, (grid, F.rms_rel(f, fo))
        assert abs(e[0] - eo) <= 1e-5 * abs(eo), (e[0], eo)
    f0 = np.zeros_like(topo.pos)
    rec.evaluate(topo.pos, f0, None)  # forces only: the same transforms
    assert np.array_equal(f0, f)
    gs.close()
