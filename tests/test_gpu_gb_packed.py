"""The packed FP32 GB passes of large molecules: the smallest molecules they
take (a last tile of 1, 8 and 32 atoms) and one below, water atoms among
them, GB alone and with ACE, against the FP64 system's passes.  Tolerance:
the repository's mixed-precision bound, 1e-5 RMS relative on the forces;
1e-6 relative on the energy (FP32 terms of 1e-7 each, summed in FP64)."""
import numpy as np
import pytest

import fixtures as F
from protomol_b200 import ForceFactory, GpuSystem, systems

pytestmark = pytest.mark.gpu

GB = "GBForce -algorithm NonbondedSimpleFull -soluteDielec 1.0 -solventDielec 78.5"
ACE = "GBACEForce -algorithm NonbondedSimpleFull"


@pytest.mark.parametrize("n,water", [(3456, 0), (3457, 0), (3488, 0), (3488, 300), (4200, 77)])
def test_mixed_equals_double(ctx, n, water):
    s = systems.gb_polymer(n, seed=3)
    s.water[n - water:] = 1
    out = []
    for precision in ("double", "mixed"):
        gs = GpuSystem(ctx, s, precision)
        ff = ForceFactory(gs)
        ff.make(GB)
        f1 = gs.evaluate_forces()
        e1, _ = gs.evaluate()
        ff.make(ACE)
        f2 = gs.evaluate_forces()
        e2, _ = gs.evaluate()
        out.append((f1, f2, e1[0], e2[0]))
        gs.close()
    d, m = out
    for k in (0, 1):
        assert F.rms_rel(m[k], d[k]) <= 1e-5, (k, F.rms_rel(m[k], d[k]))
    for k in (2, 3):
        assert abs(m[k] - d[k]) <= 1e-6 * max(1.0, abs(d[k])), (k, m[k], d[k])
