"""Pairs at the cutoff of atoms many periods away from the box (unwrapped
coordinates): forces and energies of both precisions accept by the
reference's minimal difference of the raw positions, although the wrapped
coordinates they compute with carry the rounding of the large ones (a
relative 3e-11 of r^2 at 1e6 A)."""
from types import SimpleNamespace

import numpy as np
import pytest

from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

EDGE, RC = 20.1, 8.0


def _wrap(x):
    """The list's wrapped coordinate: x - (x - minimalPosition(x))."""
    o = np.where(x < -EDGE / 2, x + EDGE, np.where(x > EDGE / 2, x - EDGE, x))
    w = o - EDGE * np.rint(o * (1.0 / EDGE))
    return x - (x - w)


def _norm2(d):
    return d[0] * d[0] + d[1] * d[1] + d[2] * d[2]


def _minimal(a, b):
    """minimalDifference's squared length (PeriodicBoundaryConditions.h:72-110)."""
    d = b - a
    d = np.where(d < -EDGE / 2, d + EDGE, np.where(d > EDGE / 2, d - EDGE, d))
    return _norm2(d - EDGE * np.rint(d * (1.0 / EDGE)))


def _wrapped(a, b):
    """The squared distance formed from the wrapped coordinates."""
    xa, xb = _wrap(a), _wrap(b)
    return _norm2((xb - EDGE * np.rint((xb - xa) / EDGE)) - xa)


def far_pairs(count=8, far=1.0e6, apart=2.0e-12):
    """Pairs the two arithmetics put on different sides of the cutoff, the
    wrapped one by more than a relative `apart` of r^2."""
    rng = np.random.default_rng(7)
    out = []
    while len(out) < count:
        a = rng.uniform(-10, 10, 3) + far * rng.choice([-1, 1], 3) * rng.uniform(0.5, 1, 3)
        u = rng.normal(size=3)
        b = a + RC * u / np.linalg.norm(u) + EDGE * rng.integers(-2, 3, 3)
        inside = _minimal(a, b) <= RC * RC
        r2 = _wrapped(a, b)
        if (r2 > RC * RC * (1 + apart)) if inside else (r2 < RC * RC * (1 - apart)):
            out.append((a, b, inside))
    return out


def test_far_pairs_exist_on_both_sides():
    inside = [p[2] for p in far_pairs(16)]
    assert any(inside) and not all(inside)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "double"])
def test_raw_positions_decide(ctx, precision):
    box = np.zeros(12)
    box[0] = box[4] = box[8] = EDGE
    for a, b, inside in far_pairs():
        s = SimpleNamespace(pos=np.array([a, b]), charge=np.ones(2), mass=np.full(2, 16.0),
                            type=np.zeros(2, np.int32), molecule=np.arange(2, dtype=np.int32),
                            lj=systems.charmm_lj_table(np.array([0.15]), np.array([1.77])),
                            exclusions=np.zeros((0, 3), np.int32), periodic=True, box=box)
        gs = GpuSystem(ctx, s, precision)
        force = ForceFactory(gs, RC).make(
            f"LennardJones -algorithm NonbondedCutoff -switchingFunction C2 -switchon 6 "
            f"-cutoff {RC} -cutoff {RC}")
        assert gs.lib.pmgpu_set_count_pairs(gs.h, 1) == 0
        gs.evaluate_forces()
        assert force.stats()["pairs_in_cutoff"] == int(inside)
        gs.evaluate()
        assert force.stats()["pairs_in_cutoff"] == int(inside)
        force.evaluate(s.pos, np.zeros((2, 3)), ScalarStructure(), virial=True)
        assert force.stats()["pairs_in_cutoff"] == int(inside)
        gs.close()
