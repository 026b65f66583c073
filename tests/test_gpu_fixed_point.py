"""Rounding of FP64 sums to fixed point (2^-32 kcal/mol and kcal/mol/A).

Every add into a fixed-point accumulator rounds its term by up to half a
unit, so N adds leave an error of sqrt(N / 12) units RMS: the only error of
FP64 forces and energies that is visible beside the FP64 oracle.  N follows
from the kernels' layout and the list's counts of clusters and tiles; bounds
on a few energies carry a factor for the scatter of their RMS over SEEDS
systems (1.5 is the 99.99 % point of 24)."""
import math

import numpy as np
import pytest

import oracle
from protomol_b200 import ForceFactory, GpuSystem, ScalarStructure, systems

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -32
SEEDS = 24
BLOCK = 8  # warps a block of the pair kernels


def _water_cluster(seed):
    """64 waters without periodicity, all within the cutoff of one another, so
    every tile of the list has pairs."""
    s = systems.tip3p_box(64, 12.42, seed=seed, lattice=4)
    s.periodic, s.box = False, np.zeros(12)
    return s, 30.0


def _water_box(seed):
    """A periodic box, whose atoms nearly fill the list's clusters."""
    return systems.tip3p_box(216, 18.64, seed=seed, jitter=0.2), 8.0


def _oracle(s):
    return oracle.System(pos=s.pos, charge=s.charge, type=s.type, molecule=s.molecule, lj=s.lj,
                         excl=s.exclusions, periodic=s.periodic, box=s.box)


def _cutoff_errors(ctx, make, precision):
    """Per seed: force errors (n, 3), energy errors (2), virial errors (9) in
    units, and the list's clusters and tiles."""
    out = []
    for seed in range(SEEDS):
        s, rc = make(seed)
        gs = GpuSystem(ctx, s, precision)
        force = ForceFactory(gs, rc).make(
            f"LennardJones Coulomb -algorithm NonbondedCutoff -switchingFunction C1 -cutoff {rc} "
            f"-switchingFunction C1 -cutoff {rc} -cutoff {rc}")
        f, e = np.zeros_like(s.pos), ScalarStructure()
        force.evaluate(s.pos, f, e, virial=True)
        st = force.stats()
        sw = oracle.Switch("C1", rc)
        fo, eo, vo = oracle.cutoff_force(_oracle(s), rc, rc,
                                         [("LennardJones", sw), ("Coulomb", sw)])
        out.append(((f - fo) / UNIT, np.array([e[0] - eo["coulomb"], e[1] - eo["lj"]]) / UNIT,
                    (e[7:16] - np.asarray(vo).ravel()) / UNIT, st["clusters"],
                    st["list_entries"]))
        gs.close()
    return out


def _rms(parts):
    return float(np.sqrt(np.mean(np.square(np.concatenate([np.ravel(p) for p in parts])))))


def test_double_pair_forces(ctx):
    """An atom takes one add for each tile that has it as a j atom, and for
    its own cluster, whose tiles go to at most 32 warps, one a block of 8."""
    got = _cutoff_errors(ctx, _water_cluster, "double")
    adds = np.mean([4 * tiles / 192 + 32 / BLOCK for *_, tiles in got])
    assert _rms([g[0] for g in got]) <= np.sqrt(adds / 12)


def test_double_pair_energies(ctx):
    """Energies and virial: one add a block, at most 32 / 8 blocks a cluster."""
    got = _cutoff_errors(ctx, _water_box, "double")
    bound = 1.5 * np.sqrt(np.mean([clusters * 32 / BLOCK for *_, clusters, _ in got]) / 12)
    assert _rms([g[1] for g in got]) <= bound
    assert _rms([g[2] for g in got]) <= bound


def test_mixed_energies(ctx):
    """The mixed path's FP64 energies and virial: at most 12 warps a cluster,
    one add a block."""
    got = _cutoff_errors(ctx, _water_box, "mixed")
    bound = 1.5 * np.sqrt(np.mean([clusters * 12 / BLOCK for *_, clusters, _ in got]) / 12)
    assert _rms([g[1] for g in got]) <= bound
    assert _rms([g[2] for g in got]) <= bound


def _coulomb_pairs(s, rc=0.0):
    """Coulomb (with rc: C1 switched) energy and virial of every pair of a
    molecule, summed exactly, and the sums of their absolute values."""
    i, j = np.triu_indices(len(s.pos), 1)
    scale = np.ones((len(s.pos),) * 2)
    for a, b, kind in s.exclusions:
        scale[a, b] = scale[b, a] = 0.0 if kind == 2 else s.coulomb_scaling
    d = s.pos[j] - s.pos[i]
    r2 = (d * d).sum(1)
    r = np.sqrt(r2)
    e = scale[i, j] * s.charge[i] * s.charge[j] / r
    f = e / r2
    if rc:  # C1SwitchingFunction.h:41-50
        value = 1.0 - 1.5 * r / rc + 0.5 * (r / rc) ** 3
        f = f * value - e * (-1.5 / rc + 1.5 * r2 / rc ** 3) / r
        e = e * value
    v = d[:, :, None] * d[:, None, :] * f[:, None, None]
    terms = np.concatenate([e[:, None], v.reshape(-1, 9)], 1)
    return np.array([math.fsum(t) for t in terms.T]), np.abs(terms).sum(0)


@pytest.mark.parametrize("rc", [0.0, 400.0], ids=["plain", "switched"])
@pytest.mark.parametrize("n", [3, 64, 200, 296, 297, 547, 1185])
def test_row_passes(ctx, n, rc):
    """The FP64 all-pairs passes: one add an atom (two where eight warps share
    it, 129 to 296 atoms), each within half a unit; energies and virial in two words, so only their FP64 sums' rounding
    is left (16 roundings of the terms' absolute sum, far less than it takes)."""
    s = systems.gb_polymer(n, seed=n)
    gs = GpuSystem(ctx, s, "double")
    sw = f" -switchingFunction C1 -cutoff {rc}" if rc else ""
    force = ForceFactory(gs).make("Coulomb -algorithm NonbondedSimpleFull" + sw)
    f, e = np.zeros_like(s.pos), ScalarStructure()
    force.evaluate(s.pos, f, e, virial=True)
    gs.close()
    o = _oracle(s)
    fo = oracle.simplefull_force(o, "Coulomb", oracle.Switch("C1", rc) if rc else None)[0]
    # a thousandth of a unit (2.3e-13) for the FP64 sums of forces up to 30
    assert np.abs(f - fo).max() <= (0.5 * (2 if 128 < n <= 296 else 1) + 1e-3) * UNIT
    exact, size = _coulomb_pairs(s, rc)
    got = np.concatenate([[e[0]], e[7:16]])
    assert (np.abs(got - exact) <= 16 * 2.0 ** -53 * size + 2.0 ** -50).all()


def test_reciprocal_root_of_the_energy_pass(ctx):
    """The mixed path's FP64 energies take 1 / r from an estimate and two Newton
    steps, within two units in the last place; a pair's Coulomb energy of about
    1e8 shows it beside a fixed-point unit of 1e-18 of it.  Distances of 21 bits
    along one axis, so r^2 is exact; two more units for the product with the
    charges, the conversion and the comparison's own roundings."""
    s = systems.tip3p_box(1, 20.0, seed=1)
    s.periodic, s.box = False, np.zeros(12)
    s.pos = np.zeros((3, 3))
    s.pos[2, 1] = 500.0  # out of reach
    s.charge = np.array([2.0 ** 15, 2.0 ** 15, 0.0])
    s.exclusions, s.molecule = np.zeros((0, 3), np.int32), np.arange(3, dtype=np.int32)
    gs = GpuSystem(ctx, s, "mixed")
    force = ForceFactory(gs, 20.0).make("Coulomb -algorithm NonbondedCutoff -switchingFunction "
                                        "Cutoff -cutoff 20 -cutoff 20")
    rng = np.random.default_rng(3)
    for r in rng.integers(2 ** 16, 20 * 2 ** 16, 300) / 2.0 ** 16:
        s.pos[1, 0] = r
        e = ScalarStructure()
        force.evaluate(s.pos, np.zeros_like(s.pos), e)
        assert abs(e[0] * r / 2.0 ** 30 - 1.0) <= 4 * 2.0 ** -52, r
    gs.close()
