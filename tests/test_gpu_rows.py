"""The pair kernels over rows of column clusters where they can go wrong: small
and flat boxes (the list's half by row parity instead of by half plane), two
different cutoffs, j-forces too large for their 32-bit sums, lists and columns
that outgrow their estimates, one-term forces evaluated as a pair, and the
constrained step's clusters of every shape.

Bounds, set before the first run: those of the parity suite (forces within 1e-5
relative RMS mixed, 1e-11 of the RMS force FP64; pair sets equal; energies
within 1e-6 of |E_LJ| + |E_C| on a few hundred atoms, 1e-11 FP64).
"""
import dataclasses

import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

from oracle import oracle
from protomol_b200 import forces as F
from protomol_b200 import integrate, systems, workloads
from protomol_b200.batch import Batch

pytestmark = pytest.mark.gpu

LJ9 = "LennardJones -switchingFunction C2 -algorithm NonbondedCutoff -switchon 8 -cutoff 9 -cutoff 9"
CUTS_8_9 = ("LennardJones CoulombEwaldReal -switchingFunction C2 -switchingFunction Cutoff "
            "-algorithm NonbondedCutoff -switchon 7 -cutoff 9 -alpha 0.35 -cutoff 8 -cutoff 9")


def _box(lengths):
    b = np.zeros((4, 3))
    b[0, 0], b[1, 1], b[2, 2] = lengths
    return b


def _fluid(positions, lengths, charges=None):
    """Oxygen-like atoms without molecules at the given places."""
    base = systems.oxygen_fluid_216()
    n = len(positions)
    return dataclasses.replace(
        base, positions=np.asarray(positions, float), scaled_charge=np.zeros(n) if charges is None else charges,
        atom_type=np.zeros(n, np.int32), molecule=np.arange(n, dtype=np.int32), mass=np.full(n, 15.9994),
        box=_box(lengths), cell_size=4.5)


def _eval(s, defs, precision):
    topo = F.Topology(s)
    fs = [F.ForceFactory.make(topo, d, precision) for d in defs]
    f, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure()
    F.evaluate_group(topo, fs, s.positions, f, e)
    return topo, fs, f, e


def _check(s, defs, precision, energy=None):
    ref = oracle.evaluate(s, [F.parse_definition(d) for d in defs])
    topo, fs, f, e = _eval(s, defs, precision)
    rms = np.sqrt((ref["forces"] ** 2).mean())
    scale = abs(ref["lennard_jones"]) + abs(ref["coulomb"])
    if precision == "fp64":
        assert np.abs(f - ref["forces"]).max() <= 1e-11 * max(rms, np.abs(ref["forces"]).max())
        tol = 1e-11
    else:
        assert np.sqrt(((f - ref["forces"]) ** 2).mean()) <= 1e-5 * rms
        tol = energy or 1e-6
    assert abs(e.lennard_jones - ref["lennard_jones"]) <= tol * scale
    assert abs(e.coulomb - ref["coulomb"]) <= tol * scale
    assert np.abs(e.virial_tensor - ref["virial"]).max() <= tol * np.abs(ref["virial"]).max()
    return topo, fs, ref


def _same_pairs(s, d, force):
    ref = oracle.evaluate(s, [F.parse_definition(d)], want_pairs=True)["pairs"]
    key = lambda p: np.sort(p[:, 0].astype(np.int64) * s.n_atoms + p[:, 1])
    assert np.array_equal(key(force.pairs(s.positions)), key(ref))


def _lj9_hessian_v(pos, v, A, B):
    """LJ9's Hessian times v for atoms of one type and no periodic image, in
    a = r^2: E = (A / a^6 - B / a^3) S(a), S the C2 switch from 8 to 9 A."""
    i, j = cKDTree(pos).query_pairs(9.0, output_type="ndarray").T
    d, u = pos[i] - pos[j], v[i] - v[j]
    a, on, c = (d * d).sum(1), 64.0, 81.0
    e, e1, e2 = A / a ** 6 - B / a ** 3, -6 * A / a ** 7 + 3 * B / a ** 4, 42 * A / a ** 8 - 12 * B / a ** 5
    k = np.where(a >= on, 1.0 / (c - on) ** 3, 0.0)
    s0 = np.where(a >= on, k * (c - a) ** 2 * (c - 3 * on + 2 * a), 1.0)
    s1, s2 = 6 * k * (c - a) * (on - a), 6 * k * (2 * a - on - c)
    E1, E2 = e1 * s0 + e * s1, e2 * s0 + 2 * e1 * s1 + e * s2
    w = 2 * E1[:, None] * u + (4 * E2 * (d * u).sum(1))[:, None] * d
    out = np.zeros_like(pos)
    np.add.at(out, i, w)
    np.add.at(out, j, -w)
    return out


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("lengths", [(18.3, 18.3, 18.3), (19.1, 23.7, 40.9), (45.2, 18.5, 27.3), (37.0, 41.0, 18.2)])
def test_small_and_flat_boxes(lengths, precision):
    k = [int(x // 3.05) for x in lengths]
    g = np.stack(np.meshgrid(*[np.arange(m) for m in k], indexing="ij"), -1).reshape(-1, 3)
    sites = (g + 0.5) * (np.array(lengths) / k) - np.array(lengths) / 2
    s = dataclasses.replace(systems.water_box(len(sites), 7), box=_box(lengths),
                            positions=systems._water_atoms(np.random.default_rng(7), sites, jitter=0.1))
    d = workloads.lj_ewald_split(8, 9, 0.35)
    topo, fs, _ = _check(s, [d], precision)
    if precision == "mixed":
        assert topo.pair_layout() == "columns"
    _same_pairs(s, d, fs[0])


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 33])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_few_atoms(n, precision):
    rng = np.random.default_rng(n)
    g = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g[rng.permutation(len(g))[:n]] + 0.5) * 4.1 - 10.2 + rng.uniform(-0.4, 0.4, (n, 3))
    s = _fluid(pos, (20.5, 20.5, 20.5))
    if n == 1:
        _, _, f, e = _eval(s, [LJ9], precision)
        assert not f.any() and e.lennard_jones == 0.0
    else:
        _check(s, [LJ9], precision)


@pytest.mark.parametrize("lengths", [(18.3, 19.0, 21.0), (38.0, 38.0, 38.0)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_two_cutoffs(lengths, precision):
    """Pairs of the outer cutoff only, with distances at the inner one."""
    rng = np.random.default_rng(5)
    k = [int(x // 3.2) for x in lengths]
    g = np.stack(np.meshgrid(*[np.arange(m) for m in k], indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5) * (np.array(lengths) / k) - np.array(lengths) / 2 + rng.uniform(-0.2, 0.2, (len(g), 3))
    for i in range(0, 60, 2):                           # partners at 8 A (1 +- 1e-9) of atom i
        u = rng.normal(size=3)
        pos[-1 - i] = pos[i] + u / np.linalg.norm(u) * 8.0 * (1.0 + (1e-9 if i % 4 else -1e-9))
    d2 = pos[:, None] - pos[None]
    d2 -= np.array(lengths) * np.rint(d2 / np.array(lengths))
    r = np.sqrt((d2 ** 2).sum(-1)) + 10.0 * np.eye(len(pos))
    keep = r.min(1) > 2.4                               # drop partners that landed on an atom
    pos = pos[keep]
    q = np.where(np.arange(len(pos)) % 2 == 0, 4.0, -4.0)
    _check(_fluid(pos, lengths, q), [CUTS_8_9], precision, energy=2e-6)


@pytest.mark.parametrize("r", [2.5, 2.25, 2.0, 1.7])
def test_forces_beyond_the_32_bit_sums(r):
    """Pairs whose force is large, or (at 1.7 A) exceeds the 2,047 kcal/mol/A
    that the j side holds in 32-bit words, several of them on one atom, among
    ordinary ones."""
    rng = np.random.default_rng(11)
    g = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5) * 5.2 - 20.8 + rng.uniform(-0.1, 0.1, (len(g), 3))
    extra = []
    for i in (0, 77, 300):
        for axis in range(3):
            u = np.zeros(3)
            u[axis] = r
            extra.append(pos[i] + u)
    _check(_fluid(np.concatenate([pos, extra]), (41.6, 41.6, 41.6)), [LJ9], "mixed")


@pytest.mark.parametrize("spacing", [3.07, 3.1, 3.15, 3.2])
def test_lattice_boxes(spacing):
    """216 waters on a lattice that divides the box: thousands of pairs at a few
    distances, whose FP32 roundings add up instead of averaging out.  Pair
    vectors and r^2 to the last bit leave about ten roundings of 2^-25 in a
    force, 1e-7 to 2e-7: 5e-7 allowed (1.3e-6 when the fixed-point difference is
    rounded first)."""
    length = 6 * spacing
    pos = systems._water_atoms(np.random.default_rng(1), systems._lattice(6, length))
    s = dataclasses.replace(systems.water_box_216(), positions=pos, box=_box((length,) * 3))
    defs = workloads.lj_c2_coulomb_c2(8, 9)
    ref = oracle.evaluate(s, [F.parse_definition(d) for d in defs])["forces"]
    topo, _, f, _ = _eval(s, defs, "mixed")
    assert topo.pair_layout() == "columns"
    assert np.sqrt(((f - ref) ** 2).mean()) <= 5e-7 * np.sqrt((ref ** 2).mean())


@pytest.mark.parametrize("scale", [1e-1, 1e-3])
def test_weak_forces(scale):
    """Energies scaled down, as in a weakly bound fluid: forces keep their
    relative error, and the sum over the atoms its zero (6,300 independent FP32
    errors of 6.5e-7: 5e-5 of the RMS force; 3e-4 allowed)."""
    s = systems.water_box(2100, 5)
    s = dataclasses.replace(s, scaled_charge=s.scaled_charge * np.sqrt(scale), lj_table=s.lj_table * scale)
    d = workloads.lj_ewald_split(8, 9, 0.35)
    ref = oracle.evaluate(s, [F.parse_definition(d)])["forces"]
    topo, _, f, _ = _eval(s, [d], "mixed")
    rms = np.sqrt((ref ** 2).mean())
    assert topo.pair_layout() == "columns"
    assert np.sqrt(((f - ref) ** 2).mean()) <= 1e-6 * rms
    assert np.abs(f.sum(0)).max() <= 3e-4 * rms


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_droplet_outgrows_the_list_estimate(precision):
    """3,375 atoms in the middle of a 150 A box: the list estimate follows the
    mean density.  The mixed evaluation is repeated with a grown list, the FP64
    one needs none."""
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(15)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g - 7.0) * 3.3 + rng.uniform(-0.2, 0.2, (len(g), 3))
    s = _fluid(pos, (150.0, 150.0, 150.0))
    _, fs, _ = _check(s, [LJ9], precision)
    _same_pairs(s, LJ9, fs[0])


def test_fp64_pair_energies_to_the_last_bits():
    """Repulsive Lennard-Jones pairs beside an electrostatic term, whose 1/r^2
    comes from the reciprocal root both share, have the errors against extended
    precision of the same pairs alone, whose 1/r^2 is a division: both half a
    unit (rms 0.43 to 0.45 of 2^-53), so their energies' within 1.3 (the square
    of a rounded root, 0.92: about 2)."""
    s = _fluid(np.zeros((2, 3)), (30.0, 30.0, 30.0))
    topo = F.Topology(s)
    both = F.ForceFactory.make(topo, "LennardJones Coulomb -switchingFunction C2 -switchingFunction C2 -algorithm "
                               "NonbondedCutoff -switchon 8 -cutoff 9 -switchon 8 -cutoff 9 -cutoff 9", "fp64")
    alone = F.ForceFactory.make(topo, LJ9, "fp64")
    A, B = (np.longdouble(x) for x in s.lj_table[0, 0, :2])
    err = {both: [], alone: []}
    for r in np.random.default_rng(6).integers(int(2.2 * 2 ** 20), int(2.8 * 2 ** 20), 200) / 2.0 ** 20:
        a = np.longdouble(r) ** 2                       # (exact: so is the kernels' r^2)
        ref = A / a ** 6 - B / a ** 3
        for force, out in err.items():
            e = F.ScalarStructure()
            F.evaluate_group(topo, [force], np.array([[0.0, 0, 0], [r, 0, 0]]), np.zeros((2, 3)), e)
            out.append(float((e.lennard_jones - ref) / ref) * 2.0 ** 53)
    rms = {f: np.sqrt(np.mean(np.square(x))) for f, x in err.items()}
    assert rms[both] <= 1.3 * rms[alone]


def test_a_list_far_beyond_its_estimate():
    """13,824 atoms in a 28th of their box, whose list is many times the
    estimate: forces, both virials and the backward pass, over and over, with
    the same energies to the last bit whichever rows found a place."""
    rng = np.random.default_rng(8)
    g = np.stack(np.meshgrid(*[np.arange(24)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g - 11.5) * 3.3 + rng.uniform(-0.2, 0.2, (len(g), 3))
    s = _fluid(pos, (240.0, 240.0, 240.0))
    ref = oracle.evaluate(s, [F.parse_definition(LJ9)])
    topo = F.Topology(s)
    force = F.ForceFactory.make(topo, LJ9, "fp64")
    topo.set_molecule_positions(pos)
    seen = set()
    scale = np.abs(ref["forces"]).max()
    v = rng.normal(size=pos.shape)
    for k in range(20):
        out, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure(virial=True, molecular_virial=k % 2 == 1)
        F.evaluate_group(topo, [force], s.positions, out, e)
        seen.add(e.lennard_jones)
        assert np.abs(out - ref["forces"]).max() <= 1e-11 * scale
        assert np.abs(e.virial_tensor - ref["virial"]).max() <= 1e-11 * np.abs(ref["virial"]).max()
        if k % 2:                                       # every atom is its own molecule
            assert np.abs(e.molecular_virial_tensor - ref["virial"]).max() <= 1e-11 * np.abs(ref["virial"]).max()
        r = F.adjoint(topo, [force], s.positions, v)
        assert abs(r["lennard_jones"] - ref["lennard_jones"]) <= 1e-11 * abs(ref["lennard_jones"])
        # the energy is linear in the table
        assert abs((r["dE_dlj"] * s.lj_table).sum() - ref["lennard_jones"]) <= 1e-9 * abs(ref["lennard_jones"])
    assert len(seen) == 1 and abs(seen.pop() - ref["lennard_jones"]) <= 1e-11 * abs(ref["lennard_jones"])
    hv = _lj9_hessian_v(pos, v, *s.lj_table[0, 0, :2])
    assert np.abs(r["hv"] - hv).max() <= 1e-11 * np.abs(hv).max()
    mixed = F.ForceFactory.make(topo, LJ9, "mixed")
    for _ in range(2):
        r = F.adjoint(topo, [mixed], s.positions, v)
        assert np.linalg.norm(r["hv"] - hv) <= 1e-5 * np.linalg.norm(hv)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("length", [2500.0, 60000.0])
def test_pairs_at_the_cutoff_in_a_long_box(length, precision):
    """Pairs just inside the cutoff along a long edge, where the list's FP32
    cluster boxes are coarse (a step of 4e-3 A at 60,000 A)."""
    rng = np.random.default_rng(4)
    n = int(length / 80)                                # pairs on each of two lines
    pos = []
    for x in (-7.5, 7.5):
        # a single atom first: every fourth pair has its atoms in two rows
        z = (np.arange(n) + 0.5) * (length - 100) / n - length / 2 + 50 + rng.uniform(-20, 20, n)
        z = np.concatenate([[-length / 2 + 1.0], np.stack([z, z + 9.0 * (1 - 1e-10)], 1).ravel()])
        pos.append(np.stack([np.full_like(z, x), np.full_like(z, x), z], 1))
    s = _fluid(np.concatenate(pos), (30.0, 30.0, length))
    force = F.ForceFactory.make(F.Topology(s), LJ9, precision)
    got = force.pairs(s.positions)
    assert len(got) >= 2 * n
    _same_pairs(s, LJ9, force)


EWALD12 = "CoulombEwaldReal -switchingFunction Cutoff -algorithm NonbondedCutoff -alpha 0.3 -cutoff 12 -cutoff 12"


@pytest.mark.parametrize("concurrent", [0, 1])
@pytest.mark.parametrize("group", ["fp64_after_mixed", "two_cutoffs_molecular_virial"])
def test_a_list_after_the_last_near_pairs(group, concurrent):
    """A list made after the last mixed force, whose near pairs may still be in
    work beside PME: the group's sums are those of its forces alone."""
    s = systems.water_box(2100, 4)
    split = workloads.lj_ewald_split(8, 9, 0.35)
    pme = workloads.pme_reciprocal((40, 40, 40), 9, 0.35)
    defs, mol = (([(split, "mixed"), (split, "fp64"), (pme, "mixed")], False) if group == "fp64_after_mixed" else
                 ([(LJ9, "mixed"), (EWALD12, "mixed"), (pme, "mixed")], True))
    topo = F.Topology(s)
    topo.set_tuning(pme_concurrent=concurrent)
    topo.set_molecule_positions(F.molecular_centers(s.molecule, s.positions, s.mass))
    fs = [F.ForceFactory.make(topo, d, p) for d, p in defs]

    def evaluate(which):
        f, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure(virial=True, molecular_virial=mol)
        F.evaluate_group(topo, which, s.positions, f, e)
        return f, np.array([e.lennard_jones, e.coulomb]), e.virial_tensor, e.molecular_virial_tensor if mol else 0 * e.virial_tensor

    alone = [evaluate([f]) for f in fs]
    f, e, v, m = [sum(a[k] for a in alone) for k in range(4)]
    scale = sum(np.abs(a[1]).sum() for a in alone)
    for _ in range(10):
        g = evaluate(fs)
        assert np.sqrt(((g[0] - f) ** 2).mean()) <= 1e-5 * np.sqrt((f ** 2).mean())
        assert np.abs(g[1] - e).max() <= 1e-6 * scale
        assert np.abs(g[2] - v).max() <= 1e-6 * np.abs(v).max()
        assert np.abs(g[3] - m).max() <= 1e-6 * max(np.abs(m).max(), 1.0)


def test_an_overflowing_mixed_list_beside_an_fp64_one_grows():
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(15)] * 3, indexing="ij"), -1).reshape(-1, 3)
    s = _fluid((g - 7.0) * 3.3 + rng.uniform(-0.2, 0.2, (len(g), 3)), (150.0, 150.0, 150.0))
    ref = oracle.evaluate(s, [F.parse_definition(LJ9)])
    topo = F.Topology(s)
    fs = [F.ForceFactory.make(topo, LJ9, p) for p in ("mixed", "fp64")]
    out, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure()
    F.evaluate_group(topo, fs, s.positions, out, e)
    assert np.sqrt(((out / 2 - ref["forces"]) ** 2).mean()) <= 1e-5 * np.sqrt((ref["forces"] ** 2).mean())
    assert abs(e.lennard_jones / 2 - ref["lennard_jones"]) <= 1e-6 * abs(ref["lennard_jones"])


def test_a_column_of_more_atoms_than_the_sort_holds():
    """2,300 atoms on one line along z: one column holds them all.  The FP64
    forces take the column unsorted."""
    rng = np.random.default_rng(3)
    z = (np.arange(2300) - 1150) * 3.9
    pos = np.stack([0.3 + 0 * z, 0.4 + 0 * z, z], 1) + rng.uniform(-0.2, 0.2, (2300, 3))
    _check(_fluid(pos, (30.0, 30.0, 2300 * 3.9)), [LJ9], "fp64")


def test_one_term_forces_as_a_pair():
    """LJ and Coulomb C2 as two forces of one group: their energies keep their
    slots, each alone still evaluates alone, and the group goes on after one of
    them is destroyed."""
    s = systems.water_box(640, 9)
    defs = workloads.lj_c2_coulomb_c2(8, 9)
    topo, fs, ref = _check(s, defs, "fp64")
    alone = []
    for f, d in zip(fs, defs):
        out, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure()
        F.evaluate_group(topo, [f], s.positions, out, e)
        r = oracle.evaluate(s, [F.parse_definition(d)])
        assert np.abs(out - r["forces"]).max() <= 1e-11 * np.abs(r["forces"]).max()
        alone.append((e.lennard_jones, e.coulomb))
    assert alone[0][1] == 0.0 and alone[1][0] == 0.0
    fs[1].close()
    again = F.ForceFactory.make(topo, defs[1], "fp64")
    out, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure()
    F.evaluate_group(topo, [again, fs[0]], s.positions, out, e)
    assert np.abs(out - ref["forces"]).max() <= 1e-11 * np.abs(ref["forces"]).max()
    assert abs(e.lennard_jones - alone[0][0]) <= 1e-11 * abs(alone[0][0])


def test_reused_list_survives_an_fp64_evaluation_between():
    """An FP64 evaluation (its own list, in the same buffers) between two
    evaluations of a reused mixed list."""
    s = systems.water_box(2100, 4)
    d = workloads.lj_ewald_split(8, 9, 0.35)
    topo = F.Topology(s)
    mixed, fp64 = F.ForceFactory.make(topo, d, "mixed"), F.ForceFactory.make(topo, d, "fp64")
    topo.set_pair_list(1.0, 10)
    ref = oracle.evaluate(s, [F.parse_definition(d)])["forces"]
    for fs in ([mixed], [fp64], [mixed], [mixed, fp64], [mixed]):
        out = np.zeros((s.n_atoms, 3))
        F.evaluate_group(topo, fs, s.positions, out, F.ScalarStructure())
        assert np.sqrt(((out / len(fs) - ref) ** 2).mean()) <= 1e-5 * np.sqrt((ref ** 2).mean())


@pytest.mark.parametrize("other", ["cells", "pairs", "batch"])
def test_a_kept_list_that_another_call_overwrote(other):
    """A reused pair list shares its buffers with every other list of its
    system: a force on the cell layout (a cutoff beyond half the box), a pair
    recording, a batch with the system as a member."""
    s = systems.water_box(700, 4)                       # 27.6 A
    d = workloads.lj_ewald_split(8, 9, 0.35)
    ref = oracle.evaluate(s, [F.parse_definition(d)])["forces"]
    topo = F.Topology(s)
    kept = F.ForceFactory.make(topo, d, "mixed")
    wide = F.ForceFactory.make(topo, LJ9.replace("cutoff 9", "cutoff 14.5"), "mixed")
    topo.set_pair_list(1.0, 10)

    def check(forces):
        assert np.sqrt(((forces - ref) ** 2).mean()) <= 1e-5 * np.sqrt((ref ** 2).mean())

    for _ in range(3):
        out = np.zeros((s.n_atoms, 3))
        F.evaluate_group(topo, [kept], s.positions, out, F.ScalarStructure())
        check(out)
        if other == "cells":
            F.evaluate_group(topo, [wide], s.positions, np.zeros((s.n_atoms, 3)), F.ScalarStructure())
        elif other == "pairs":
            wide.pairs(s.positions)
        else:
            b = Batch()
            moved = systems.perturbed(s, 0.3, 5)
            b.add(topo, [kept], moved.positions)
            torch.cuda.synchronize()
            b.evaluate()
            b.synchronize()
            m = oracle.evaluate(moved, [F.parse_definition(d)])["forces"]
            got = b.members[0][3].cpu().numpy()
            assert np.sqrt(((got - m) ** 2).mean()) <= 1e-5 * np.sqrt((m ** 2).mean())
    assert topo.pair_list_builds() == 3


def test_reused_list_and_a_first_molecular_virial():
    """The molecular virial asked for while the pair list of an evaluation
    without it is kept: that of a system that never kept one."""
    s = systems.water_box(2100, 4)
    d = workloads.lj_ewald_split(8, 9, 0.35)
    centers = F.molecular_centers(s.molecule, s.positions, s.mass)
    got = []
    for every in (1, 10):
        topo = F.Topology(s)
        topo.set_molecule_positions(centers)
        force = F.ForceFactory.make(topo, d, "mixed")
        topo.set_pair_list(1.0, every)
        for mol in (False, True, True):
            f, e = np.zeros((s.n_atoms, 3)), F.ScalarStructure(virial=True, molecular_virial=mol)
            F.evaluate_group(topo, [force], s.positions, f, e)
        got.append(e.molecular_virial_tensor)
        if every > 1:
            assert topo.pair_list_builds() == 2         # the second has the slots the virial reads
    assert np.abs(got[0] - got[1]).max() <= 1e-11 * np.abs(got[0]).max()


def test_constrained_step_with_many_free_atoms():
    """A few constrained triangles among thousands of free atoms, every one of
    them advanced as the oracle does."""
    m = 14
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    length = 4.0 * m
    pos = (g + 0.5) * 4.0 - length / 2
    held = 7
    tri = np.array([[0.0, 0.0, 0.0], [0.95, 0.0, 0.0], [-0.3, 0.9, 0.0]])
    every = np.concatenate([(pos[:held, None] + tri).reshape(-1, 3), pos[held:]])
    o = 3 * np.arange(held)
    atoms = np.concatenate([np.stack([o + a, o + b], 1) for a, b in ((0, 1), (0, 2), (1, 2))]).astype(np.int32)
    excl = np.array([(a, b, systems.EXCLUSION_FULL) for a, b in atoms], np.int32)
    s = dataclasses.replace(_fluid(every, (length,) * 3), exclusions=excl, exclusion_check=excl[:, 2].copy(),
                            molecule=np.concatenate([np.repeat(np.arange(held), 3),
                                                     held + np.arange(len(pos) - held)]).astype(np.int32))
    con = {"atoms": atoms, "rest": np.linalg.norm(every[atoms[:, 0]] - every[atoms[:, 1]], axis=1),
           "shake": (1e-8, 100), "rattle": (1e-8, 100), "mass": s.mass}
    v = integrate.maxwell_boltzmann(s.mass, 300.0, 3)
    ref = oracle.leapfrog(s, [F.parse_definition(LJ9)], v, 1.0, 3, constraints=con)
    topo = F.Topology(s)
    lf = integrate.Leapfrog(topo, [F.ForceFactory.make(topo, LJ9, "fp64")], s.positions, v, s.mass, 1.0, virial=True,
                            constraints=con).initialize()
    lf.run(3)
    x, vel, f, e = lf.state()
    assert np.abs(x - ref[0]).max() <= 1e-10
    assert np.abs(vel - ref[1]).max() <= 1e-9 * np.abs(ref[1]).max()


@pytest.mark.parametrize("shape", ["pairs", "stars", "triangles", "mixed_order", "chains", "many"])
def test_constrained_steps(shape):
    """Clusters of two and three atoms in any order of their constraints (the
    one-launch step), four-atom chains and more clusters than it takes (the
    separate kernels), free atoms beside them, against the oracle."""
    m = 9 if shape == "many" else 6
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    length = 4.0 * m
    pos = (g + 0.5) * 4.0 - length / 2
    n0 = len(pos)
    tri = np.array([[0.0, 0.0, 0.0], [0.95, 0.0, 0.0], [-0.3, 0.9, 0.0], [0.2, 0.3, 0.95]])
    per = {"pairs": 2, "chains": 4}.get(shape, 3)
    held = n0 - 5                                       # the last five sites hold single atoms
    every = np.concatenate([(pos[:held, None] + tri[None, :per]).reshape(-1, 3), pos[held:]])
    o = per * np.arange(held)
    cons = {"pairs": [(0, 1)], "stars": [(1, 0), (0, 2)], "triangles": [(0, 1), (0, 2), (1, 2)],
            "mixed_order": [(2, 1), (0, 2), (1, 0)], "chains": [(0, 1), (1, 2), (2, 3)],
            "many": [(0, 1), (0, 2), (1, 2)]}[shape]
    atoms = np.concatenate([np.stack([o + a, o + b], 1) for a, b in cons]).astype(np.int32)
    s = _fluid(every, (length,) * 3)
    mol = np.concatenate([np.repeat(np.arange(held), per), held + np.arange(5)])
    # everything inside a molecule excluded
    pairs = [(k + a, k + b) for k in o for a in range(per) for b in range(a + 1, per)]
    excl = np.array([(a, b, systems.EXCLUSION_FULL) for a, b in pairs], np.int32)
    s = dataclasses.replace(s, molecule=mol.astype(np.int32), exclusions=excl, exclusion_check=excl[:, 2].copy())
    rest = np.linalg.norm(every[atoms[:, 0]] - every[atoms[:, 1]], axis=1)
    con = {"atoms": atoms, "rest": rest, "shake": (1e-8, 100), "rattle": (1e-8, 100), "mass": s.mass}
    v = integrate.maxwell_boltzmann(s.mass, 300.0, 3)
    steps = 3
    ref = oracle.leapfrog(s, [F.parse_definition(LJ9)], v, 1.0, steps, constraints=con)
    topo = F.Topology(s)
    lf = integrate.Leapfrog(topo, [F.ForceFactory.make(topo, LJ9, "fp64")], s.positions, v, s.mass, 1.0, virial=True,
                            constraints=con).initialize()
    lf.run(steps)
    x, vel, f, e = lf.state()
    assert np.abs(x - ref[0]).max() <= 1e-10
    assert np.abs(vel - ref[1]).max() <= 1e-9 * np.abs(ref[1]).max()
    assert lf.constraint_limit_hits() == 0
