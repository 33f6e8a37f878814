"""The force evaluations, integrator runs, batches and backward passes that a
user of the library runs, as a list of cases with their inputs.

Every case is one call sequence through the public entry points: the C ABI's
device evaluation (``pmgpu_evaluate_device``, what a resident integrator
calls), ``forces.evaluate_group`` (what a host program's ForceGroup calls),
``forces.adjoint``, ``batch.Batch`` and ``integrate.Leapfrog``.  The systems
are TIP3P water boxes at 0.0334 molecules/A^3, the same waters around a
random-walk chain, and an ionic Lennard-Jones fluid, from 300 to 1,000,000
atoms, cubic and not.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from protomol_b200 import _lib, batch, integrate, systems, workloads
from protomol_b200 import forces as F

DENSITY = 0.0334            # water molecules per A^3
RIGID = 1e-5                # SHAKE / RATTLE tolerance
TIMEFACTOR = 48.88821290839616

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: 216 waters, LJ and Coulomb C2 as two forces, as
        # a resident integrator evaluates them
        dict(name="water216_c2", kind="device", system="water", n=216, aspect="cube", forces="c2c2", rc=9.0,
             order=4, precision="mixed"),
        # rigid-water dynamics on the device: SHAKE, RATTLE and one FP64
        # evaluation per step, 20 steps a call
        dict(name="rigid216_leapfrog", kind="rigid", n=216, rc=9.0, steps=20, precision="fp64"),
        # a constant-pressure host program: 1,500 waters, PME, atomic and
        # molecular virial, host arrays in and out
        dict(name="water1500_molvir_host", kind="host", system="water", n=1500, aspect="cube", forces="ewald",
             rc=9.0, order=4, precision="mixed", molvir=True),
        # the solvated chain: 14,281 atoms, cutoff 12 A and PME 64^3 on the
        # device, mixed precision (production dynamics)
        dict(name="chain14281", kind="device", system="chain", n=4463, chain=892, aspect="cube", forces="ewald",
             rc=12.0, order=4, precision="mixed"),
        # the same through the FP64 kernels (reference-quality energies)
        dict(name="chain14281_fp64", kind="device", system="chain", n=4463, chain=892, aspect="cube",
             forces="ewald", rc=12.0, order=4, precision="fp64"),
        # the same from a host program: positions up, forces and energies back
        dict(name="chain14281_host", kind="host", system="chain", n=4463, chain=892, aspect="cube",
             forces="ewald", rc=12.0, order=4, precision="mixed", molvir=False),
        # its backward pass: charge and LJ-table gradients and a
        # Hessian-vector product (parameter fitting, normal modes)
        dict(name="chain14281_adjoint", kind="adjoint", system="chain", n=4463, chain=892, aspect="cube",
             forces="ewald", rc=12.0, order=4, precision="mixed"),
        # 24 independent boxes of 100 to 3,000 waters in one launch (replicas,
        # ensembles)
        dict(name="batch24", kind="batch", members=24, lo=100, hi=3000, rc=9.0, precision="mixed"),
        # dynamics of an ionic fluid with a pair list kept for 10 steps, 20
        # steps a call
        dict(name="fluid20k_leapfrog", kind="fluid", n=20001, rc=9.0, steps=20, every=10, precision="mixed"),
        # an interface-like slab, 1 : 1 : 3, with order-6 interpolation
        dict(name="slab61k_order6", kind="device", system="water", n=20411, aspect="slab", forces="ewald",
             rc=10.0, order=6, precision="mixed"),
        # the look-up-table potentials in FP64 on a plate of 192,000 atoms
        dict(name="plate192k_tables_fp64", kind="device", system="water", n=64001, aspect="plate", forces="tables",
             rc=10.0, order=4, precision="fp64"),
        # the largest: 1,000,000 atoms, cutoff 12 A and PME 216^3
        dict(name="water1m", kind="device", system="water", n=333333, aspect="cube", forces="ewald", rc=12.0,
             order=4, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device"] * 6 + ["host"] * 2 + ["adjoint", "batch", "rigid", "fluid"])
    if kind == "rigid":
        return dict(kind=kind, n=rng.randint(100, 400), rc=7.0, steps=rng.randint(10, 30), precision="fp64")
    if kind == "fluid":
        return dict(kind=kind, n=_log(rng, 6000, 27000), rc=round(rng.uniform(8.0, 10.0), 2),
                    steps=rng.randint(10, 25), every=rng.choice([5, 10]), precision="mixed")
    if kind == "batch":
        return dict(kind=kind, members=rng.randint(6, 28), lo=100, hi=rng.randint(400, 3000), rc=9.0,
                    precision="mixed")
    if rng.random() < 0.25 or (kind == "adjoint" and rng.random() < 0.7):
        chain = rng.randint(50, 892)
        c = dict(system="chain", n=_log(rng, 700, 4463), chain=chain, aspect="cube")
        rc = rng.choice([9.0, 10.0, 12.0])
        length = _chain_length(c["n"], chain)
    else:
        hi = {"device": 333333, "host": 40000, "adjoint": 4800}[kind]
        c = dict(system="water", n=_log(rng, 216, hi), aspect=rng.choice(["cube", "cube", "slab", "plate"]))
        length = min(_lengths(c["n"], c["aspect"]))
        rc = rng.choice([8.0, 9.0, 10.0, 12.0])
    rc = min(rc, math.floor(5.0 * length - 0.2) / 10.0)       # one periodic image inside the cutoff
    precision = "fp64" if rng.random() < 0.3 and c["n"] <= 80000 else "mixed"
    forces = rng.choice(["ewald", "ewald", "ewald", "c2c2", "shift"] + (["tables"] if precision == "fp64" else []))
    if kind == "adjoint" and forces == "tables":
        forces = "ewald"
    c.update(kind=kind, forces=forces, rc=rc, order=rng.choice([4, 4, 6]), precision=precision)
    if kind == "host":
        c["molvir"] = rng.random() < 0.4 and c["n"] <= 12000
    return c


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------


def _lengths(n_water, aspect):
    shape = {"cube": (1.0, 1.0, 1.0), "slab": (1.0, 1.0, 3.0), "plate": (1.6, 1.3, 1.0)}[aspect]
    a = (n_water / DENSITY / np.prod(shape)) ** (1.0 / 3.0)
    return [float(round(a * s, 2)) for s in shape]


def _chain_length(n_water, chain):
    return round(52.3 * ((n_water + 0.35 * chain) / (4463 + 0.35 * 892)) ** (1.0 / 3.0), 2)


def _box(lengths):
    b = np.zeros((4, 3))
    b[0, 0], b[1, 1], b[2, 2] = lengths
    return b


def _sites(n, lengths, rng):
    """n of the smallest lattice's sites, centred on the origin."""
    spacing = (np.prod(lengths) / n) ** (1.0 / 3.0)
    k = [max(1, int(math.ceil(x / spacing - 1e-9))) for x in lengths]
    g = [(np.arange(m) + 0.5) * (x / m) - 0.5 * x for m, x in zip(k, lengths)]
    sites = np.stack([a.ravel() for a in np.meshgrid(*g, indexing="ij")], axis=1)
    return sites[np.sort(rng.choice(len(sites), n, replace=False))]


def _water(n, lengths, seed, cell_size):
    """n rigid TIP3P waters with random orientations, in atom order O, H, H."""
    rng = np.random.default_rng(seed)
    oxygen = _sites(n, lengths, rng) + rng.normal(0.0, 0.1, (n, 3))
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                    2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                    2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], axis=1).reshape(n, 3, 3)
    half, oh = math.radians(52.26), 0.9572
    arm = np.array([[0.0, 0.0, 0.0], [oh * math.sin(half), 0.0, oh * math.cos(half)],
                    [-oh * math.sin(half), 0.0, oh * math.cos(half)]])
    o = 3 * np.arange(n)
    pairs = np.concatenate([np.stack([np.stack([o, o + 1], 1), np.stack([o, o + 2], 1)], 1).reshape(-1, 2),
                            np.stack([o + 1, o + 2], 1)])
    excl = np.concatenate([pairs, np.full((len(pairs), 1), systems.EXCLUSION_FULL)], 1).astype(np.int32)
    types = np.array([[0.1521, 1.7682, 0.1521, 1.7682], [0.0, 0.2245, 0.0, 0.2245]])
    return systems.System(
        name=f"water{n}", positions=(oxygen[:, None, :] + np.einsum("nij,aj->nai", rot, arm)).reshape(-1, 3),
        scaled_charge=np.tile(np.array([-0.834, 0.417, 0.417]) * systems.SQRT_COULOMB_CONSTANT, n),
        atom_type=np.tile(np.array([0, 1, 1], np.int32), n), molecule=np.repeat(np.arange(n, dtype=np.int32), 3),
        mass=np.tile(np.array([15.9994, 1.008, 1.008]), n), type_params=types,
        lj_table=systems.lj_table_from_types(types), exclusions=excl, exclusion_check=excl[:, 2].copy(),
        box=_box(lengths), cell_size=cell_size)


@functools.lru_cache(maxsize=4)
def _chain_base(n_water, chain, length):
    return systems.chain_in_water(chain, n_water, length, 2)


def _chain(n_water, chain, length, seed):
    """The solvated chain, its atoms displaced from the built configuration."""
    import dataclasses
    s = _chain_base(n_water, chain, length)
    rng = np.random.default_rng(seed)
    return dataclasses.replace(s, positions=s.positions + rng.normal(0.0, 0.03, s.positions.shape))


def _fluid(n, seed):
    """Oxygen-sized ions of +-0.4 e, no molecules."""
    rng = np.random.default_rng(seed)
    length = round((n / DENSITY) ** (1.0 / 3.0), 2)
    pos = _sites(n, [length] * 3, rng) + rng.normal(0.0, 0.1, (n, 3))
    q = np.where(np.arange(n) % 2 == 0, 0.4, -0.4)
    q -= q.mean()
    types = np.array([[0.1521, 1.7682, 0.1521, 1.7682]])
    return systems.System(
        name=f"fluid{n}", positions=pos, scaled_charge=q * systems.SQRT_COULOMB_CONSTANT,
        atom_type=np.zeros(n, np.int32), molecule=np.arange(n, dtype=np.int32), mass=np.full(n, 15.9994),
        type_params=types, lj_table=systems.lj_table_from_types(types), exclusions=np.zeros((0, 3), np.int32),
        exclusion_check=np.zeros(0, np.int32), box=_box([length] * 3), cell_size=4.5)


def _system(case, seed):
    if case["kind"] == "fluid":
        return _fluid(case["n"], seed)
    if case["kind"] == "rigid":
        return _water(case["n"], _lengths(case["n"], "cube"), seed, 4.5)
    cell = 0.5 * case["rc"]
    if case["system"] == "chain":
        return _chain(case["n"], case["chain"], _chain_length(case["n"], case["chain"]), seed)
    return _water(case["n"], _lengths(case["n"], case["aspect"]), seed, cell)


def _members(case, seed):
    """(system, grid size) of every box of a batch; their sizes belong to the
    case, their configurations to the seed."""
    sizes = np.random.default_rng(case["members"] + case["hi"]).integers(case["lo"], case["hi"] + 1, case["members"])
    out = []
    for k, n in enumerate(sizes):
        lengths = _lengths(int(n), "cube")
        out.append((_water(int(n), lengths, 1000 * seed + k, 4.5), systems.smooth_grid_size(lengths[0])))
    return out


def _alpha(rc):
    return 0.32 if rc == 12.0 else round(systems.ewald_alpha(rc), 4)


def _terms(case):
    """(cutoff forces as lists of (potential, switch), PME or not)"""
    return {"c2c2": ([[("LennardJones", "C2")], [("Coulomb", "C2")]], False),
            "shift": ([[("LennardJones", "C2"), ("Coulomb", "Shift")]], False),
            "fused": ([[("LennardJones", "C2"), ("Coulomb", "C2")]], False),
            "ewald": ([[("LennardJones", "C2"), ("CoulombEwaldReal", "Cutoff")]], True),
            "tables": ([[("LennardJonesTable", "C2"), ("CoulombEwaldRealTable", "Cutoff")]], True)}[case["forces"]]


def _switchon(rc):
    return rc - (2.0 if rc > 10.0 else 1.0)


def _definitions(case, system):
    rc = case["rc"]
    on, alpha = _switchon(rc), _alpha(rc)
    if case["forces"] == "c2c2":
        return workloads.lj_c2_coulomb_c2(on, rc)
    if case["forces"] == "fused":
        return [f"LennardJones Coulomb -switchingFunction C2 -switchingFunction C2 -algorithm NonbondedCutoff "
                f"-switchon {on} -cutoff {rc} -switchon {on} -cutoff {rc} -cutoff {rc}"]
    if case["forces"] == "shift":
        return [f"LennardJones Coulomb -switchingFunction C2 -switchingFunction Shift -algorithm NonbondedCutoff "
                f"-switchon {on} -cutoff {rc} -cutoff {rc} -cutoff {rc}"]
    pme = workloads.pme_reciprocal(_grid(system), rc, alpha, case["order"])
    if case["forces"] == "tables":
        return [f"LennardJonesTable CoulombEwaldRealTable -switchingFunction C2 -algorithm NonbondedCutoff "
                f"-switchon {on} -cutoff {rc} -cutoff {rc} -alpha {alpha} -cutoff {rc}", pme]
    return [workloads.lj_ewald_split(on, rc, alpha), pme]


def _grid(system):
    """About 1 A per point, as the configurations choose it: 64^3 for the
    52.3 A chain box, 216^3 for the 215.4 A box of 1,000,000 atoms."""
    lengths = [float(x) for x in system.box_lengths]
    if len(set(lengths)) == 1 and abs(lengths[0] - 52.3) < 0.2:
        return 64, 64, 64
    return tuple(systems.smooth_grid_size(x) for x in lengths)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
_VP = C.c_void_p


class _Device:
    """A program that keeps its positions, forces and energies on the GPU."""

    def __init__(self, system, definitions, precision):
        self.topo = F.Topology(system)
        self.forces = [F.ForceFactory.make(self.topo, d, precision) for d in definitions]
        self.handles = (_VP * len(self.forces))(*[f.handle for f in self.forces])
        n = system.n_atoms
        self.positions = torch.tensor(system.positions, device="cuda")
        self.out = torch.zeros(3 * n + 11, dtype=torch.float64, device="cuda")
        self.accumulated = self.out[:3 * n].view(n, 3), self.out[3 * n:]
        self.stream = torch.cuda.ExternalStream(self.topo.stream)
        self.lib = _lib.load()

    def evaluate(self):
        with torch.cuda.stream(self.stream):
            self.out.zero_()
        f, e = self.accumulated
        _lib.check(self.lib.pmgpu_evaluate_device(self.topo.handle, len(self.forces), self.handles,
                                                  _VP(self.positions.data_ptr()), _VP(f.data_ptr()),
                                                  _VP(e.data_ptr()), _lib.FLAG_VIRIAL), self.topo.handle)
        return {"forces": f, "energies": e}


def _settle(call, synchronize):
    """The first evaluation of a run, repeated while a pair list outgrows its
    first estimate."""
    for attempt in range(4):
        call()
        try:
            return synchronize()
        except _lib.PmgpuError as e:
            if e.code != 7 or attempt == 3:
                raise


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = batch.Batch()
        b.set_pair_launch(True)
        for system, grid in _members(case, seed):
            topo = F.Topology(system)
            alpha = _alpha(case["rc"])
            defs = [workloads.lj_ewald_split(_switchon(case["rc"]), case["rc"], alpha),
                    workloads.pme_reciprocal((grid,) * 3, case["rc"], alpha)]
            b.add(topo, [F.ForceFactory.make(topo, d, case["precision"]) for d in defs], system.positions)
        stream = torch.cuda.ExternalStream(b.stream)
        torch.cuda.synchronize()
        _settle(b.evaluate, b.synchronize)
        return {"kind": kind, "batch": b, "stream": stream}
    system = _system(case, seed)
    if kind in ("rigid", "fluid"):
        defs = _definitions(dict(case, forces="c2c2" if kind == "rigid" else "fused"), system)
        topo = F.Topology(system)
        forces = [F.ForceFactory.make(topo, d, case["precision"]) for d in defs]
        cons = None
        if kind == "rigid":
            cons = _constraints(case["n"])
            v = np.repeat(integrate.maxwell_boltzmann(np.full(case["n"], 18.0154), 300.0, seed + 1), 3, axis=0)
        else:
            v = integrate.maxwell_boltzmann(system.mass, 300.0, seed + 1)
        lf = integrate.Leapfrog(topo, forces, system.positions, v, system.mass, 1.0, virial=True, constraints=cons)
        if kind == "fluid":
            topo.set_pair_list(1.0, case["every"])
        state = {"kind": kind, "lf": lf, "steps": case["steps"], "stream": torch.cuda.ExternalStream(topo.stream),
                 "start": (lf.pos.clone(), lf.vel.clone())}
        torch.cuda.synchronize()
        _settle(lambda: run(state), lf.synchronize)
        return state
    defs = _definitions(case, system)
    if kind == "device":
        d = _Device(system, defs, case["precision"])
        torch.cuda.synchronize()
        _settle(d.evaluate, lambda: _lib.check(d.lib.pmgpu_synchronize(d.topo.handle), d.topo.handle))
        return {"kind": kind, "device": d}
    topo = F.Topology(system)
    forces = [F.ForceFactory.make(topo, x, case["precision"]) for x in defs]
    state = {"kind": kind, "topo": topo, "forces": forces, "positions": system.positions}
    if kind == "adjoint":
        state["v"] = np.random.default_rng(seed + 1).normal(size=system.positions.shape)
    else:
        state["molvir"] = case["molvir"]
        if case["molvir"]:
            topo.set_molecule_positions(F.molecular_centers(system.molecule, system.positions, system.mass))
    return state


def _constraints(n_water):
    """The waters' bonds, then their H-H distances, SHAKE and RATTLE."""
    o = 3 * np.arange(n_water)
    bonds = np.stack([np.stack([o, o + 1], 1), np.stack([o, o + 2], 1)], 1).reshape(-1, 2)
    oh = 0.9572
    hh = 2.0 * oh * math.sin(math.radians(52.26))
    return {"atoms": np.concatenate([bonds, np.stack([o + 1, o + 2], 1)]).astype(np.int32),
            "rest": np.concatenate([np.full(2 * n_water, oh), np.full(n_water, hh)]),
            "shake": (RIGID, 30), "rattle": (RIGID, 30)}


def run(state):
    kind = state["kind"]
    if kind == "device":
        return state["device"].evaluate()
    if kind == "host":
        n = state["topo"].n_atoms
        f, e = np.zeros((n, 3)), F.ScalarStructure(virial=True, molecular_virial=state["molvir"])
        F.evaluate_group(state["topo"], state["forces"], state["positions"], f, e)
        out = {"forces": f, "energies": np.concatenate([[e.lennard_jones, e.coulomb], e.virial_tensor])}
        if state["molvir"]:
            out["molecular_virial"] = e.molecular_virial_tensor
        return out
    if kind == "adjoint":
        r = F.adjoint(state["topo"], state["forces"], state["positions"], state["v"])
        r["pair_energies"] = np.array([r.pop("lennard_jones"), r.pop("coulomb")])
        return r
    if kind == "batch":
        b = state["batch"]
        with torch.cuda.stream(state["stream"]):
            b.zero()
            b.evaluate()
            return {"forces": torch.cat([m[3] for m in b.members]), "energies": torch.stack([m[4] for m in b.members])}
    lf = state["lf"]
    with torch.cuda.stream(state["stream"]):
        lf.pos.copy_(state["start"][0])
        lf.vel.copy_(state["start"][1])
        lf.initialize()
        lf.run(state["steps"])
    return {"positions": lf.pos, "velocities": lf.vel, "forces": lf.force, "energies": lf.energy}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _work_eval(n, volume, rc, pme, order, adjoint=False):
    """One evaluation of n atoms: positions, charges, types and molecules
    read, forces written; 95 flop per pair inside the cutoff (twice that with
    derivatives), the spline products of spread and gather and the two real
    transforms of the mesh."""
    pairs = 0.5 * n * (n / volume) * 4.0 / 3.0 * math.pi * rc ** 3
    points = volume if pme else 0.0
    flops = pairs * 95.0 * (2.0 if adjoint else 1.0)
    if pme:
        flops += n * order ** 3 * 10.0 + 5.0 * points * math.log2(points)
    return {"bytes": n * (24 + 8 + 4 + 4 + 24 + (24 + 8 if adjoint else 0)), "flops": flops}


def work(case):
    kind = case["kind"]
    total = {"bytes": 0.0, "flops": 0.0}
    if kind == "batch":
        sizes = np.random.default_rng(case["members"] + case["hi"]).integers(case["lo"], case["hi"] + 1,
                                                                             case["members"])
        parts = [_work_eval(3 * int(n), int(n) / DENSITY, case["rc"], True, 4) for n in sizes]
    elif kind in ("rigid", "fluid"):
        n = case["n"] * (3 if kind == "rigid" else 1)
        one = _work_eval(n, case["n"] / DENSITY, case["rc"], False, 0)
        one["bytes"] += 2 * 48 * n                      # positions and velocities read and written
        parts = [{k: v * (case["steps"] + (1 if k == "flops" else 0)) for k, v in one.items()}]
    else:
        chain = case.get("chain", 0)
        volume = _chain_length(case["n"], chain) ** 3 if case["system"] == "chain" else case["n"] / DENSITY
        parts = [_work_eval(3 * case["n"] + chain, volume, case["rc"], _terms(case)[1], case["order"],
                            kind == "adjoint")]
    for p in parts:
        for k in total:
            total[k] += p[k]
    return total


# ---------------------------------------------------------------------------
# the same outputs in plain FP64 torch
# ---------------------------------------------------------------------------


def _pairs(pos, lengths, rc, rows=1 << 24):
    """Chunks (i, j, x_j - x_i) of the ordered pairs within rc, minimal image."""
    n = pos.shape[0]
    L = torch.tensor(lengths, dtype=torch.float64, device=pos.device)
    k = [int(x // rc) for x in lengths]

    def near(i, j):
        d = pos[j] - pos[i]
        d = d - L * torch.round(d / L)
        a = (d * d).sum(-1)
        keep = (a <= rc * rc) & (i != j)
        return i[keep], j[keep], d[keep]

    if min(k) < 3 or n < 20000:
        step = max(1, rows // n)
        every = torch.arange(n, device=pos.device)
        for b in range(0, n, step):
            i = every[b:b + step]
            d = pos[None, :, :] - pos[i][:, None, :]
            d -= L * torch.round(d / L)
            a = (d * d).sum(-1)
            a[torch.arange(len(i), device=pos.device), i] = math.inf
            u, v = torch.nonzero(a <= rc * rc, as_tuple=True)
            yield i[u], v, d[u, v]
        return
    kd = torch.tensor(k, device=pos.device)
    c = torch.floor((pos / L - torch.floor(pos / L)) * kd).long().clamp_(min=0)
    c = torch.minimum(c, kd - 1)
    cell = (c[:, 0] * k[1] + c[:, 1]) * k[2] + c[:, 2]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=int(np.prod(k)))
    first = torch.cumsum(count, 0) - count
    width = int(count.max())
    slot = torch.arange(width, device=pos.device)
    table = torch.where(slot < count[:, None], order[(first[:, None] + slot).clamp(max=n - 1)],
                        torch.full((1, 1), -1, device=pos.device))
    cells = torch.arange(int(np.prod(k)), device=pos.device)
    cx, cy, cz = cells // (k[1] * k[2]), (cells // k[2]) % k[1], cells % k[2]
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                other = (((cx + dx) % k[0]) * k[1] + (cy + dy) % k[1]) * k[2] + (cz + dz) % k[2]
                step = max(1, 2 * rows // (width * width))
                for b in range(0, len(cells), step):
                    i = table[b:b + step][:, :, None].expand(-1, -1, width)
                    j = table[other[b:b + step]][:, None, :].expand(-1, width, -1)
                    ok = (i >= 0) & (j >= 0)
                    yield near(i[ok], j[ok])


def _switch(name, a, on, rc):
    """A switching function's value and 2 dS/da at a = r^2."""
    c2 = rc * rc
    if name == "C2":
        o2 = on * on
        u = c2 - a
        v = u * (c2 - 3.0 * o2 + 2.0 * a)
        s1 = 1.0 / (c2 - o2) ** 3
        inside = a >= o2
        return torch.where(inside, s1 * u * v, torch.ones_like(a)), torch.where(inside, 4.0 * s1 * (u * u - v),
                                                                              torch.zeros_like(a))
    if name == "Shift":
        x = 1.0 - a / c2
        return x * x, -4.0 / c2 * x
    return torch.ones_like(a), torch.zeros_like(a)


def _potential(name, a, qq, A, B, alpha):
    """Energy and force factor (force on j = factor * (x_j - x_i))."""
    if name == "LennardJones":
        r6 = 1.0 / (a * a * a)
        return A * r6 * r6 - B * r6, (12.0 * A * r6 * r6 - 6.0 * B * r6) / a
    if name == "Coulomb":
        e = qq / torch.sqrt(a)
        return e, e / a
    r = torch.sqrt(a)
    x = alpha * r
    t = 1.0 / (1.0 + 0.3275911 * x)                      # Abramowitz & Stegun 7.1.26, as the force defines it
    p = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    g = qq * torch.exp(-x * x)
    e = p * g / r
    return e, (e + 2.0 * alpha / math.sqrt(math.pi) * g) / a


class _Exact:
    """Forces, energies, virials and derivatives of one system in FP64."""

    def __init__(self, system, case):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda x, d=torch.float64: torch.tensor(np.asarray(x), dtype=d, device=dev)
        self.s, self.case, self.dev = system, case, dev
        self.lengths = [float(x) for x in system.box_lengths]
        self.q, self.type = t(system.scaled_charge), t(system.atom_type, torch.int64)
        self.mol, self.lj = t(system.molecule, torch.int64), t(system.lj_table)
        ex = t(system.exclusions.reshape(-1, 3), torch.int64)
        self.excl = ex
        key, where = torch.sort(ex[:, 0] * system.n_atoms + ex[:, 1])
        self.key, self.cls = key, t(system.exclusion_check, torch.int64)[where]

    def classes(self, i, j):
        n = self.s.n_atoms
        out = torch.zeros_like(i)
        if len(self.key):
            m = torch.nonzero(self.mol[i] == self.mol[j]).squeeze(1)
            k = torch.minimum(i[m], j[m]) * n + torch.maximum(i[m], j[m])
            p = torch.searchsorted(self.key, k).clamp(max=len(self.key) - 1)
            out[m] = torch.where(self.key[p] == k, self.cls[p], torch.zeros_like(k))
        return out

    def pair_terms(self, pos, center=None, v=None):
        """Sums over the cutoff forces; center: molecule positions; v: the
        vector of a Hessian-vector product, with the parameter gradients."""
        n, nt, rc = pos.shape[0], self.lj.shape[0], self.case["rc"]
        on, alpha, csf = _switchon(rc), _alpha(rc), float(self.s.csf)
        L = torch.tensor(self.lengths, dtype=torch.float64, device=self.dev)
        z = lambda *sh: torch.zeros(*sh, dtype=torch.float64, device=self.dev)
        out = {"forces": z(n, 3), "lj": z(()), "coulomb": z(()), "virial": z(3, 3), "molvir": z(3, 3), "hv": z(n, 3),
               "dq": z(n), "dlj": z(nt * nt, 4)}
        for i, j, d in _pairs(pos, self.lengths, rc):
            cls = self.classes(i, j)
            keep = cls != systems.EXCLUSION_FULL
            i, j, d, cls = i[keep], j[keep], d[keep], cls[keep]
            mod = cls == systems.EXCLUSION_MODIFIED
            a = (d * d).sum(-1)
            kappa = torch.where(mod, torch.full_like(a, csf), torch.ones_like(a))
            tt = self.type[i] * nt + self.type[j]
            par = self.lj.reshape(-1, 4)[tt]
            A, B = torch.where(mod, par[:, 2], par[:, 0]), torch.where(mod, par[:, 3], par[:, 1])
            factor = torch.zeros_like(a)
            slope = torch.zeros_like(a)
            for force in _terms(self.case)[0]:
                for pot, sw in force:
                    if v is not None:
                        b = a.clone().requires_grad_(True)
                        e, f = _potential(pot, b, kappa * self.q[i] * self.q[j], A, B, alpha)
                        s, ds = _switch(sw, b, on, rc)
                        ft = f * s - e * ds
                        slope += torch.autograd.grad(ft.sum(), b)[0]
                        e, ft = (e * s).detach(), ft.detach()
                        s = s.detach()
                        if pot == "LennardJones":
                            r6 = 1.0 / (a * a * a)
                            g = torch.stack([r6 * r6 * s, -r6 * s], 1) * 0.5
                            for m, cols in ((~mod, slice(0, 2)), (mod, slice(2, 4))):
                                out["dlj"][:, cols].index_add_(0, tt[m], g[m])
                        else:
                            unit = _potential(pot, a, kappa, A, B, alpha)[0] * s
                            out["dq"].index_add_(0, i, self.q[j] * unit)
                    else:
                        e, f = _potential(pot, a, kappa * self.q[i] * self.q[j], A, B, alpha)
                        s, ds = _switch(sw, a, on, rc)
                        ft = f * s - e * ds
                        e = e * s
                    out["lj" if pot == "LennardJones" else "coulomb"] += 0.5 * e.sum()
                    factor += ft
            fij = d * factor[:, None]
            out["forces"].index_add_(0, i, -fij)
            out["virial"] += 0.5 * fij.T @ d
            if center is not None:
                m = self.mol[i] != self.mol[j]
                dc = center[self.mol[j[m]]] - center[self.mol[i[m]]]
                dc = dc - L * torch.round(dc / L)
                out["molvir"] += 0.5 * fij[m].T @ dc
            if v is not None:
                dv = v[j] - v[i]
                out["hv"].index_add_(0, i, factor[:, None] * dv + 2.0 * (slope * (d * dv).sum(-1))[:, None] * d)
        return out

    def splines(self, w):
        """B-spline values theta[0 .. order-1] at the fractions w, by the
        Cox-de Boor recursion."""
        th = [1.0 - w, w]
        for k in range(3, self.case["order"] + 1):
            th = self._raise(th, w, k)
        return torch.stack(th, -1)

    @staticmethod
    def _raise(th, w, k):
        """Order k - 1 -> k; th[m] = M_{k-1}(w + k - 2 - m): weight of the
        m-th point of the support, counted from its lower end."""
        out = []
        for m in range(k):
            u = w + (k - 1 - m)                          # argument of M_k at point m
            lo = th[m - 1] if m >= 1 else 0.0            # M_{k-1}(u)
            hi = th[m] if m < k - 1 else 0.0             # M_{k-1}(u - 1)
            out.append((u * lo + (k - u) * hi) / (k - 1.0))
        return out

    def reciprocal(self, pos, q, want_virial=False):
        """Energy of the smooth PME reciprocal term (differentiable) and its
        virial."""
        K = _grid(self.s) if "grid" not in self.case else (self.case["grid"],) * 3
        p, alpha = self.case["order"], _alpha(self.case["rc"])
        V = float(np.prod(self.lengths))
        idx, wts = [], []
        for c in range(3):
            x = pos[:, c] * (K[c] / self.lengths[c])
            x = x - K[c] * torch.floor(x.detach() / K[c])
            base = torch.floor(x.detach())
            wts.append(self.splines(x - base))
            idx.append((base.long()[:, None] - (p - 1) // 2 + torch.arange(p, device=self.dev)) % K[c])
        Q = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=self.dev)
        for u in range(p):                               # one plane of the support at a time
            w = (q * wts[0][:, u])[:, None, None] * wts[1][:, :, None] * wts[2][:, None, :]
            at = (idx[0][:, u, None, None] * K[1] + idx[1][:, :, None]) * K[2] + idx[2][:, None, :]
            Q = Q.index_add(0, at.reshape(-1), w.reshape(-1))
        S = torch.fft.rfftn(Q.view(*K))
        m, b2 = [], []
        for c in range(3):
            k = torch.arange(K[c], device=self.dev)
            k = torch.where(k <= K[c] // 2, k, k - K[c]).double()
            m.append(k / self.lengths[c])
            th = self.splines(torch.zeros(1, dtype=torch.float64, device=self.dev))[0]
            ph = 2.0 * math.pi * torch.arange(K[c], device=self.dev).double()[:, None] * torch.arange(
                p, device=self.dev).double() / K[c]
            b2.append(1.0 / ((th * torch.cos(ph)).sum(1) ** 2 + (th * torch.sin(ph)).sum(1) ** 2))
        h = K[2] // 2 + 1
        mx, my, mz = m[0][:, None, None], m[1][None, :, None], m[2][None, None, :h].abs()
        m2 = mx * mx + my * my + mz * mz
        m2[0, 0, 0] = 1.0
        fac = math.pi ** 2 / alpha ** 2
        theta = (torch.exp(-fac * m2) / (math.pi * V * m2) * b2[0][:, None, None] * b2[1][None, :, None]
                 * b2[2][None, None, :h])
        theta[0, 0, 0] = 0.0
        twice = torch.full((h,), 2.0, dtype=torch.float64, device=self.dev)
        twice[0] = 1.0
        if K[2] % 2 == 0:
            twice[-1] = 1.0
        e = 0.5 * (S.real ** 2 + S.imag ** 2) * theta * twice
        vir = None
        if want_virial:
            ed = e.detach()
            g = 2.0 * (1.0 / m2 + fac)
            vir = torch.zeros(3, 3, dtype=torch.float64, device=self.dev)
            comp = (mx, my, mz)
            for a in range(3):
                for b in range(3):
                    vir[a, b] = (ed * ((1.0 if a == b else 0.0) - g * comp[a] * comp[b])).sum()
        return e.sum(), vir

    def correction(self, pos, q):
        """Excluded pairs, self and charged-system terms (differentiable), and
        the excluded pairs' vectors."""
        alpha, csf = _alpha(self.case["rc"]), float(self.s.csf)
        L = torch.tensor(self.lengths, dtype=torch.float64, device=self.dev)
        i, j, cls = self.excl[:, 0], self.excl[:, 1], self.excl[:, 2]
        d = pos[j] - pos[i]
        d = d - (L * torch.round(d / L)).detach()
        r = torch.sqrt((d * d).sum(-1))
        scale = torch.where(cls == systems.EXCLUSION_MODIFIED, torch.full_like(r, 1.0 - csf), torch.ones_like(r))
        pair = -(q[i] * q[j] * scale * torch.erf(alpha * r) / r)
        e = pair.sum() - alpha / math.sqrt(math.pi) * (q * q).sum()
        return e, pair, r, d

    def evaluate(self, pos, center=None):
        out = self.pair_terms(pos, center)
        forces, coulomb, virial, molvir = out["forces"], out["coulomb"], out["virial"], out["molvir"]
        if _terms(self.case)[1]:
            x = pos.clone().requires_grad_(True)
            e, vir = self.reciprocal(x, self.q, True)
            fr = -torch.autograd.grad(e, x)[0]
            ec, pair, r, d = self.correction(x, self.q)
            gr = torch.autograd.grad(pair.sum(), r, retain_graph=True)[0]
            fd = -(gr / r)[:, None] * d
            fc = -torch.autograd.grad(ec, x)[0]
            forces = forces + fr + fc
            coulomb = coulomb + e.detach() + ec.detach()
            virial = virial + vir + fd.detach().T @ d.detach()
            if center is not None:
                L = torch.tensor(self.lengths, dtype=torch.float64, device=self.dev)
                dm = center[self.mol] - pos
                dm = dm - L * torch.round(dm / L)
                molvir = molvir + vir + fr.T @ dm
        energies = torch.cat([out["lj"].reshape(1), coulomb.reshape(1), _sym(virial)])
        return {"forces": forces, "energies": energies, "molvir": _sym(molvir)}

    def adjoint(self, pos, v):
        out = self.pair_terms(pos, None, v)
        hv, dq = out["hv"], out["dq"]
        if _terms(self.case)[1]:
            x, q = pos.clone().requires_grad_(True), self.q.clone().requires_grad_(True)
            e = self.reciprocal(x, q)[0] + self.correction(x, q)[0]
            gx, gq = torch.autograd.grad(e, (x, q), create_graph=True)
            hv = hv + torch.autograd.grad((gx * v).sum(), x)[0]
            dq = dq + gq.detach()
        nt = self.lj.shape[0]
        return {"dE_dq": dq, "dE_dlj": out["dlj"].view(nt, nt, 4), "hv": hv,
                "pair_energies": torch.stack([out["lj"], out["coulomb"]])}


def _sym(t):
    """The nine slots as they are accumulated: the upper triangle, mirrored."""
    u = torch.triu(t)
    return (u + torch.triu(t, 1).T).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "rigid" or case.get("forces") == "tables":
        return None               # defined by their own iterations and tables, in FP64 throughout
    if kind == "batch":
        parts = []
        for system, grid in _members(case, seed):
            x = _Exact(system, dict(case, forces="ewald", order=4, grid=grid))
            parts.append(x.evaluate(torch.tensor(system.positions, device=x.dev)))
        return {"forces": torch.cat([p["forces"] for p in parts]), "energies": torch.stack([p["energies"] for p in parts])}
    system = _system(case, seed)
    if kind == "fluid":
        return _exact_run(case, system, seed)
    x = _Exact(system, case)
    pos = torch.tensor(system.positions, device=x.dev)
    if kind == "adjoint":
        v = np.random.default_rng(seed + 1).normal(size=system.positions.shape)
        return x.adjoint(pos, torch.tensor(v, device=x.dev))
    center = None
    if case.get("molvir"):
        m = np.zeros(int(system.molecule.max()) + 1)
        c = np.zeros((len(m), 3))
        np.add.at(m, system.molecule, system.mass)
        np.add.at(c, system.molecule, system.positions * system.mass[:, None])
        center = torch.tensor(c / m[:, None], device=x.dev)
    r = x.evaluate(pos, center)
    molvir = r.pop("molvir")
    if center is not None:
        r["molecular_virial"] = molvir
    return r


def _exact_run(case, system, seed):
    """The Leapfrog's kicks and drifts over the forces above."""
    x = _Exact(system, dict(case, forces="fused"))
    pos = torch.tensor(system.positions, device=x.dev)
    vel = torch.tensor(integrate_velocities(system, seed), device=x.dev)
    m = torch.tensor(system.mass, device=x.dev)[:, None]
    h = 1.0 / TIMEFACTOR
    r = x.evaluate(pos)
    for _ in range(case["steps"]):
        vel = vel + 0.5 * h * r["forces"] / m
        pos = pos + h * vel
        r = x.evaluate(pos)
        vel = vel + 0.5 * h * r["forces"] / m
    return {"positions": pos, "velocities": vel, "forces": r["forces"], "energies": r["energies"]}


def integrate_velocities(system, seed):
    """The seeded 300 K velocities that the run starts from."""
    m = np.asarray(system.mass)
    v = np.random.default_rng(seed + 1).normal(size=(len(m), 3)) * np.sqrt(0.001987191 * 300.0 / m)[:, None]
    return v - (m[:, None] * v).sum(0) / m.sum()
