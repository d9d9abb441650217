"""The work a user has this engine do, as cases that can be timed and compared.

Every case goes through the package's public entry points (Engine, Deck,
Batch): frozen-field bulk boxes, self-consistent devices from decks, the
frozen-potential heat phase, a Poisson solve on its own, the quantum
correction and a batch of small simulations.  Sizes are those of the
benchmark, the tests and the precision study, or generic.

The band tables an engine reads are computed here, since none ship with the
repository: silicon's bands from the local empirical pseudopotential of
Cohen and Bergstresser (Phys. Rev. 141, 789, 1966) on tetrahedral meshes of
the irreducible wedge, graded towards the band edges and about as large as
the tables the engine is meant for (54,000 tetrahedra), with the densities
of states of the linear tetrahedron method.
"""
from __future__ import annotations

import functools
import itertools
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("c-mc_electron_b200"))  # the package is not installed: its folder in this checkout

import mcb200  # noqa: E402
from mcb200 import FLIGHT_FP32, FLIGHT_FP64, Batch, Deck, Engine, batching, decks  # noqa: E402
from mcb200.workloads import motion_rules, uniform_fields  # noqa: E402

KELVIN = 300.0
PRECISION = {32: FLIGHT_FP32, 64: FLIGHT_FP64}


def listed():
    return [
        # a small contacted bar, Poisson every step: the smallest device, launches and latency
        dict(name="bar_fp64", kind="deck", deck="bar", nx=8, ny=10, nz=6, electrons=4000, holes=0, vd=0.3, bits=64,
             steps=20, poisson_every=1, window=1),
        # the smallest simulations of a sweep: a bulk box with few carriers
        dict(name="bulk_5k_fp32", kind="bulk", nx=20, ny=20, nz=20, particles=5000, kv_cm=30.0, bits=32, steps=20),
        # the velocity-field study: a box 1 um along the field, at its largest field
        dict(name="bulk_100k_fp64", kind="bulk", nx=200, ny=10, nz=10, particles=100000, kv_cm=100.0, bits=64,
             steps=20),
        # large ensembles, a store that does not fit in L2, in both flight precisions
        dict(name="bulk_2m_fp32", kind="bulk", nx=40, ny=20, nz=20, particles=2000000, kv_cm=10.0, bits=32, steps=10),
        dict(name="bulk_2m_fp64", kind="bulk", nx=40, ny=20, nz=20, particles=2000000, kv_cm=10.0, bits=64, steps=10),
        # the n-FinFET (20 nm gate, 511,200 carriers) over one refresh period with its statistics
        dict(name="finfet20_fp32", kind="deck", deck="finfet", lg_nm=20, electrons=300000, holes=50000, floor=3,
             vg=0.8, bits=32, steps=50, poisson_every=10, window=1),
        dict(name="finfet20_fp64", kind="deck", deck="finfet", lg_nm=20, electrons=300000, holes=50000, floor=3,
             vg=0.8, bits=64, steps=50, poisson_every=10, window=1),
        # a bias point of a sweep: short gate, few carriers, no statistics
        dict(name="finfet15_fp32", kind="deck", deck="finfet", lg_nm=15, electrons=20000, holes=3000, floor=1, vg=0.4,
             bits=32, steps=20, poisson_every=10, window=0),
        # the heat phase: the mean potential frozen, phonon heat and statistics tallied
        dict(name="heat30_fp32", kind="deck", deck="finfet", lg_nm=30, electrons=300000, holes=50000, floor=3, vg=0.8,
             bits=32, steps=20, poisson_every=0, window=1),
        # quantum-corrected FinFET
        dict(name="quantum20_fp64", kind="deck", deck="finfet", lg_nm=20, electrons=100000, holes=10000, floor=1,
             vg=0.8, bits=64, steps=20, poisson_every=10, window=0, quantum=1),
        # deposition and the first Poisson solve of a bias point, from a flat potential
        dict(name="solve_288k", kind="solve", nx=80, ny=90, nz=40, particles=600000, vg=0.8, vd=0.7),
        # a batch of small simulations
        dict(name="batch32_fp32", kind="batch", members=32, n_min=5000, n_max=50000, bits=32, steps=20),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bulk", "bulk", "bar", "finfet", "finfet", "solve", "batch"])
    bits = rng.choice([32, 64])
    if kind == "bulk":
        return dict(kind="bulk", nx=rng.randint(20, 80), ny=rng.randint(10, 40), nz=rng.randint(10, 50),
                    particles=log_int(5000, 1500000), kv_cm=round(rng.uniform(1.0, 100.0), 2), bits=bits, steps=10)
    if kind == "bar":
        return dict(kind="deck", deck="bar", nx=rng.randint(5, 20), ny=rng.randint(8, 24), nz=rng.randint(5, 20),
                    electrons=log_int(2000, 100000), holes=rng.choice([0, 1000]), vd=round(rng.uniform(0.05, 0.7), 2),
                    bits=bits, steps=20, poisson_every=rng.choice([1, 5]), window=rng.choice([0, 1]))
    if kind == "finfet":
        return dict(kind="deck", deck="finfet", lg_nm=rng.randint(12, 30), electrons=log_int(5000, 400000),
                    holes=log_int(1000, 50000), floor=rng.choice([1, 3]), vg=round(rng.uniform(0.0, 0.8), 2), bits=bits,
                    steps=20, poisson_every=rng.choice([0, 10, 10, 20]), window=rng.choice([0, 1]),
                    quantum=rng.choice([0, 0, 0, 1]))
    if kind == "solve":
        return dict(kind="solve", nx=rng.randint(11, 80), ny=rng.randint(13, 90), nz=rng.randint(9, 40),
                    particles=log_int(20000, 600000), vg=round(rng.uniform(0.0, 0.8), 2),
                    vd=round(rng.uniform(0.05, 0.7), 2))
    return dict(kind="batch", members=rng.randint(6, 32), n_min=5000, n_max=log_int(10000, 50000), bits=bits, steps=20)


# ---- silicon band tables -------------------------------------------------------
LATTICE_M = 5.43e-10
PLANCK_EV_S = 6.582119e-16  # hbar
ENERGY_POINTS = 7501        # the engine's energy tables: 1 meV steps
VERTEX = {"G": (0, 0, 0), "X": (1, 0, 0), "L": (0.5, 0.5, 0.5), "W": (1, 0.5, 0), "K": (0.75, 0.75, 0),
          "U": (1, 0.25, 0.25), "D": (0.85, 0, 0)}  # D: the conduction-band minimum
# the outer planes of the wedge kx >= ky >= kz >= 0, in the order of the table file's codes -1 .. -5
PLANES = [((0, 0, 1), 0.0), ((1, -1, 0), 0.0), ((0, 1, -1), 0.0), ((1, 1, 1), 1.5), ((1, 0, 0), 1.0)]
ELECTRON_MESH = (["DGKL", "DKLW", "DLWU", "DWUX"], 12, 1.5)  # tetrahedra of the wedge, subdivisions, grading
HOLE_MESH = (["GKLW", "GLWU", "GWUX"], 13, 1.5)


def wedge_mesh(coarse, n, grading):
    """Points [p, 3] (units of 2 pi / a) and tetrahedra [t, 4] of the wedge:
    every coarse tetrahedron cut into n^3, its layers drawn towards its first
    vertex as (distance)^grading.  Shared vertices come in the same order in
    every coarse tetrahedron, so the cuts meet on their faces."""
    index, points, tets = {}, [], []

    def point(v, abc):
        w = np.array([n - abc[0], abc[0] - abc[1], abc[1] - abc[2], abc[2]]) / n
        p = w @ v
        if abc[0]:
            p = v[0] + (abc[0] / n) ** (grading - 1.0) * (p - v[0])
        key = tuple(np.round(p, 9) + 0.0)
        if key not in index:
            index[key] = len(points)
            points.append(p)
        return index[key]

    for names in coarse:
        v = np.array([VERTEX[c] for c in names], dtype=float)
        for corner in itertools.product(range(n), repeat=3):
            for order in itertools.permutations(range(3)):
                path = [np.array(corner)]
                for axis in order:
                    path.append(path[-1] + np.eye(3, dtype=int)[axis])
                if all(n >= p[0] >= p[1] >= p[2] >= 0 for p in path):
                    tets.append([point(v, tuple(p)) for p in path])
    return np.array(points), np.array(tets)


def silicon_bands(k):
    """Energies [k, 8] in eV of the four valence and four lowest conduction
    bands (local pseudopotential, form factors in Ry, origin between the two
    atoms so that the Hamiltonian is real)."""
    ry, form = 13.605693, {3: -0.21, 8: 0.04, 11: 0.08}
    kinetic = 3.80998212 * (2 * math.pi / (LATTICE_M * 1e10)) ** 2  # hbar^2 / 2m (eV A^2) in units of (2 pi / a)^2
    g = np.array([v for v in itertools.product(range(-4, 5), repeat=3)
                  if len({c % 2 for c in v}) == 1 and sum(c * c for c in v) <= 12])
    d = g[:, None, :] - g[None, :, :]
    v = np.vectorize(lambda s: form.get(s, 0.0))((d ** 2).sum(-1)) * np.cos(math.pi / 4 * d.sum(-1)) * ry
    out = np.empty((len(k), 8))
    for i, q in enumerate(k):
        out[i] = np.linalg.eigvalsh(v + np.diag(kinetic * ((q + g) ** 2).sum(-1)))[:8]
    return out


def neighbours(points, tets):
    """For each tetrahedron's face opposite vertex f: the tetrahedron behind it
    (1-based) or the negative code of the wedge's outer plane."""
    out = np.zeros((len(tets), 4), dtype=int)
    open_faces = {}
    for t, tet in enumerate(tets):
        for f in range(4):
            key = tuple(sorted(np.delete(tet, f)))
            if key in open_faces:
                t2, f2 = open_faces.pop(key)
                out[t, f], out[t2, f2] = t2 + 1, t + 1
            else:
                open_faces[key] = (t, f)
    for key, (t, f) in open_faces.items():
        p = points[list(key)]
        out[t, f] = next(-1 - i for i, (nrm, at) in enumerate(PLANES) if np.all(np.abs(p @ np.array(nrm) - at) < 1e-9))
    return out


def density_of_states(points, tets, energy):
    """(DOS per spin in 1/(eV m^3), largest area / velocity of a tetrahedron in
    1/m^2 / (m/s)) at the 1 meV grid: the volume a tetrahedron holds below E
    grows as the cut's area over the gradient."""
    e = np.sort(energy[tets], axis=1)
    p = points[tets]
    vol = np.abs(np.linalg.det(p[:, 1:] - p[:, :1])) / 6.0
    lo = np.clip(np.ceil(e[:, 0] * 1e3).astype(int), 0, ENERGY_POINTS)
    hi = np.clip(np.ceil(e[:, 3] * 1e3).astype(int), 0, ENERGY_POINTS)
    t = np.repeat(np.arange(len(tets)), hi - lo)
    i = np.arange(len(t)) - np.repeat(np.cumsum(hi - lo) - (hi - lo), hi - lo) + lo[t]
    x = i * 1e-3
    e0, e1, e2, e3 = e[t].T
    gap = lambda a: np.maximum(a, 1e-9)  # noqa: E731
    low = (x - e0) ** 2 / (gap(e1 - e0) * gap(e2 - e0) * gap(e3 - e0))
    mid = ((e1 - e0) + 2 * (x - e1) - (x - e1) ** 2 * (e2 - e0 + e3 - e1) / (gap(e2 - e1) * gap(e3 - e1))) / \
        (gap(e2 - e0) * gap(e3 - e0))
    top = (e3 - x) ** 2 / (gap(e3 - e0) * gap(e3 - e1) * gap(e3 - e2))
    grown = 3.0 * vol[t] * np.where(x <= e1, low, np.where(x < e2, mid, top))
    dos = np.bincount(i, grown, ENERGY_POINTS) * 48.0 / LATTICE_M ** 3
    biggest = np.zeros(ENERGY_POINTS)
    np.maximum.at(biggest, i, grown)
    return dos, biggest * (2 * math.pi / LATTICE_M) ** 3 * PLANCK_EV_S


@functools.lru_cache(maxsize=None)
def silicon():
    """The tables as arrays: bands of electrons (4), holes (3) and oxide
    electrons (1), each with its own copy of its mesh's points."""
    ep, et = wedge_mesh(*ELECTRON_MESH)
    hp, ht = wedge_mesh(*HOLE_MESH)
    ee, eh = silicon_bands(ep), silicon_bands(hp)
    top = silicon_bands(np.zeros((1, 3)))[0, 3]
    bands = [(ep, et, ee[:, 4 + b] - ee[:, 4].min()) for b in range(4)]
    bands += [(hp, ht, top - eh[:, 3 - b]) for b in range(3)]
    bands += [(hp, ht, 8.5 * (hp ** 2).sum(1))]
    near = {id(ep): neighbours(ep, et), id(hp): neighbours(hp, ht)}
    k, energy, tet, neib, band, dos, most = [], [], [], [], [], [], []
    node0 = tet0 = 0
    for b, (p, t, e) in enumerate(bands):
        e = np.maximum(np.round(e, 6), 0.0)
        order = np.argsort(e[t], axis=1, kind="stable")  # vertices in ascending energy, faces with them
        tet.append(np.take_along_axis(t, order, 1) + node0)
        nb = np.take_along_axis(near[id(p)], order, 1)
        neib.append(np.where(nb > 0, nb + tet0, nb))
        band.append(np.full(len(t), b))
        k.append(p)
        energy.append(e)
        d, m = density_of_states(p, t, e)
        dos.append(d)
        most.append(m)
        node0 += len(p)
        tet0 += len(t)
    return dict(k=np.concatenate(k), energy=np.concatenate(energy), tet=np.concatenate(tet), neib=np.concatenate(neib),
                band=np.concatenate(band), dos=np.array(dos), most=np.array(most))


def write_tables(folder):
    """The table files an engine reads (bs.si.asc, zd.si.asc and the phonon
    dispersion tables of the quantum correction) into `folder`."""
    s = silicon()

    def put(f, values, fmt):
        f.write("\n".join(fmt % v for v in np.asarray(values).reshape(-1)) + "\n")

    with open(os.path.join(folder, "bs.si.asc"), "w") as f:
        f.write("4 3 1\n%d\n" % len(s["k"]))
        for axis in range(3):
            put(f, s["k"][:, axis], "%.15g")
        put(f, s["energy"], "%.6f")
        f.write("%d\n" % len(s["tet"]))
        put(f, s["tet"].T + 1, "%d")
        put(f, s["neib"].T, "%d")
        put(f, s["band"] + 1, "%d")
    with open(os.path.join(folder, "zd.si.asc"), "w") as f:
        for table in (s["dos"], s["most"]):
            f.write("%d\n" % (ENERGY_POINTS - 1))
            for i in range(ENERGY_POINTS):
                f.write("%.3f " % (i * 1e-3) + " ".join("%.9e" % v for v in table[:, i]) + "\n")
    # final-energy distributions of the dispersive phonons: each column sums to one over its rows
    for name, rows, cols in (("kloem", 201, 120), ("kloab", 201, 110), ("ktoem", 51, 160), ("ktoab", 51, 150),
                             ("klaem", 51, 160), ("klaab", 51, 150)):
        w = np.exp(-np.arange(rows) / (0.2 * rows))
        with open(os.path.join(folder, name + ".txt"), "w") as f:
            put(f, np.tile(w / w.sum(), cols), "%.9f")


@functools.lru_cache(maxsize=None)
def tables_owner():
    """The engine whose band tables every other one shares, as a program with
    several simulations has it."""
    with tempfile.TemporaryDirectory() as folder:
        write_tables(folder)
        return Engine(table_dir=folder, kelvin=KELVIN, max_particles=1)


# ---- what a program has in hand ------------------------------------------------
def prepare(case, seed):
    return {"bulk": prepare_bulk, "deck": prepare_deck, "solve": prepare_solve, "batch": prepare_batch}[case["kind"]](
        case, seed)


def prepare_bulk(case, seed):
    m = batching.bulk_member(tables_owner(), case["nx"], case["ny"], case["nz"], case["kv_cm"], case["particles"],
                             1 + seed, PRECISION[case["bits"]])
    m.eng.stat_begin(1)
    return dict(case=case, eng=m.eng, dt=m.cfg["dt"], seed=1 + seed, step=0)


def prepare_deck(case, seed):
    root = tables_owner()
    with tempfile.TemporaryDirectory() as folder:
        if case["deck"] == "bar":
            d = decks.contact_bar(folder, nx=case["nx"], ny=case["ny"], nz=case["nz"], vd=case["vd"],
                                  electrons=case["electrons"], holes=case["holes"], kelvin=KELVIN, surfaces=True)
        else:
            d = decks.finfet(folder, electrons=case["electrons"], holes=case["holes"], vg=case["vg"],
                             lg_nm=float(case["lg_nm"]), min_per_cell=(case["floor"], 1 if case["floor"] > 1 else 0),
                             mr_step=50, kelvin=KELVIN, quantum=(3.0, 0.5, 3.1, 0) if case.get("quantum") else None)
        deck = Deck(d["input"])
    deck.prepare(root)
    carriers = int(deck.int_array("electron_num").sum() + deck.int_array("hole_num").sum())
    eng = Engine(max_particles=2 * carriers + 65536, precision=PRECISION[case["bits"]], like=root)
    deck.apply(eng)
    deck.seed(eng, 1 + seed)
    info = deck.info()
    s = dict(case=case, eng=eng, dt=info["dt"], seed=1 + seed, step=0, eeff=deck.int_array("eeff_direction"),
             surface=dict(delta_m=0.4e-9, ail_m=1.5e-9, roughness=info["flag_surface_roughness"],
                          phonon=info["flag_surface_phonon"]),
             targets=(deck.int_array("refresh_electrons"), deck.int_array("refresh_holes")))
    deck.close()
    if case["deck"] == "finfet":
        eng.set_refresh_targets(*s["targets"])
    if case.get("quantum"):
        eng.set_quantum_correction(enable=True, setup=False)
    eng.deposit()
    eng.solve_poisson(1e-10, 20000)
    if case["poisson_every"] == 0:
        eng._check(mcb200.lib().mcb200_set_heat_tally(eng._ctx, 1), "set_heat_tally")
    return s


def gated_bar(case):
    """Mesh widths (m), materials, doping (1/m^3) and contact planes of a gated
    n+ / p / n+ silicon bar under a thin oxide: finer cells towards the gate
    (x), around the channel (y) and in mid-width (z)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    grade = lambda n, at, ratio: 0.5e-9 * (1.0 + ratio * np.abs((np.arange(n) + 0.5) / n - at))  # noqa: E731
    dx, dy, dz = grade(nx, 0.0, 2.0), grade(ny, 0.5, 3.0), grade(nz, 0.5, 2.0)
    oxide = max(1, nx // 20)
    j, i, _ = np.meshgrid(np.arange(ny), np.arange(nx), np.arange(nz), indexing="ij")  # cell order (j, i, k)
    silicon_cell = i >= oxide
    lead = np.minimum(j, ny - 1 - j) < ny // 4
    donor = np.where(silicon_cell & lead, 1e26, 0.0)
    acceptor = np.where(silicon_cell & ~lead, 1e23, 0.0)
    planes = [(0, oxide, nx, 0, 0, 0, nz), (1, oxide, nx, ny, ny, 0, nz), (2, 0, 0, ny // 4, ny - ny // 4, 0, nz)]
    volts = [(0.0, 0.0), (case["vd"], 0.0), (case["vg"], -0.46)]  # applied, work-function difference
    return (dx, dy, dz), np.where(silicon_cell, 3, 2).astype(np.int32), donor, acceptor, planes, volts


def scales():
    """The engine's normalised units at KELVIN, from the physical constants."""
    ec, em, c, e0, kb = 1.602176e-19, 9.109383e-31, 299792458.0, 8.854187817e-12, 8.617343e-5
    ev0 = kb * KELVIN
    spr0 = PLANCK_EV_S / math.sqrt(em / ec * ev0)
    fine = ec / (PLANCK_EV_S * c * 4.0 * math.pi * e0)
    speed = c / (spr0 / (PLANCK_EV_S / ev0))
    return dict(ev0=ev0, spr0=spr0, conc0=spr0 ** -3, eps=1.0 / (4.0 * math.pi * speed * fine))


def gated_bar_carriers(case, seed):
    """Electrons for gated_bar, grouped by cell: numbers follow the charge the
    cells hold (leads full, channel thin) with counting noise."""
    (dx, dy, dz), material, donor, _, _, _ = gated_bar(case)
    rng = np.random.default_rng(seed)
    sc = scales()
    dx, dy, dz = (w / sc["spr0"] for w in (dx, dy, dz))
    held = np.where(material == 3, np.maximum(donor, 2e24), 0.0) / sc["conc0"] * \
        (dy[:, None, None] * dx[None, :, None] * dz[None, None, :])
    cell = np.sort(rng.choice(held.size, case["particles"], p=held.ravel() / held.sum()))
    j, r = np.divmod(cell, case["nx"] * case["nz"])
    i, k = np.divmod(r, case["nz"])
    u = rng.random((3, len(cell)))
    edge = [np.concatenate([[0.0], np.cumsum(w)]) for w in (dx, dy, dz)]
    pos = [e[a] + f * w[a] for e, w, a, f in zip(edge, (dx, dy, dz), (i, j, k), u)]
    charge = np.full(len(cell), -held.sum() / len(cell)) * rng.uniform(0.5, 1.5, len(cell))
    zero = np.zeros(len(cell))
    none = np.zeros(len(cell), dtype=np.int32)
    return dict(x=pos[0], y=pos[1], z=pos[2], kx=zero + 0.85, ky=zero + 0.01, kz=zero + 0.005, charge=charge,
                energy=zero + 1.0, i=i.astype(np.int32), j=j.astype(np.int32), k=k.astype(np.int32), itet=none, isym=none,
                type=none, uid=np.arange(len(cell), dtype=np.uint32)), (dx, dy, dz), edge


def prepare_solve(case, seed):
    _, material, donor, acceptor, planes, volts = gated_bar(case)
    p, widths, edge = gated_bar_carriers(case, seed)
    sc = scales()
    eng = Engine(max_particles=case["particles"] + 4096, like=tables_owner())
    eng.set_mesh(*edge, *widths)
    donor, acceptor = donor / sc["conc0"], acceptor / sc["conc0"]
    eng.set_cells(motion_rules(case["nx"], case["ny"], case["nz"]), np.abs(donor - acceptor))
    eng.set_device(material.ravel(), donor.ravel(), acceptor.ravel(), [v[0] / sc["ev0"] for v in volts],
                   [v[1] / sc["ev0"] for v in volts], planes)
    eng.upload(p)
    return dict(case=case, eng=eng, flat=np.zeros(eng.mesh.nnodes))


def prepare_batch(case, seed):
    shapes = np.random.default_rng(case["members"])  # the sweep's simulations; `seed` sets their fields and ensembles
    rng = np.random.default_rng(seed)
    root = tables_owner()
    members = []
    for _ in range(case["members"]):
        n = int(math.exp(shapes.uniform(math.log(case["n_min"]), math.log(case["n_max"]))))
        nx, ny, nz = (int(shapes.integers(20, 41)) for _ in range(3))
        members.append(batching.bulk_member(root, nx, ny, nz, float(rng.uniform(1.0, 100.0)), n,
                                            int(rng.integers(1, 1 << 30)), PRECISION[case["bits"]]))
    batch = Batch([(m.eng, m.cfg) for m in members])
    batch.use_graphs(True)
    return dict(case=case, batch=batch, members=members)


# ---- one pass ------------------------------------------------------------------
NODE_SUMS = ["qvx", "qvy", "qvz", "q", "qe"]


def run(state):
    return {"bulk": run_bulk, "deck": run_deck, "solve": run_solve, "batch": run_batch}[state["case"]["kind"]](state)


def run_bulk(s):
    """Time steps, then the drift velocities, energies and counts of the cells."""
    eng = s["eng"]
    for _ in range(s["case"]["steps"]):
        eng.step(s["step"], s["seed"], s["dt"])
        s["step"] += 1
    eng.stat_begin(1)
    eng.stat_accumulate()
    out = {n: eng.stat("electron_" + n) for n in NODE_SUMS}
    out["cell_count"] = eng.stat("cell_count")
    out["tallies"] = eng.tallies()
    return out


def run_deck(s):
    """One window of the self-consistent loop, then its results."""
    case, eng = s["case"], s["eng"]
    every = case["poisson_every"]
    eng.reset_tallies()
    if case["window"]:
        eng.stat_begin(case["steps"])
    for _ in range(case["steps"]):
        if case["window"]:
            eng.stat_accumulate()
        eng.deposit()
        if every and s["step"] % every == 0:
            eng.solve_poisson_async(1e-10, 20000)
        eng.surface_rates(s["eeff"], **s["surface"])
        eng.step(s["step"], s["seed"], s["dt"])
        if case["deck"] == "finfet" and s["step"] % 50 == 49:
            eng.multiple_refresh(*s["targets"], s["step"], s["seed"], wait=False)
        s["step"] += 1
    out = dict(tallies=eng.tallies(), potential=eng.array("potential"), density=eng.array("node_density"))
    if case["window"]:
        for n in NODE_SUMS:
            out["electron_" + n] = eng.stat("electron_" + n)
    return out


def run_solve(s):
    """Deposition and a solve from the flat potential, with the fields."""
    eng = s["eng"]
    eng.set_potential(s["flat"])
    eng.deposit()
    eng.solve_poisson_async(1e-10, 20000)
    return {n: eng.array(n) for n in ("cell_charge_e", "node_density", "rho", "potential", "efield")}


def run_batch(s):
    """Time steps of every member, then each member's counters."""
    s["batch"].run(s["case"]["steps"])
    s["batch"].sync()
    t = [m.eng.tallies() for m in s["members"]]
    return dict(counters=np.array([[v[n] for n in mcb200.COUNTER_NAMES] for v in t]),
                left=np.concatenate([v["lcurrent"] for v in t]), right=np.concatenate([v["rcurrent"] for v in t]))


# ---- results in 64 bits ----------------------------------------------------------
def exact(case, seed):
    """The solve's results from the definitions, in plain numpy and torch.  The
    others follow particles on their own random streams, which have no other
    source of values."""
    if case["kind"] != "solve":
        return None
    _, material, donor, acceptor, planes, volts = gated_bar(case)
    p, (dx, dy, dz), _ = gated_bar_carriers(case, seed)
    sc = scales()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    px, py, pz = nx + 1, ny + 1, nz + 1
    vol = dy[:, None, None] * dx[None, :, None] * dz[None, None, :]
    cell = (p["j"] * nx + p["i"]) * nz + p["k"]
    charge = np.bincount(cell, p["charge"], nx * ny * nz)
    net = (donor - acceptor) / sc["conc0"]
    rho = np.maximum(np.abs(charge) / vol.ravel(), 0.5 * np.abs(net).ravel())
    edge = [np.concatenate([[0.0], np.cumsum(w)]) for w in (dx, dy, dz)]
    f = [(p[a] - e[p[c]]) / w[p[c]] for a, c, e, w in zip("xyz", "ijk", edge, (dx, dy, dz))]
    q = np.zeros(px * py * pz)
    corner_vol, corner_dop = np.zeros((py, px, pz)), np.zeros((py, px, pz))
    share = np.where(material == 3, vol / 8.0, 0.0)
    for b, a, c in itertools.product((0, 1), repeat=3):
        w = (f[0] if a else 1 - f[0]) * (f[1] if b else 1 - f[1]) * (f[2] if c else 1 - f[2])
        q += np.bincount(((p["j"] + b) * px + p["i"] + a) * pz + p["k"] + c, p["charge"] * w, q.size)
        corner_vol[b:ny + b, a:nx + a, c:nz + c] += share
        corner_dop[b:ny + b, a:nx + a, c:nz + c] += share * net
    pvol, pdop = corner_vol.ravel(), corner_dop.ravel()
    density = np.where(pvol > 0, q / np.where(pvol > 0, pvol, 1.0), q)
    # finite volumes: each cell couples the ends of its twelve edges
    eps = sc["eps"] * np.where(material == 3, 11.7, 3.9)
    widths = (dy[:, None, None], dx[None, :, None], dz[None, None, :])
    couple = []
    for ax in range(3):
        o = [a for a in range(3) if a != ax]
        g = 0.25 * eps * widths[o[0]] * widths[o[1]] / widths[ax]
        shape = [py, px, pz]
        shape[ax] -= 1
        c = np.zeros(shape)
        for u, v in itertools.product((0, 1), repeat=2):
            at = [slice(None)] * 3
            at[o[0]], at[o[1]] = slice(u, u + (ny, nx, nz)[o[0]]), slice(v, v + (ny, nx, nz)[o[1]])
            c[tuple(at)] += g
        couple.append(torch.from_numpy(c).cuda())
    rhs = np.where(np.abs(density) > 0, density * pvol + pdop, 0.0).reshape(py, px, pz)
    alfa = np.where(pvol > 1e-16, pdop / np.where(pvol > 1e-16, pvol, 1.0), 0.0) / (2.0 * intrinsic_density())
    built_in = np.arcsinh(alfa).reshape(py, px, pz)
    built_in[-1], built_in[0] = built_in[-2].copy(), built_in[1].copy()
    fixed, value = np.zeros((py, px, pz), dtype=bool), np.zeros((py, px, pz))
    for n, i0, i1, j0, j1, k0, k1 in planes:
        at = (slice(j0, j1 + 1), slice(i0, i1 + 1), slice(k0, k1 + 1))
        fixed[at] = True
        value[at] = (sum(volts[n]) / sc["ev0"]) + built_in[at]
    pot = solve_poisson(couple, torch.from_numpy(rhs).cuda(), torch.from_numpy(fixed).cuda(),
                        torch.from_numpy(value).cuda()).cpu().numpy()
    field = []
    for ax, w in ((1, widths[1]), (0, widths[0]), (2, widths[2])):
        d = np.diff(pot, axis=ax)
        for o in [a for a in range(3) if a != ax]:
            n = d.shape[o] - 1
            d = np.take(d, range(n), o) + np.take(d, range(1, n + 1), o)
        field.append((d / (4.0 * w)).ravel())  # as felt by an electron
    return dict(cell_charge_e=charge, node_density=density, rho=rho, potential=pot.ravel(),
                efield=np.stack(field, 1).ravel())


def intrinsic_density():
    """Normalised n_i: both bands' DOS, linear between its points, times exp(-E)."""
    s, sc = silicon(), scales()
    x = np.arange(ENERGY_POINTS) * (0.001 / sc["ev0"])
    held = []
    for rows in (slice(0, 4), slice(4, 7)):
        d = np.array([float("%.9e" % v) for v in s["dos"][rows].ravel()]).reshape(-1, ENERGY_POINTS).sum(0)
        d = d * sc["ev0"] * sc["spr0"] ** 3
        a, b, u, v = x[:-1], x[1:], d[:-1], d[1:]
        held.append(2.0 * np.sum(((u * b - v * a) * (np.exp(-a) - np.exp(-b)) + (v - u) *
                                  ((a + 1) * np.exp(-a) - (b + 1) * np.exp(-b))) / (b - a)))
    gap = (1.2060 - 2.730e-4 * KELVIN) / sc["ev0"]
    return math.sqrt(held[0] * held[1] * math.exp(-gap))


def solve_poisson(couple, rhs, fixed, value):
    """Conjugate gradients in 64 bits on the free nodes, to the last digits."""
    def apply(x):
        y = torch.zeros_like(x)
        for ax, c in enumerate(couple):
            flux = c * torch.diff(x, dim=ax)
            y.narrow(ax, 0, c.shape[ax]).sub_(flux)
            y.narrow(ax, 1, c.shape[ax]).add_(flux)
        return torch.where(fixed, 0.0, y)

    diag = torch.zeros_like(rhs)
    for ax, c in enumerate(couple):
        diag.narrow(ax, 0, c.shape[ax]).add_(c)
        diag.narrow(ax, 1, c.shape[ax]).add_(c)
    x = torch.where(fixed, value, 0.0)
    r = torch.where(fixed, 0.0, rhs) - apply(x)
    stop = 1e-28 * torch.sum(r * r)
    z = r / diag
    p, rz = z.clone(), torch.sum(r * z)
    for it in range(20000):
        q = apply(p)
        alpha = rz / torch.sum(p * q)
        x += alpha * p
        r -= alpha * q
        if it % 50 == 49:
            if torch.sum(r * r) <= stop:
                break
        z = r / diag
        new = torch.sum(r * z)
        p = z + (new / rz) * p
        rz = new
    return x


# ---- what a pass cannot do without -------------------------------------------------
def work(case):
    """Bytes of the state and the results of a pass, read once and written once
    per time step (a step's state is the next one's input)."""
    if case["kind"] == "bulk":
        nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        store = 56 if case["bits"] == 32 else 80
        return dict(bytes=case["steps"] * 2.0 * store * case["particles"] + 48.0 * nodes, flops=0.0)
    if case["kind"] == "batch":
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        store = 56 if case["bits"] == 32 else 80
        return dict(bytes=case["steps"] * 2.0 * store * mean * case["members"], flops=0.0)
    if case["kind"] == "solve":
        nodes, cells = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1), case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=32.0 * case["particles"] + (7 + 4) * 8.0 * nodes + 8.0 * 5 * cells, flops=0.0)
    if case["deck"] == "bar":
        cells = case["nx"] * case["ny"] * case["nz"]
        particles = case["electrons"] + case["holes"]
    else:
        x, y, z = decks.finfet_grid(float(case["lg_nm"]))
        cells = (len(x) - 1) * (len(y) - 1) * (len(z) - 1)
        particles = max(case["electrons"] + case["holes"], cells * (case["floor"] if case["floor"] > 1 else 0.6))
    store = 56 if case["bits"] == 32 else 80
    solves = case["steps"] // case["poisson_every"] if case["poisson_every"] else 0
    # per step the store, the cells' charge, fields and surface rates; per solve the stencil and the potential
    return dict(bytes=case["steps"] * (2.0 * store * particles + 8.0 * 12 * cells) + solves * 8.0 * 11 * cells,
                flops=0.0)
