"""Batched devices against the same devices stepped alone, on computed band
tables (perf/cases.py): boxes with contacts and scattering faces whose carriers
together pass the line from which a step's final-state draws have a launch of
their own, while each alone does not; and FinFETs that solve Poisson on
different steps, so that they fly beside one another's solves, some in launches
of their own.  Every particle, tally and potential bit for bit."""
import numpy as np
import pytest

import mcb200
from mcb200.workloads import motion_rules, uniform_fields
from test_flight_launches_gpu import by_uid, cases, root  # noqa: F401 (fixtures)
from test_flight_split_gpu import SPLIT, same

pytestmark = pytest.mark.gpu
BITS = {mcb200.FLIGHT_FP64: 64, mcb200.FLIGHT_FP32: 32}
SCATTOX, GENERATE, CATCH, GENREF = 3, 5, 6, 8
UP, DOWN, LEFT, RIGHT, FRONT, BACK = range(6)


def device_box(root, precision, n, seed, planes, surface):  # noqa: F811
    """A frozen-field box of n electrons and 500 holes with a contact at each
    end of y, scattering faces at x = 0 and z = 0, and `planes` of faces that
    make copies of what meets them."""
    nx, ny, nz = 12, 16, 9
    cells = nx * ny * nz
    eng = mcb200.Engine(max_particles=2 * n + 65536, precision=precision, like=root)
    u = eng.units()
    h = 5e-9 / u["spr0"]
    eng.set_mesh(*(np.arange(d + 1) * h for d in (nx, ny, nz)))
    faces = motion_rules(nx, ny, nz).reshape(ny, nx, nz, 6)
    faces[:, 0, :, UP] = faces[:, :, 0, FRONT] = SCATTOX
    faces[1, :, :, LEFT] = faces[ny - 2, :, :, RIGHT] = CATCH
    faces[0, :, :, RIGHT] = faces[ny - 1, :, :, LEFT] = GENERATE
    for j in planes:
        faces[j, :, :, RIGHT] = faces[j + 1, :, :, LEFT] = GENREF
    contact = np.zeros((ny, nx, nz), np.int32)
    contact[0], contact[ny - 1] = 1, 2
    i, k = np.meshgrid(np.arange(nx), np.arange(nz), indexing="ij")
    near = np.broadcast_to(np.where(i <= k, 0, 1), (ny, nx, nz))
    in_surf = np.zeros((ny, nx, nz), np.int32)
    in_surf[:, :3, :] = in_surf[:, :, :3] = int(surface)
    eng.set_cells(faces.reshape(-1), np.full(cells, 1e23 / u["conc0"]), contact.ravel(), in_surf.ravel(), near.ravel(),
                  [UP, FRONT], mcb200.FLAG_HEAT | (mcb200.FLAG_SURFACE_SCATTER if surface else 0))
    eng.set_fields(*uniform_fields(eng, 5e6, 1e23))
    if surface:
        eng.set_surface_rates(*(np.full(cells, 1e13 * u["time0"] * f) for f in (1.0, 2.0, 0.5, 1.5)))
    rng = np.random.default_rng(seed)
    eng.seed(np.sort(rng.integers(0, cells, n)), np.full(n, -1e-3), 0, seed)
    eng.seed(np.sort(rng.integers(0, cells, 500)), np.full(500, 1e-3), 1, seed)
    return eng, dict(dt=1e-15 / u["time0"], seed=seed, first_step=0, self_consistent=0)


@pytest.mark.parametrize("precision, n, planes, surface, copies", [
    (mcb200.FLIGHT_FP64, SPLIT[mcb200.FLIGHT_FP64] // 2 + 100, [5], False, 100),
    (mcb200.FLIGHT_FP64, SPLIT[mcb200.FLIGHT_FP64] // 2 + 100, [5], True, 100),
    (mcb200.FLIGHT_FP32, SPLIT[mcb200.FLIGHT_FP32] // 2 + 100, [3, 5, 7, 9, 11], False, 5000),
    (mcb200.FLIGHT_FP32, SPLIT[mcb200.FLIGHT_FP32] // 2 + 100, [5], True, 1000)])
def test_split_batch_of_devices(root, precision, n, planes, surface, copies):  # noqa: F811
    steps = 4
    pairs = [[device_box(root, precision, n, seed, planes, surface) for _ in range(2)] for seed in (3, 4)]
    assert n + 500 + copies < SPLIT[precision] <= 2 * n
    for (eng, cfg), _ in pairs:
        for step in range(steps):
            eng.step(step, cfg["seed"], cfg["dt"])
        assert eng.num_particles() < SPLIT[precision]  # alone it took one launch throughout
    batch = mcb200.Batch([b for _, b in pairs])
    batch.run(steps)
    batch.sync()
    for (a, _), (b, _) in pairs:
        same(by_uid(a), by_uid(b))
        t = a.tallies()
        same(t, b.tallies())
        assert t["phonon"] > 100 and t["generated"] > copies and t["caught"] > 10
        assert np.any(t["heat_e"] != 0) and np.any(t["contact"] != 0)
    batch.close()
    for pair in pairs:
        for eng, _ in pair:
            eng.close()


def finfet(cases, precision, lg_nm, electrons, seed):  # noqa: F811
    s = cases.prepare(dict(kind="deck", deck="finfet", lg_nm=lg_nm, electrons=electrons, holes=2000, floor=1, vg=0.6,
                           bits=BITS[precision], steps=1, poisson_every=4, window=0), seed)
    s["eng"].surface_rates(s["eeff"], **s["surface"])
    return s


@pytest.mark.parametrize("precision, graphs, overlap, solo",
                         [(mcb200.FLIGHT_FP64, False, True, False), (mcb200.FLIGHT_FP64, True, True, True),
                          (mcb200.FLIGHT_FP32, True, True, False), (mcb200.FLIGHT_FP32, False, False, True)])
def test_finfets_beside_one_anothers_solves(cases, precision, graphs, overlap, solo):  # noqa: F811
    steps, every, first = 9, 4, [0, 1, 2]
    shapes = [(20, 20000, 3), (14, 8000, 4), (16, 30000, 5)]
    pairs = [[finfet(cases, precision, *shape) for _ in range(2)] for shape in shapes]
    for (a, _), f in zip(pairs, first):
        for step in range(f, f + steps):
            a["eng"].deposit()
            if step % every == 0:
                a["eng"].solve_poisson_async(1e-10, 20000)
            a["eng"].surface_rates(a["eeff"], **a["surface"])
            a["eng"].step(step, a["seed"], a["dt"])
    batch = mcb200.Batch([(b["eng"], dict(dt=b["dt"], seed=b["seed"], first_step=f, self_consistent=1,
                                          poisson_every=every, surface_rates=1))
                          for (_, b), f in zip(pairs, first)])
    batch.use_graphs(graphs)
    batch.set_overlap(overlap)
    if solo:
        most = max(b["eng"].num_particles() for _, b in pairs)
        assert batch.set_solo(most) == 1
    batch.run(4)
    batch.run(steps - 4)
    batch.sync()
    for a, b in pairs:
        same(by_uid(a["eng"]), by_uid(b["eng"]))
        t = a["eng"].tallies()
        same(t, b["eng"].tallies())
        assert t["generated"] > 10 and t["phonon"] > 10
        for name in ("potential", "efield", "node_density"):
            same({name: a["eng"].array(name)}, {name: b["eng"].array(name)})
    batch.close()
    for pair in pairs:
        for s in pair:
            s["eng"].close()
