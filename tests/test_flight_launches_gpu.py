"""The launches a step's flight is made of, at the sizes where they change:
the drift pass's tiles of 256, warps with fewer particles than lanes, and the
store size from which final-state draws have a launch of their own.

Particles of a frozen-field box do not see one another, and each draws from
its own stream, so a store flown whole and the same particles flown in parts
must end bit for bit alike.  The drift itself is compared with numpy.

The band tables are computed (perf/cases.py), so nothing here needs the
reference."""
import importlib.util
import os

import numpy as np
import pytest

import mcb200
from mcb200.workloads import motion_rules, uniform_fields

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NX, NY, NZ, CELL_M, DONOR = 12, 7, 9, 5e-9, 1e23


@pytest.fixture(scope="module")
def cases():
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.fixture(scope="module")
def root(cases):
    return cases.tables_owner()


def box(root, capacity, precision, field=1e7, donor=DONOR, dims=(NX, NY, NZ)):
    eng = mcb200.Engine(max_particles=capacity, precision=precision, like=root)
    u = eng.units()
    h = CELL_M / u["spr0"]
    eng.set_mesh(*(np.arange(d + 1) * h for d in dims))
    eng.set_cells(motion_rules(*dims), np.full(int(np.prod(dims)), donor / u["conc0"]))
    eng.set_fields(*uniform_fields(eng, field, DONOR))
    return eng


def ensemble(root, n, precision, carrier=0):
    eng = box(root, n + 64, precision)
    rng = np.random.default_rng(n)
    eng.seed(np.sort(rng.integers(0, NX * NY * NZ, n)), np.full(n, -1e-3 if carrier == 0 else 1e-3), carrier, 5)
    return by_uid(eng)


def by_uid(eng):
    p = eng.download()
    order = np.argsort(p["uid"])
    return {k: v[order] for k, v in p.items()}


@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
@pytest.mark.parametrize("n, parts", [(1, [1]), (257, [1, 255, 1]), (2401, [256, 2145]), (70001, [35000, 35001])])
def test_whole_store_as_its_parts(root, precision, n, parts):
    p = ensemble(root, n, precision)
    whole = box(root, n + 64, precision)
    whole.upload(p)
    u = whole.units()
    dt = 1e-15 / u["time0"]
    for step in range(4):
        whole.step(step, 7, dt)
    got = by_uid(whole)
    ends, events, phonons, impurities = [], 0, 0, 0
    at = 0
    for m in parts:
        eng = box(root, m + 64, precision)
        eng.upload({k: v[at:at + m] for k, v in p.items()})
        for step in range(4):
            eng.step(step, 7, dt)
        ends.append(by_uid(eng))
        t = eng.tallies()
        events, phonons, impurities = events + t["events"], phonons + t["phonon"], impurities + t["impurity"]
        at += m
    for k in got:
        expect = np.concatenate([e[k] for e in ends])
        assert np.array_equal(got[k].view(np.uint8), expect.view(np.uint8)), k
    t = whole.tallies()
    assert (t["events"], t["phonon"], t["impurity"]) == (events, phonons, impurities)
    if n > 70000:
        assert phonons > 100 and impurities > 1000  # the draws and the impurity events are in it


@pytest.mark.parametrize("carrier", [0, 1])
def test_holes_and_electrons_as_parts_in_a_hot_field(root, carrier):
    """Zone-boundary crossings, impact ionisation's neighbours: 30 kV/mm."""
    p = ensemble(root, 1031, mcb200.FLIGHT_FP64, carrier)
    engines = []
    for take in (slice(None), slice(0, 500), slice(500, None)):
        eng = box(root, 2000, mcb200.FLIGHT_FP64, field=3e7)
        eng.upload({k: v[take] for k, v in p.items()})
        for step in range(30):
            eng.step(step, 3, 1e-15 / eng.units()["time0"])
        engines.append(by_uid(eng))
    for k in engines[0]:
        both = np.concatenate([engines[1][k], engines[2][k]])
        assert np.array_equal(engines[0][k].view(np.uint8), both.view(np.uint8)), k


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
def test_batch_tails_at_tile_edges(root, precision, graphs):
    """A batch's records, appends and sorts take its members' tiles of 256
    particles together: members of none, one, and a tile more or less one end
    as alone, also when a member's sort buckets change between steps."""
    counts = [257, 0, 1, 255, 256, 513]
    engines = []
    for m in counts:
        pair = [box(root, m + 64, precision) for _ in range(2)]
        if m:
            for eng in pair:
                eng.upload(ensemble(root, m, precision))
        engines.append(pair)
    dt = 1e-15 / engines[0][0].units()["time0"]
    batch = mcb200.Batch([(pair[1], dict(dt=dt, seed=9 + k, first_step=k, self_consistent=0, poisson_every=1))
                          for k, pair in enumerate(engines)])
    batch.use_graphs(graphs)
    for at, steps, bucket in ((0, 3, 1), (3, 2, 8), (5, 2, 1)):
        for k, pair in enumerate(engines):
            for eng in pair if k % 2 == 0 else ():
                eng.set_sort_bucket(bucket)
            for step in range(at, at + steps):
                pair[0].step(k + step, 9 + k, dt)
        batch.run(steps)
    batch.sync()
    for m, (alone, member) in zip(counts, engines):
        a, b = by_uid(alone), by_uid(member)
        assert a["uid"].size == m
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg=f"{m} {key}")
        ta, tb = alone.tallies(), member.tallies()
        assert [ta[key] for key in ("events", "phonon", "impurity")] == [tb[key] for key in ("events", "phonon", "impurity")]
    batch.close()


@pytest.mark.parametrize("bucket", [1, 4])
@pytest.mark.parametrize("dims", [(1, 1, 1), (11, 31, 3), (32, 32, 1), (41, 25, 1), (129, 128, 64)])
def test_step_sorts_the_store(root, dims, bucket):
    """The step's sort over 1 to 1,056,768 buckets: tiles of 1024 (one short by
    one, full, one more by one) and more than 1024 tiles."""
    cells, n = int(np.prod(dims)), 20000
    eng = box(root, n + 64, mcb200.FLIGHT_FP64, dims=dims)
    eng.set_sort_bucket(bucket)
    rng = np.random.default_rng(cells)
    eng.seed(rng.integers(0, cells, n), np.full(n, -1e-3), 0, 5)
    before = np.sort(eng.download()["uid"])
    for step in range(2):
        eng.step(step, 7, 1e-16 / eng.units()["time0"])
    p = eng.download()
    i, j, k = (p[a].astype(np.int64) for a in ("i", "j", "k"))
    keys = ((j * dims[0] + i) * dims[2] + k) // bucket
    assert before.size == n and np.array_equal(np.sort(p["uid"]), before)
    assert keys.min() >= 0 and keys.max() <= (cells - 1) // bucket
    assert np.all(np.diff(keys) >= 0)


def philox_block0(uid, step, seed):
    """The stream's first Philox4x32-10 block per uid (include/mcb200_rng.h), words [4, n]."""
    c = [np.zeros(len(uid), np.uint64), uid.astype(np.uint64), np.full(len(uid), step, np.uint64),
         np.zeros(len(uid), np.uint64)]
    k0, k1, low = seed & 0xffffffff, seed >> 32, np.uint64(0xffffffff)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return c


@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
def test_drift_against_numpy(root, precision):
    """Particles without an event in the step (no face within it, both clocks
    longer than it, computed here in 64 bits with a 1e-3 margin) end where
    the free drift takes them: FP64 to 1e-12, FP32 (float positions in a 5 nm
    cell, float k) to 1e-6 of the cell and of the zone.  No impurities: their
    clock then runs at the 1 / scrt0 floor."""
    n, seed, step = 5000, 11, 4
    eng = box(root, n + 64, precision, donor=0.0)
    p = ensemble(root, n, precision)
    eng.upload(p)
    u = eng.units()
    dt = 0.5e-15 / u["time0"]
    nt = root.table("ibt", np.int32).size
    vt = root.table("vt", np.float64).reshape(nt, 4)
    face = root.table("datantlin", np.float64).reshape(4, 4, nt)
    sym = root.table("matsym", np.int32).reshape(6, 48)
    gam, band = root.table("gamtet", np.float64), root.table("ibt", np.int32)
    perm, sign = sym[:3, p["isym"]] - 1, sym[3:, p["isym"]]
    cols = np.arange(n)
    vw = vt[p["itet"], :3].T
    v = np.array([vw[perm[c], cols] * sign[c] for c in range(3)])
    field = -1e7 / u["field0"]
    k = np.array([p["kx"], p["ky"], p["kz"]])
    e = np.array([np.full(n, field), np.zeros(n), np.zeros(n)])

    def wedge(a):
        out = np.zeros((3, n))
        for c in range(3):
            out[perm[c], cols] = a[c] * sign[c]
        return out

    kw, ew = wedge(k), wedge(e)
    f = face[:, :, p["itet"]]
    rate = np.einsum("cfn,cn->fn", f[:3], ew)
    gap = f[3] - np.einsum("cfn,cn->fn", f[:3], kw)
    tet_time = np.where(rate < 0, np.maximum(gap / np.where(rate < 0, rate, 1), 0), np.inf).min(0)
    h = CELL_M / u["spr0"]
    pos = np.array([p["x"], p["y"], p["z"]]) - h * np.array([p["i"], p["j"], p["k"]])
    with np.errstate(divide="ignore", invalid="ignore"):
        cell_time = np.where(v > 0, (h - pos) / v, np.where(v < 0, -pos / v, np.inf)).min(0)
    w = philox_block0(p["uid"], step, seed)
    if precision == mcb200.FLIGHT_FP64:
        unit = lambda hi, lo: (((hi << np.uint64(32)) | lo) >> np.uint64(12)).astype(float) * 2.0 ** -52 + 2.0 ** -53  # noqa: E731
        u0, u1 = unit(w[1], w[0]), unit(w[3], w[2])
    else:
        u0, u1 = ((x >> np.uint64(9)).astype(float) * 2.0 ** -23 + 2.0 ** -24 for x in w[:2])
    ph_time = -np.log(u0) / gam[p["itet"]]
    imp_time = np.where(band[p["itet"]] == 0, -np.log(u1) * u["scrt0"], np.inf)
    quiet = np.minimum.reduce([tet_time, cell_time, ph_time, imp_time]) > dt * 1.001
    assert quiet.sum() > 1000 and (~quiet).sum() > 100
    eng.step(step, seed, dt)
    got = by_uid(eng)
    assert np.array_equal(got["uid"], p["uid"])
    tol = 1e-12 if precision == mcb200.FLIGHT_FP64 else 1e-6
    for c, name in enumerate("xyz"):
        assert np.max(np.abs(got[name] - (p[name] + v[c] * dt))[quiet]) <= tol * h * NX, name
        kn = "k" + name
        assert np.max(np.abs(got[kn] - (p[kn] + e[c] * dt))[quiet]) <= tol * u["a0pi"], kn
    assert np.max(np.abs(got["energy"] - (p["energy"] + (v * e).sum(0) * dt))[quiet]) <= tol * p["energy"].max()
    for name in ("i", "j", "k", "itet", "isym"):
        assert np.array_equal(got[name][quiet], p[name][quiet]), name


@pytest.mark.parametrize("dims", [(11, 13, 9), (24, 30, 22)])
def test_poisson_against_plain_conjugate_gradients(cases, dims):
    """A 1e-10 residual leaves these systems within 1e-8 of the solution."""
    case = dict(kind="solve", nx=dims[0], ny=dims[1], nz=dims[2], particles=20000, vg=0.7, vd=0.3)
    got, want = cases.run(cases.prepare(case, 3)), cases.exact(case, 3)
    for name, tol in (("node_density", 1e-11), ("potential", 1e-8), ("efield", 1e-7)):
        assert np.linalg.norm(got[name] - want[name]) <= tol * np.linalg.norm(want[name]), name


@pytest.mark.parametrize("dims", [(3, 3, 3), (9, 5, 7), (14, 11, 8)])
def test_effective_potential_against_the_sum(root, dims):
    """The window sum of erf products, term by term, on a graded mesh with a
    vacuum corner and an oxide layer; 1e-12 of the potential's scale."""
    from math import erf, sqrt

    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    width = [rng.uniform(0.3, 0.9, m) for m in dims]
    edge = [np.concatenate([[0.0], np.cumsum(w)]) for w in width]
    material = np.full((ny, nx, nz), 3, np.int32)  # cell order (j, i, k)
    material[:, 0, :] = 2
    material[0, nx - 1, :nz // 2] = 1
    region = np.zeros((ny, nx, nz), np.int32)
    region[ny // 3:, :, nz // 4:] = 1
    ratio, theta, eb = (2.0, 2.5, 1.5), (0.5, 0.4, 0.7), 3.0
    eng = mcb200.Engine(max_particles=64, like=root)
    eng.set_mesh(*edge)
    eng.set_quantum_correction(material.ravel(), region.ravel(), ratio, theta, eb, enable=False)
    pot = rng.normal(size=(ny + 1, nx + 1, nz + 1)) * 10
    flags = {m: np.zeros(pot.shape, bool) for m in ("si", "ox", "q")}
    for b in (0, 1):
        for a in (0, 1):
            for c in (0, 1):
                at = (slice(b, ny + b), slice(a, nx + a), slice(c, nz + c))
                flags["si"][at] |= material == 3
                flags["ox"][at] |= material == 2
                flags["q"][at] |= region != 0
    inside = flags["si"] | flags["ox"]
    shape = [nx + 1, ny + 1, nz + 1]

    def outside(n):
        return not (all(0 <= n[a] < shape[a] for a in range(3)) and inside[n[1], n[0], n[2]])

    window = []
    for a in range(3):
        x, reach = edge[a], ratio[a] * theta[a]
        low = [max(np.searchsorted(x[:i], x[i] - reach) - 1, 0) for i in range(len(x))]
        up = [min(np.searchsorted(x, x[i] + reach, side="right"), len(x) - 1) for i in range(len(x))]
        window.append(list(zip(low, up)))
    want = pot.copy()
    for j, i, k in np.argwhere(flags["q"]):
        total, at = 0.0, (i, j, k)
        ranges = [range(window[a][at[a]][0], window[a][at[a]][1] + 1) for a in range(3)]
        for p in ranges[0]:
            for q in ranges[1]:
                for r in ranges[2]:
                    if not inside[q, p, r]:
                        continue
                    term = pot[q, p, r] - (eb if flags["ox"][q, p, r] and not flags["si"][q, p, r] else 0.0)
                    for a, n in ((2, r), (1, q), (0, p)):
                        node = [p, q, r]
                        node[a] = n - 1
                        lo = edge[a][n] - (ratio[a] * theta[a] if outside(node) else 0.5 * width[a][n - 1])
                        node[a] = n + 1
                        hi = edge[a][n] + (ratio[a] * theta[a] if outside(node) else 0.5 * width[a][n])
                        s = sqrt(2.0) * theta[a]
                        term *= erf((hi - edge[a][at[a]]) / s) - erf((lo - edge[a][at[a]]) / s)
                    total += term
        want[j, i, k] = total / 8
    got = eng.quantum_potential(pot.ravel()).reshape(pot.shape)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(pot)) * 8
