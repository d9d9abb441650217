"""The statistics' particle sums: chunks of 32 particles and their remainders,
runs of one to many particles of a cell and type, stores in cell order and
mixed, both carrier types.

The charge sums are numpy's bit for bit: the same rounded products in the same
fixed point (2^62 over the sum's bound, a power of two).  An FP32 store's
positions come back with a cell's corner added, so its sums are held to 1e-6
of the largest.  All five sums are whole numbers, so a store in any order
gives the same bits."""
import importlib.util
import os

import numpy as np
import pytest

import mcb200
from mcb200.workloads import motion_rules

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def root():
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m.tables_owner()


FIELDS = ("qvx", "qvy", "qvz", "q", "qe")


@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
@pytest.mark.parametrize("n, dims", [(1, (1, 1, 1)), (31, (2, 1, 3)), (33, (1, 1, 2)), (700, (5, 3, 7)),
                                     (10000, (6, 5, 4)), (9999, (40, 30, 20))])
def test_statistics_sums(root, precision, n, dims):
    nx, ny, nz = dims
    h = 5e-9 / root.units()["spr0"]
    edges = [np.arange(d + 1) * h for d in dims]
    rng = np.random.default_rng(n)

    def engine():
        eng = mcb200.Engine(max_particles=n + 64, precision=precision, like=root)
        eng.set_mesh(*edges)
        eng.set_cells(motion_rules(*dims), np.full(nx * ny * nz, 1e-3))
        return eng

    def sums(eng):
        eng.stat_begin(2)
        for _ in range(2):
            eng.stat_accumulate()
        out = {(t, f): eng.stat(f"{name}_{f}") for t, name in ((0, "electron"), (1, "hole")) for f in FIELDS}
        out["cells"] = eng.stat("cell_count")
        return out

    eng, mixed = engine(), engine()
    cell, half = np.sort(rng.integers(0, nx * ny * nz, n)), n // 2
    eng.seed(cell[:half], np.full(half, -1e-3), 0, 5)
    eng.seed(cell[half:], rng.uniform(1e-4, 2e-3, n - half), 1, 6)
    p = eng.download()
    order = rng.permutation(n)
    mixed.upload({k: v[order] for k, v in p.items()})
    got, other = sums(eng), sums(mixed)
    for k in got:
        assert np.array_equal(got[k], other[k]), k

    count = np.bincount((p["j"].astype(np.int64) * nx + p["i"]) * nz + p["k"], minlength=nx * ny * nz)
    assert np.array_equal(got["cells"], 2.0 * count)
    r = [(p[c] - e[p[i]]) / (e[p[i] + 1] - e[p[i]]) for c, e, i in zip("xyz", edges, "ijk")]
    nodes = (nx + 1) * (ny + 1) * (nz + 1)
    for t in (0, 1):
        of = p["type"] == t
        if not np.any(of):
            continue
        unit = 2.0 ** (62 - np.ceil(np.log2(np.count_nonzero(of) * np.max(np.abs(p["charge"][of])) * 2 * 4.0)))
        q = np.zeros(nodes, dtype=np.int64)
        for b in (0, 1):
            for a in (0, 1):
                for d in (0, 1):
                    wx, wy, wz = (x if up else 1 - x for x, up in zip(r, (a, b, d)))
                    node = ((p["j"].astype(np.int64) + b) * (nx + 1) + p["i"] + a) * (nz + 1) + p["k"] + d
                    term = np.rint(np.abs(p["charge"] * (wx * wy * wz)) * unit).astype(np.int64)
                    np.add.at(q, node[of], term[of])
        want = (2 * q).astype(np.float64) / unit
        if precision == mcb200.FLIGHT_FP64:
            assert np.array_equal(got[t, "q"], want)
        else:
            assert np.all(np.abs(got[t, "q"] - want) <= 1e-6 * np.max(want))
        if n > 9000:
            assert all(np.any(got[t, f] != 0) for f in FIELDS)
