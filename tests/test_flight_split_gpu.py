"""The flight in two launches -- the listed particles first, then those that
came to a final-state draw -- against the flight in one: which of them a step
takes is decided by the number of carriers (65,536 in FP64, a million in FP32,
a batch's members together) and must not show in any result.

The band tables are computed (perf/cases.py)."""
import numpy as np
import pytest

import mcb200
from mcb200.workloads import motion_rules, uniform_fields
from test_flight_launches_gpu import box, by_uid, cases, ensemble, philox_block0, root  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu
SPLIT = {mcb200.FLIGHT_FP64: 65536, mcb200.FLIGHT_FP32: 1000000}


def same(a, b, where=""):
    for k in a:
        if isinstance(a[k], np.ndarray):
            assert np.array_equal(a[k].view(np.uint8), b[k].view(np.uint8)), (where, k)
        else:
            assert a[k] == b[k], (where, k)


@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
def test_draw_due_at_the_end_of_the_step(root, precision):  # noqa: F811
    """A phonon event at exactly the end of the step is the particle's, in one
    launch or two: no field, and a time step that is one particle's time to its
    phonon to the last bit (the one at which that particle, flown alone, counts
    it and nothing else: a shorter step ends before it, a longer one goes on)."""
    real = np.float64 if precision == mcb200.FLIGHT_FP64 else np.float32
    n, seed, step = SPLIT[precision] + 1, 7, 3
    p = ensemble(root, n, precision)

    def fly(take, dt):
        some = {k: v[take] for k, v in p.items()}
        eng = box(root, some["uid"].size + 64, precision, field=0.0, donor=0.0)
        eng.upload(some)
        eng.step(step, seed, float(dt))
        out, t = by_uid(eng), eng.tallies()
        eng.close()
        return out, t

    gam = root.table("gamtet", np.float64)
    w = philox_block0(p["uid"], step, seed)
    if precision == mcb200.FLIGHT_FP64:
        u0 = (((w[1] << np.uint64(32)) | w[0]) >> np.uint64(12)).astype(float) * 2.0 ** -52 + 2.0 ** -53
    else:
        u0 = (w[0] >> np.uint64(9)).astype(float) * 2.0 ** -23 + 2.0 ** -24
    clock = -np.log(u0) / gam[p["itet"]]
    due = np.argsort(np.abs(clock * root.units()["time0"] - 0.3e-15))  # a third of a step of the other tests
    tie = None
    for q in due[:40]:
        t = real(clock[q])
        for _ in range(10):
            t = np.nextafter(t, real(0))
        counted = []
        for _ in range(20):
            tally = fly(slice(q, q + 1), t)[1]
            counted.append((t, tally["phonon"], tally["events"]))
            t = np.nextafter(t, real(1e9))
        first = [i for i, c in enumerate(counted) if c[1]]
        if first and first[0] > 0 and counted[first[0]][2] == 1:
            tie = counted[first[0]][0]
            break
    assert tie is not None
    whole, tw = fly(slice(None), tie)
    half = n // 2
    parts = [fly(slice(0, half), tie), fly(slice(half, None), tie)]
    same({k: np.concatenate([parts[0][0][k], parts[1][0][k]]) for k in whole}, whole)
    assert np.any(whole["uid"] == p["uid"][q])
    for k in ("events", "phonon", "impurity"):
        assert tw[k] == parts[0][1][k] + parts[1][1][k], k


def test_copies_beyond_4096_in_a_step(root):  # noqa: F811
    """A carrier that makes thousands of copies between two of its draws (a
    plane of cells 0.1 pm thick between a mirror and a face that makes copies):
    each copy has a stream of its own, numbered on through a launch for the
    draws as in one launch."""
    precision, (nx, ny, nz), thin, specials = mcb200.FLIGHT_FP64, (4, 6, 4), 3, 8
    n = SPLIT[precision] + 1
    widths = np.full(ny, 5e-9)
    widths[thin] = 1e-13

    def slab(count):
        eng = mcb200.Engine(max_particles=1 << 22, precision=precision, like=root)
        u = eng.units()
        x, y, z = (np.concatenate([[0.0], np.cumsum(w)]) / u["spr0"]
                   for w in (np.full(nx, 5e-9), widths, np.full(nz, 5e-9)))
        eng.set_mesh(x, y, z)
        faces = motion_rules(nx, ny, nz).reshape(ny, nx, nz, 6)
        reflect, genref, left, right = 2, 8, 2, 3
        faces[thin - 1, :, :, right] = faces[thin, :, :, left] = faces[thin + 1, :, :, left] = reflect
        faces[thin, :, :, right] = genref
        cells = nx * ny * nz
        eng.set_cells(faces.reshape(-1), np.zeros(cells))
        eng.set_fields(*uniform_fields(eng, 0.0, 1e23))
        rng = np.random.default_rng(1)
        plane = rng.permutation(np.repeat([0, 1, 2, 4, 5], (count - specials) // 5 + 1))[:count - specials]
        cell = np.concatenate([np.full(specials, thin * nx * nz + 5),
                               plane * nx * nz + rng.integers(0, nx * nz, count - specials)])
        eng.seed(cell, np.full(count, -1e-3), 0, 5)
        return eng, u

    ends = []
    for count in (n, 300):
        eng, u = slab(count)
        eng.step(0, 7, 6e-14 / u["time0"])
        p, t = by_uid(eng), eng.tallies()
        ends.append({k: v[(p["uid"] < specials) | (p["uid"] >= count)] for k, v in p.items()})
        ends[-1]["uid"] = np.where(ends[-1]["uid"] < specials, ends[-1]["uid"], ends[-1]["uid"] - count + specials)
        assert t["generated"] > specials * 4096 and t["child_overflow"] == 0
        eng.close()
    same(*ends)
