"""The effective potential of the quantum correction: its set-up and the order
of its sum.  The band tables are computed (perf/cases.py)."""
import bisect
import importlib.util
import os

import numpy as np
import pytest

import mcb200

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def root():
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m.tables_owner()


def graded(root, dims):
    """An engine on a graded mesh, and its cells' materials and quantum region:
    silicon under an oxide layer, with a corner of neither."""
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    eng = mcb200.Engine(max_particles=64, like=root)
    eng.set_mesh(*(np.concatenate([[0.0], np.cumsum(rng.uniform(0.3, 0.9, m))]) for m in dims))
    material = np.full((ny, nx, nz), 3, np.int32)  # cell order (j, i, k)
    material[:, 0, :] = 2
    material[0, nx - 1, :nz // 2] = 1
    region = np.zeros((ny, nx, nz), np.int32)
    region[ny // 3:, :, nz // 4:] = 1
    return eng, material.ravel(), region.ravel()


def test_set_up_again(root):
    """A correction set up again, larger, smaller and as before, is the one a
    new engine has: no launch sees an array that is still on its way."""
    dims = (24, 40, 22)
    widths = [((2.0, 2.5, 1.5), (0.5, 0.4, 0.7)), ((3.0, 3.0, 3.0), (0.9, 0.8, 0.7)), ((1.0, 1.0, 1.0), (0.3, 0.3, 0.3)),
              ((2.0, 2.5, 1.5), (0.5, 0.4, 0.7))]
    pot = np.random.default_rng(1).normal(size=(dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1)) * 10
    again, material, region = graded(root, dims)
    for ratio, theta in widths:
        new, _, _ = graded(root, dims)
        got = []
        for eng in (again, new):
            eng.set_quantum_correction(material, region, ratio, theta, 3.0, enable=False)
            got.append(eng.quantum_potential(pot))
        assert np.all(np.isfinite(got[0])) and np.any(got[0] != pot)
        assert np.array_equal(got[0].view(np.uint64), got[1].view(np.uint64))
        new.close()
    again.close()


@pytest.mark.parametrize("dims, ratio", [((5, 7, 4), (2.0, 2.5, 1.5)), ((9, 4, 11), (1.5, 3.0, 2.0)),
                                         ((3, 3, 20), (9.0, 9.0, 9.0))])
def test_sum_in_the_reference_order(root, dims, ratio):
    """The window is summed in the reference's order (x outer, z inner), one
    term after another, to the last bit.  The terms themselves come from the
    potentials of single nodes; a node's potential is +-2^e, so that its term
    is theirs times a power of two, exactly, and the sum here is the sum there."""
    px, py, pz = (d + 1 for d in dims)
    eng, material, region = graded(root, dims)
    eng.set_quantum_correction(material, region, ratio, (0.5, 0.4, 0.7), 0.0, enable=False)
    nodes = px * py * pz
    term = np.empty((nodes, nodes))  # [source][target]
    for m in range(nodes):
        term[m] = eng.quantum_potential(np.eye(1, nodes, m)[0]) * 8
    rng = np.random.default_rng(2)
    pot = rng.choice([-1.0, 1.0], nodes) * 2.0 ** rng.integers(-8, 9, nodes)
    got = eng.quantum_potential(pot)
    want, backwards = np.zeros(nodes), np.zeros(nodes)
    order = [(j * px + i) * pz + k for i in range(px) for j in range(py) for k in range(pz)]
    for m in order:
        want += pot[m] * term[m]
    for m in reversed(order):
        backwards += pot[m] * term[m]
    corrected = got != pot
    assert corrected.sum() > nodes // 4 and np.any(want != backwards)
    assert np.array_equal(got[corrected].view(np.uint64), (want / 8)[corrected].view(np.uint64))
    eng.close()


def widths(dims):
    rng = np.random.default_rng(dims[0])  # as graded's mesh
    return [rng.uniform(0.3, 0.9, m) for m in dims]


def window(line, reach):
    """An axis's windows as the set-up's lower_bound / upper_bound walk finds them."""
    low = up = 0
    out = []
    for i, at in enumerate(line):
        low = bisect.bisect_left(line, at - reach, min(low, i), i)
        up = bisect.bisect_right(line, at + reach, up)
        low -= low > 0
        up -= up == len(line)
        out.append((low, up))
    return out


@pytest.mark.parametrize("ratio", [(2.0, -6.0, -6.0), (-6.0, 2.0, -6.0), (-6.0, -6.0, -6.0), (2.0, 2.0, -6.0)])
def test_empty_windows(root, ratio):
    """Under a negative ratio a window ends before its start, on two axes at
    once too: it holds no node, and the sum over it is zero."""
    dims, theta = (8, 11, 9), (0.5, 0.4, 0.7)
    px, py, pz = (d + 1 for d in dims)
    eng, material, region = graded(root, dims)
    eng.set_quantum_correction(material, region, ratio, theta, 0.0, enable=False)
    pot = np.random.default_rng(3).normal(size=px * py * pz)
    got = eng.quantum_potential(pot)
    lines = [np.concatenate([[0.0], np.cumsum(w)]) for w in widths(dims)]
    empty = [np.array([up < low for low, up in window(list(line), r * t)])
             for line, r, t in zip(lines, ratio, theta)]
    none = (empty[1][:, None, None] | empty[0][None, :, None] | empty[2][None, None, :]).ravel()
    corrected = got != pot
    assert np.all(np.isfinite(got)) and np.any(none & corrected)
    assert np.all(got[none & corrected] == 0.0)
    eng.close()
