"""The drift pass at screening densities no float holds: the Brooks-Herring
rate of a doped cell grows without bound as its density goes to zero, so its
electrons of the lowest band have their impurity event at once, however the
pass estimates the rate.  A zero time catches an FP64 particle; an FP32 one
goes on, and so takes a pass for the event and one or more after it.

The band tables are computed (perf/cases.py)."""
import numpy as np
import pytest

import mcb200
from mcb200.workloads import uniform_fields
from test_flight_launches_gpu import CELL_M, DONOR, NX, NY, NZ, box, by_uid, cases, ensemble, root  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [mcb200.FLIGHT_FP64, mcb200.FLIGHT_FP32])
def test_tiny_screening_density(root, precision):  # noqa: F811
    n = 5000
    eng = box(root, n + 64, precision, field=0.0)
    p = ensemble(root, n, precision)
    u = eng.units()
    e, h, _ = uniform_fields(eng, 0.0, DONOR)
    rho = 10.0 ** np.linspace(-41.0, -37.0, NX * NY * NZ)
    eng.set_fields(e, h, rho)
    nt = root.table("ibt", np.int32).size
    band = root.table("ibt", np.int32)[p["itet"]]
    low = root.table("eek", np.float64)[root.table("tet", np.int32).reshape(4, nt)[0, p["itet"]]]
    at_once = (band == 0) & (low > 0) & (low < 0.99 * 0.120 / u["eV0"])
    if precision == mcb200.FLIGHT_FP32:  # where the rate's denominator is nearly the largest float
        meld, melt = (0.9116 * 0.1946 ** 2) ** (1 / 3), 0.1946
        cell = (p["j"].astype(int) * NX + p["i"]) * NZ + p["k"]
        eebeta = 4 * np.pi * rho[cell] / (2 * meld * u["eps_silicon"])
        under = 4 * melt / (eebeta * meld) * low
        at_once &= (under > 1.001 * 2.0 ** 126) & (under < 0.999 * 2.0 ** 128)
    m = int(at_once.sum())
    assert m > 50
    eng.upload({k: v[at_once] for k, v in p.items()})
    eng.step(0, 7, 0.1e-15 / u["time0"])
    t = eng.tallies()
    if precision == mcb200.FLIGHT_FP64:
        assert t["caught"] == m and eng.num_particles() == 0
    else:
        assert t["events"] >= 2 * m
    eng.close()
