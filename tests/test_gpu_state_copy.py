"""States read back on both sides of the size from which they are copied without
staging (640 KB, 13,653 elements): what was set, to the engines' rounding of the
deviation from rest, with the channels' states or without."""
import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec,n", [({}, 10368), (wl.config2_mesh_specs()[1], 15288)])
@pytest.mark.parametrize("prec,engine", [(64, 0), (32, 0), (32, 1)])
def test_state_read_back(srs, tmp_path, spec, n, prec, engine):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **spec)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4)
    g = srs.Grid(p, base)
    assert g.n_ele == n
    sim = srs.Simulation(g, p, 2, prec, engine, seeds=[1, 2])
    first = sim.get_state(1)
    rest = first["states"]
    want = rest * (1 + 0.2 * np.random.default_rng(7).random(rest.shape))
    ryr = 1 - first["ryr"]
    sim.set_state(1, want, ryr=ryr)
    if prec == 32:
        want = rest + (want - rest).astype(np.float32).astype(np.float64)
    got = sim.get_state(1)
    assert np.array_equal(got["states"], want) and np.array_equal(got["ryr"], ryr)
    for k in ("lcc", "lccv", "residuals"):
        assert np.array_equal(got[k], first[k])
    assert np.array_equal(sim.get_state(0)["states"], rest)
