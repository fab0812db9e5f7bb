"""The resident engine at the configuration that the library chooses, against the
plain engine, bit for bit: few and many realizations, meshes of one cluster size
and another, and one whose partitions fill a block's shared memory."""
import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index,R", [(0, 1), (0, 100), (1, 37), (2, 3), (2, 20), (3, 9)])
def test_default_configuration(srs, tmp_path, index, R):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **wl.config2_mesh_specs()[index])
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    sims = [srs.Simulation(g, p, R, 32, e, seeds=list(range(1, R + 1)))
            for e in (srs.ENGINE_RESIDENT, srs.ENGINE_PLAIN)]
    cfg = sims[0].config()
    assert cfg["cluster_size"] > 0 and cfg["threads_per_cta"] % 32 == 0
    for s in sims:
        s.explicit_step(41)
    for r in (0, R // 2, R - 1):
        x, y = (s.get_state(r) for s in sims)
        for k in ("states", "ryr", "lcc", "lccv", "residuals"):
            assert np.array_equal(x[k], y[k]), (r, k)
