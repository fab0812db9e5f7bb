"""Small meshes are left to a single CTA by the resident engine's default, which
needs no cluster barrier.  Bit for bit with the plain engine."""
import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

BOX = dict(box_x=1.0, box_y=1.0, box_z=1.0, n_foot_x=2, n_foot_y=2, n_out_x=2, n_out_y=2, n_above_z=4, ryr_mode=1,
           ryr_count=4, ryr_radius=0.052, ryr_pitch=0.030, foot_half_x=0.102, foot_half_y=0.102, n_lcc=1,
           lcc_half=0.102, seed=11, lcc_seed=21)


@pytest.mark.parametrize("spec,n", [(wl.TINY_DYAD, 384), (BOX, 1296)])
@pytest.mark.parametrize("R", [1, 40, 300])
def test_small_mesh_takes_one_cta(srs, tmp_path, spec, n, R):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **spec)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=1, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    assert g.n_ele == n
    x, y = (srs.Simulation(g, p, R, 32, e, seeds=list(range(1, R + 1)))
            for e in (srs.ENGINE_RESIDENT, srs.ENGINE_PLAIN))
    assert x.config()["cluster_size"] == 1
    for s in (x, y):
        s.explicit_step(41)
    for r in (0, R - 1):
        u, v = x.get_state(r), y.get_state(r)
        for k in u:
            assert np.array_equal(u[k], v[k]), (r, k)
