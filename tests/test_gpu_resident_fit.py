"""Meshes that all but fill the shared memory of a named cluster: the channel
group of three warps, or the staged gating constants, would leave them no room.
Bit for bit with the plain engine."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# hexahedra along each axis, six elements each; RyRs; cluster; threads (0: open)
@pytest.mark.parametrize("shape,n_ryr,C,T", [((7, 10, 12), 4, 1, 512), ((7, 10, 12), 4, 1, 0),
                                             ((10, 12, 13), 49, 2, 512), ((10, 12, 13), 49, 2, 0),
                                             ((9, 10, 17), 49, 2, 384), ((15, 18, 18), 4, 6, 320),
                                             ((8, 14, 59), 4, 8, 640)])
def test_named_cluster_holds_the_mesh(srs, tmp_path, shape, n_ryr, C, T):
    a, b, c = shape
    rad = 0.026 * math.sqrt(n_ryr)
    base = str(tmp_path / "m")
    rep = srs.write_box_mesh(base, box_x=3.0, box_y=3.0, box_z=3.0, foot_half_x=rad + 0.05, foot_half_y=rad + 0.05,
                             n_foot_x=a - 4, n_foot_y=b - 4, n_out_x=2, n_out_y=2, n_above_z=c - 2, ryr_mode=1,
                             ryr_count=n_ryr, ryr_radius=rad, ryr_pitch=0.030, n_lcc=1, lcc_half=rad + 0.05, seed=11,
                             lcc_seed=21)
    assert rep["n_tets"] == 6 * a * b * c
    p = srs.default_parameters().set(T_STEP=1e-6, INIT_RYR=1, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    x = srs.Simulation(g, p, 2, 32, srs.ENGINE_RESIDENT, seeds=[3, 4], cluster_size=C, threads_per_cta=T)
    y = srs.Simulation(g, p, 2, 32, srs.ENGINE_PLAIN, seeds=[3, 4])
    assert x.config()["cluster_size"] == C
    for s in (x, y):
        s.explicit_step(40)
    # new constants reach the steps wherever they are kept
    for s in (x, y):
        s.set_globals(-20.0, 900.0)
        s.explicit_step(41)
    for r in range(2):
        u, v = x.get_state(r), y.get_state(r)
        for k in u:
            assert np.array_equal(u[k], v[k]), (r, k)
