"""New constants (set_globals) around the steps of a batch, also where a member's
mesh leaves no shared memory for its gating constants.  Bit for bit with the plain
engine."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# cluster, threads: room for the constants, none
CONFIGS = [(2, 256), (1, 512)]


def _pair(srs, tmp_path, C, T):
    """The resident and the plain simulation of 7 x 10 x 12 hexahedra, 5,040 elements."""
    rad = 0.026 * math.sqrt(4)
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, box_x=3.0, box_y=3.0, box_z=3.0, foot_half_x=rad + 0.05, foot_half_y=rad + 0.05,
                       n_foot_x=3, n_foot_y=6, n_out_x=2, n_out_y=2, n_above_z=10, ryr_mode=1, ryr_count=4,
                       ryr_radius=rad, ryr_pitch=0.030, n_lcc=1, lcc_half=rad + 0.05, seed=11, lcc_seed=21)
    p = srs.default_parameters().set(T_STEP=1e-6, INIT_RYR=1, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    return (srs.Simulation(g, p, 2, 32, srs.ENGINE_RESIDENT, seeds=[3, 4], cluster_size=C, threads_per_cta=T),
            srs.Simulation(g, p, 2, 32, srs.ENGINE_PLAIN, seeds=[3, 4]))


def _same(x, y):
    for r in range(2):
        u, v = x.get_state(r), y.get_state(r)
        for k in u:
            assert np.array_equal(u[k], v[k]), (r, k)


@pytest.mark.parametrize("C,T", CONFIGS)
def test_steps_on_their_way_keep_their_constants(srs, tmp_path, C, T):
    x, y = _pair(srs, tmp_path, C, T)
    batch = srs.Batch([x], steps_per_launch=256)
    batch.advance_async(1024)
    x.set_globals(60.0, 900.0)
    batch.synchronize()
    y.explicit_step(1024)
    _same(x, y)


@pytest.mark.parametrize("C,T", CONFIGS)
@pytest.mark.parametrize("n", [20, 532])  # by one launch; by replays and a launch
def test_steps_after_take_the_new_constants(srs, tmp_path, C, T, n):
    x, y = _pair(srs, tmp_path, C, T)
    batch = srs.Batch([x], steps_per_launch=256)
    batch.advance_async(n)
    x.set_globals(60.0, 900.0)
    batch.advance_async(n)
    batch.synchronize()
    y.explicit_step(n)
    y.set_globals(60.0, 900.0)
    y.explicit_step(n)
    _same(x, y)
