"""The plain engines' steps in one launch against one launch per step, bit for
bit, where a thread takes one, two and four elements, where the last block is
ragged and where the number of steps is odd.  A parameter set with the fidelity
criterion takes the one-launch-per-step form; explicit steps do not evaluate
the criterion, so both forms compute the same thing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b, realizations):
    for r in realizations:
        x, y = a.get_state(r), b.get_state(r)
        for k in ("states", "ryr", "lcc", "lccv", "residuals"):
            assert np.array_equal(x[k], y[k]), (r, k)


def _sims(srs, g, p, R, prec):
    seeds = list(range(3, 3 + R))
    q = p.copy().set(FLAG_FIDELITY_SIM=1)
    return [srs.Simulation(g, v, R, prec, srs.ENGINE_PLAIN, seeds=seeds) for v in (p, q)]


@pytest.mark.parametrize("prec,R", [(64, 1), (64, 4), (64, 9), (32, 1), (32, 15), (32, 33)])
def test_loop_equals_single_steps(srs, box_mesh, prec, R):
    # every RyR's rate raised, so that channels open and close in a few steps
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=24, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, box_mesh[0])
    loop, single = _sims(srs, g, p, R, prec)
    for n in (1, 2, 33, 64):
        k0 = [s.config()["kernel_launches"] for s in (loop, single)]
        loop.explicit_step(n)
        single.explicit_step(n)
        k1 = [s.config()["kernel_launches"] for s in (loop, single)]
        assert k1[0] - k0[0] == 1 and k1[1] - k0[1] == n  # both forms ran
        _same(loop, single, (0, R // 2, R - 1))
    assert not np.array_equal(loop.get_state(0)["ryr"], np.eye(g.n_ryr, dtype=np.int32)[24])


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("noflux", [1, 0])
def test_loop_on_a_small_mesh(srs, tmp_path, prec, noflux):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, box_x=0.4, box_y=0.4, box_z=0.4, foot_half_x=0.1, foot_half_y=0.1, n_foot_x=2,
                       n_foot_y=3, n_out_x=1, n_out_y=1, n_above_z=3, ryr_nx=3, ryr_ny=3, n_lcc=2, lcc_half=0.1)
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3,
                                     FLAG_NO_FLUX_BOUNDARY=noflux)
    g = srs.Grid(p, base)
    loop, single = _sims(srs, g, p, 5, prec)
    for n in (7, 120):
        loop.explicit_step(n)
        single.explicit_step(n)
        _same(loop, single, range(5))


def test_long_loop_crosses_launches(srs, tmp_path):
    """More steps than one launch takes, and an odd rest."""
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, box_x=0.4, box_y=0.4, box_z=0.4, foot_half_x=0.1, foot_half_y=0.1, n_foot_x=2,
                       n_foot_y=2, n_out_x=1, n_out_y=1, n_above_z=2, ryr_nx=3, ryr_ny=3, n_lcc=2, lcc_half=0.1)
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=4)
    g = srs.Grid(p, base)
    loop, single = _sims(srs, g, p, 2, 32)
    for s in (loop, single):
        s.explicit_step(2 * 4096 + 15)
    _same(loop, single, range(2))
