"""The forms of the FP64 step by launch at the edges of their ranges: an element dealt
to four warps up to 912 tiles and from 913 to 1,600 blocks of 64, else a thread an
element.  Six blocks of 64 (twelve tiles) a realization; bit for bit the step of one."""
import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [76, 77, 152, 153, 266, 267])
@pytest.mark.parametrize("coupled", [False, True])
def test_forms_agree(srs, tmp_path, R, coupled):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **wl.TINY_DYAD)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=1, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3,
                                     RYR_A_STAR=1.0 if coupled else 0.0)
    g = srs.Grid(p, base)
    assert g.n_ele == 384
    seeds = list(range(1, R + 1))
    many = srs.Simulation(g, p, R, 64, srs.ENGINE_PLAIN, seeds=seeds)
    for _ in range(9):
        many.explicit_step(1)
    for r in (0, R - 1):
        one = srs.Simulation(g, p, 1, 64, srs.ENGINE_PLAIN, seeds=[seeds[r]])
        one.explicit_step(9)
        u, v = many.get_state(r), one.get_state(0)
        for k in u:
            assert np.array_equal(u[k], v[k]), (r, k)
