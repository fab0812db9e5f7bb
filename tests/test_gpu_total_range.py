"""Total Ca of the FP32 engines over the whole range of their numbers: deviations
and compensations are widened to double by integer operations, which is exact for
zeros, denormals, the largest values, infinities and NaNs alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [0, 1])
def test_total_ca_of_any_number(srs, tmp_path, engine):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, box_x=0.5, box_y=0.5, box_z=0.5, foot_half_x=0.1, foot_half_y=0.1, n_foot_x=2,
                       n_foot_y=3, n_out_x=1, n_out_y=1, n_above_z=3, ryr_nx=3, ryr_ny=3, n_lcc=2, lcc_half=0.1)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4)
    g = srs.Grid(p, base)
    el, N = g.elements(), g.n_ele
    dev = np.float32([0.0, -0.0, 1e-45, -3e-42, 1.1754942e-38, 1.17549435e-38, -1.1754945e-38, 1e-30, 3.0, -0.015,
                      2.0 ** -24, 1.0 - 2.0 ** -24, 65504.0, 1e15, 3.4028235e38, np.inf, -np.inf, np.nan])
    sim = srs.Simulation(g, p, len(dev), 32, engine, seeds=list(range(len(dev))))
    S0 = sim.get_state(0)["states"].reshape(6, N)
    cyt = np.flatnonzero(el["domain"] == 0)
    bhi = el["TT"] * p.reals[srs.R["B_TOT_SL_HI"]] / (el["V0"] * 1e-15)
    off, on = cyt[bhi[cyt] == 0][7], cyt[bhi[cyt] != 0][3]  # an element off the membrane, one on it
    for sp, j in ((0, off), (0, on), (1, off), (2, on), (5, off)):
        for r, d in enumerate(dev):
            S = S0.copy()
            S[sp, j] += float(d)
            sim.set_state(r, states=S.ravel())
        with np.errstate(all="ignore"):
            for r, got in enumerate(sim.total_ca()):
                S = sim.get_state(r)["states"].reshape(6, N)
                c = S[0]
                t = el["V0"] * (S.sum(0) + bhi * c / (p.reals[srs.R["K_D_SL_HI"]] + c))
                # blocks add up to a thousand terms in another order: 1e-13 of the largest of them
                for k in (0, 1):
                    want = t[el["domain"] == k].sum()
                    if np.isfinite(want):
                        assert abs(got[k] - want) <= 1e-13 * np.abs(t[el["domain"] == k]).sum(), (sp, j, r)
                    else:
                        assert str(got[k]) == str(want), (sp, j, r, got, want)
