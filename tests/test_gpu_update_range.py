"""The FP32 element update at the limits of its in-range divisions, against the
oracle's FP32 restatement (IEEE divisions), bit for bit: Ca below, at and above
the limit, tiny and zero numerators of the rapid-buffer division, negative Ca."""
import numpy as np
import pytest

from conftest import GOLDEN_MESH, params_from_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k_d_i", [910.0, 1e-3, 1e9])  # the last two: no range the host can vouch for
def test_update_matches_oracle_at_extreme_states(srs, oracle, k_d_i):
    from oracle import Mesh
    p, _ = params_from_golden(srs, "spark")
    p.set(FLAG_NO_GATING=1, INIT_RYR=-1, K_D_i=k_d_i)
    g = srs.Grid(p, GOLDEN_MESH)
    N = g.n_ele
    sim = srs.Simulation(g, p, 1, srs.FP32, srs.ENGINE_PLAIN, seeds=[1])
    st = sim.get_state(0)
    S = st["states"].copy()
    rng = np.random.RandomState(5)
    ca = S[:N]
    pick = rng.permutation(N)
    ca[pick[:40]] = 16384.0 * (1 + rng.uniform(-1e-6, 1e-6, 40))
    ca[pick[40:80]] = rng.uniform(2e4, 3e5, 40)
    ca[pick[80:100]] = -rng.uniform(0, 12.9, 20)
    ca[pick[100:160]] += 10.0 ** rng.uniform(-20, -1, 60)
    sim.set_state(0, states=S)
    m = Mesh(oracle, GOLDEN_MESH, p.ints[9], np.array(p.reals[:]))
    f = m.to_fp32(S)
    ryr, lcc, lccv, res = (st[k].copy() for k in ("ryr", "lcc", "lccv", "residuals"))
    for n in (1, 3):
        sim.explicit_step(n)
        m.steps_fp32(f, 1, 0, n, ryr, lcc, lccv, res, gating=False, compact=True)
        assert np.array_equal(sim.get_state(0)["states"], m.from_fp32(f), equal_nan=True)
