"""Read-outs of an ensemble at the sizes where their kernels split the work:
the tiled line scan (tiles of 32 realizations, groups of eight samples,
chunks of 64 elements) and the total Ca over several blocks a realization."""
import numpy as np
import pytest

from conftest import GOLDEN_MESH, LINESCAN_DESC, linescan_weights, params_from_golden

pytestmark = pytest.mark.gpu


def _states(srs, sim, R, seed):
    """Some different state in every realization."""
    rng = np.random.RandomState(seed)
    S0 = sim.get_state(0)["states"]
    out = []
    for r in range(R):
        S = S0 * (1.0 + 0.2 * rng.rand(len(S0)))
        sim.set_state(r, states=S)
        out.append(sim.get_state(r)["states"])  # as the engine holds it
    return out


# FP64 sums of a few hundred positive terms in another order: 1e-12 relative,
# the bar of the untiled form's test
@pytest.mark.parametrize("prec,eng", [(64, 0), (32, 0), (32, 1)])
@pytest.mark.parametrize("R,res", [(15, 0.02), (16, 0.05), (33, 0.004), (64, 0.0061)])
def test_linescan_tiles(srs, prec, eng, R, res):
    p, _ = params_from_golden(srs, "spark")
    g = srs.Grid(p, GOLDEN_MESH)
    # a threshold that gives each sample its own part of the mesh
    desc = dict(LINESCAN_DESC, res=res, r_thresh=0.03)
    sim = srs.Simulation(g, p, R, prec, eng, seeds=list(range(1, R + 1)))
    ns = sim.linescan_setup(**desc)
    states = _states(srs, sim, R, 3)
    F, _ = sim.linescan()
    W, pad = linescan_weights(g, desc)
    N = g.n_ele
    want = np.array([pad + W @ S[5 * N:] for S in states])
    assert F.shape == want.shape == (R, ns)
    assert np.allclose(F, want, rtol=1e-12, atol=0)


@pytest.mark.parametrize("prec,eng,R", [(64, 0, 1), (32, 0, 3), (32, 1, 40)])
def test_total_ca_over_several_blocks(srs, box_mesh, prec, eng, R):
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=24)
    g = srs.Grid(p, box_mesh[0])
    sim = srs.Simulation(g, p, R, prec, eng, seeds=list(range(1, R + 1)))
    states = _states(srs, sim, R, 4)
    el, N = g.elements(), g.n_ele
    bhi = el["TT"] * p.reals[srs.R["B_TOT_SL_HI"]] / (el["V0"] * 1e-15)
    for got, S in zip(sim.total_ca(), states):
        c = S[:N]
        t = el["V0"] * (S.reshape(6, N).sum(0) + bhi * c / (p.reals[srs.R["K_D_SL_HI"]] + c))
        want = [t[el["domain"] == 0].sum(), t[el["domain"] == 1].sum()]
        assert np.allclose(got, want, rtol=1e-12, atol=0)
