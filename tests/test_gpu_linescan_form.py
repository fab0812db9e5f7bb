"""Which of its two forms the line scan takes (one kernel by sample, two tiled),
and that both give the weighted sums at the tiles' edges."""
import numpy as np
import pytest

from conftest import LINESCAN_DESC
from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# 6,000 elements, not a multiple of the chunk's 64; samples not a multiple of
# eight; 33 and 40 realizations: a tile of one, and a part of a warp's lanes
@pytest.mark.parametrize("prec,eng,R,over,tiled", [
    (32, 0, 40, dict(res=0.0033), True), (32, 1, 33, dict(res=0.0027), True), (64, 0, 97, dict(res=0.0031), True),
    (32, 0, 12, dict(res=0.0005), True), (32, 0, 200, dict(res=0.05, r_thresh=0.01), False),
    (32, 1, 64, dict(res=0.2), False), (64, 0, 1, dict(), False)])
def test_form_and_sums(srs, tmp_path, prec, eng, R, over, tiled):
    from oracle import linescan
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **wl.config2_mesh_specs()[0])
    p = srs.default_parameters().set(T_STEP=9e-7, INIT_RYR=4)
    g = srs.Grid(p, base)
    N = g.n_ele
    assert N % 64 != 0
    desc = dict(LINESCAN_DESC, **over)
    sim = srs.Simulation(g, p, R, prec, eng, seeds=list(range(1, R + 1)))
    ns = sim.linescan_setup(**desc)
    rng = np.random.RandomState(2)
    S0 = sim.get_state(0)["states"]
    for r in range(R):
        sim.set_state(r, states=S0 * (1.0 + 0.2 * rng.rand(len(S0))))
    n0 = sim.config()["kernel_launches"]
    F, _ = sim.linescan()
    assert sim.config()["kernel_launches"] - n0 == (2 if tiled else 1)
    W, pad = linescan.weights(base, g.elements()["order"], desc)
    states = [sim.get_state(r)["states"] for r in (0, R // 2, R - 1)]
    # FP64 sums of positive terms in another order
    assert np.allclose(F[[0, R // 2, R - 1]], [pad + W @ S[5 * N:] for S in states], rtol=1e-12, atol=0)
    assert F.shape == (R, ns)
