"""The bytes of a reset that a simulation states: control blocks, residuals,
channel states and the arrival counter of each realization."""
import pytest

from conftest import GOLDEN_MESH, params_from_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,eng", [(64, 0), (32, 0), (32, 1)])
def test_reset_bytes(srs, prec, eng):
    p, _ = params_from_golden(srs, "spark")
    g = srs.Grid(p, GOLDEN_MESH)
    c = srs.Simulation(g, p, 5, prec, eng).config()
    per = 8 * (g.n_ryr + g.n_lcc) + 4 * (g.n_ryr + 2 * g.n_lcc) + 4
    assert c["reset_h2d_bytes"] == 5 * per + c["ctl_bytes"]
