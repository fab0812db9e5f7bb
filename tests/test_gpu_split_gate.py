"""Steps of large meshes (element update, then gating, as two launches) against
the FP64 engine: uncoupled gating, coupled gating, no gating, and the protocol of
a run (voltage clamp, RyR hold, rows at the ticks).

Both engines gate from Ca in single precision.  The FP32 engine's Ca is within a
few 1e-6 of the FP64 engine's, a channel's rate (at most Ca^2.1) within 1e-5, and a
residual, the rates' sum since the channel's last transition of less than about
ten, within 1e-4: no transition of the channels here comes that near to another
step, so their states are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def big(srs, tmp_path_factory):
    base = str(tmp_path_factory.mktemp("split") / "big")
    srs.write_box_mesh(base, box_x=3.0, box_y=3.0, box_z=3.0, foot_half_x=0.232, foot_half_y=0.232, n_foot_x=10,
                       n_foot_y=10, n_out_x=6, n_out_y=6, n_above_z=22, ryr_nx=7, ryr_ny=7, n_lcc=7,
                       lcc_half=0.232)
    return base


def _pair(srs, base, p, R=3):
    g = srs.Grid(p, base)
    assert g.n_ele >= 65536
    return [srs.Simulation(g, p, R, prec, srs.ENGINE_PLAIN, seeds=[5 + r for r in range(R)]) for prec in (32, 64)]


def _same(a, b, R=3):
    for r in range(R):
        x, y = a.get_state(r), b.get_state(r)
        for k in ("ryr", "lcc", "lccv"):
            assert np.array_equal(x[k], y[k]), (r, k)
        assert np.abs(x["residuals"] - y["residuals"]).max() < 1e-4
    return a.get_state(0)


@pytest.mark.parametrize("astar", [0.0, 0.4])
@pytest.mark.parametrize("nogating", [0, 1])
def test_gating_after_the_update(srs, big, astar, nogating):
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=24, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3, RYR_A_STAR=astar,
                                     FLAG_NO_GATING=nogating)
    a, b = _pair(srs, big, p)
    r0 = a.get_state(0)["residuals"]
    for n in (1, 32, 35):
        a.explicit_step(n)
        b.explicit_step(n)
        x = _same(a, b)
    assert np.array_equal(x["residuals"], r0) == bool(nogating)


@pytest.mark.parametrize("clamp", [0, 1])
def test_run_protocol(srs, big, clamp):
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=24, T_FINAL=1.4e-4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3,
                                     OUTPUT_STATES_INTERVAL=2e-5, FLAG_V_CLAMP=clamp)
    a, b = _pair(srs, big, p)
    ra, rb = a.run_simulation(), b.run_simulation()
    _same(a, b)
    for x, y in zip(ra[0], rb[0]):
        assert len(x) > 3 and np.array_equal(x[:, [0, 2, 3]], y[:, [0, 2, 3]])  # t, open RyRs, open LCCs
        np.testing.assert_allclose(x[:, [1, 4, 5, 6]], y[:, [1, 4, 5, 6]], rtol=1e-4)


def test_rows_of_many_channels(srs, tmp_path):
    """Rows whose channels' Ca is gathered beforehand (up to 2,048 values) and read in
    place: the same sums, up to the engine's Ca."""
    for n in (20, 34):  # 400 and 1,156 RyRs: 807 and 2,319 values
        base = str(tmp_path / str(n))
        srs.write_box_mesh(base, box_x=3.0, box_y=3.0, box_z=3.0, foot_half_x=0.6, foot_half_y=0.6, n_foot_x=10,
                           n_foot_y=10, n_out_x=6, n_out_y=6, n_above_z=22, ryr_nx=n, ryr_ny=n, n_lcc=7,
                           lcc_half=0.5)
        p = srs.default_parameters().set(T_STEP=1e-6, INIT_RYR=24, T_FINAL=1e-5, OUTPUT_STATES_INTERVAL=3e-6)
        a, b = _pair(srs, base, p, 2)
        assert (2 * a.grid.n_ryr + a.grid.n_lcc <= 2048) == (n == 20)
        ra, rb = a.run_simulation(), b.run_simulation()
        for x, y in zip(ra[0], rb[0]):
            assert len(x) > 3 and np.array_equal(x[:, [0, 2, 3]], y[:, [0, 2, 3]])
            np.testing.assert_allclose(x[:, [1, 4, 5, 6]], y[:, [1, 4, 5, 6]], rtol=1e-4)
