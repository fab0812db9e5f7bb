"""A step barrier of the looping plain engines that gives up: every call that
waits for the device says so until the next reset, and a run after it is right."""
import numpy as np
import pytest

from conftest import LINESCAN_DESC
from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
TIMEOUT = -8


@pytest.fixture(scope="module")
def mesh(srs, tmp_path_factory):
    base = str(tmp_path_factory.mktemp("m") / "m")
    srs.write_box_mesh(base, **wl.config2_mesh_specs()[0])
    return base


def _sim(srs, mesh, prec, R, **over):
    p = srs.default_parameters().set(T_STEP=2e-6, T_FINAL=1e-4, OUTPUT_STATES_INTERVAL=5e-5, INIT_RYR=4,
                                     RYR_K_PLUS=30.0, RYR_K_MINUS=4e3, **over)
    return srs.Simulation(srs.Grid(p, mesh), p, R, prec, srs.ENGINE_PLAIN, seeds=list(range(5, 5 + R)))


def _raises(srs, f):
    with pytest.raises(srs.SrsError) as e:
        f()
    assert e.value.status == TIMEOUT


def _same(a, b):
    for r in range(a.R):
        x, y = a.get_state(r), b.get_state(r)
        for k in x:
            assert np.array_equal(x[k], y[k]), (r, k)


@pytest.mark.parametrize("prec,R", [(64, 1), (32, 3)])
def test_every_waiting_call_reports_it(srs, mesh, prec, R):
    s, good = _sim(srs, mesh, prec, R), _sim(srs, mesh, prec, R)
    s.linescan_setup(**LINESCAN_DESC)
    calls = [lambda: s.explicit_step(7), lambda: s.run_simulation(), lambda: s.time_advance(8),
             lambda: (s.advance_async(8), s.synchronize()), lambda: (s.advance_async(8), s.get_state(0)),
             lambda: (s.advance_async(8), s.linescan()), lambda: (s.advance_async(8), s.total_ca())]
    for f in calls:
        s.set_wait_limit(0)
        _raises(srs, f)
        assert s.status() & 2
        # not forgotten by the call that said so, nor passed by a longer limit
        s.set_wait_limit(64)
        _raises(srs, lambda: s.explicit_step(6))
        _raises(srs, lambda: s.get_state(0))
        s.reset()
        good.reset()
        s.explicit_step(9)
        good.explicit_step(9)
        _same(s, good)
        s.reset()


def test_adjoint_reports_it(srs, mesh):
    s, good = _sim(srs, mesh, 32, 2), _sim(srs, mesh, 32, 2)
    for x in (s, good):
        x.linescan_setup(**LINESCAN_DESC)
    _, f0 = s.linescan()
    desc = dict(n_steps=24, tick_every=4, f0=f0, checkpoint_every=8)
    # the first forward pass, and every launch after it in the same call
    s.set_wait_limit(0)
    _raises(srs, lambda: s.adjoint(**desc))
    s.set_wait_limit(64)
    _raises(srs, lambda: s.adjoint(**desc))
    s.reset()
    a, b = s.adjoint(**desc), good.adjoint(**desc)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_wait_limit_is_checked(srs, mesh):
    s = _sim(srs, mesh, 32, 1)
    with pytest.raises(srs.SrsError) as e:
        s.set_wait_limit(-1)
    assert e.value.status == -1
    # fidelity runs take a launch a step: nothing waits
    s = _sim(srs, mesh, 32, 1, FLAG_FIDELITY_SIM=1)
    with pytest.raises(srs.SrsError):
        s.set_wait_limit(1)
