"""Step loops of the plain engines where the device is not theirs alone: a launch
that is refused (the steps are then taken one launch each), and two simulations
stepping at once on two threads.  Bit for bit with the undisturbed run."""
import threading

import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def _sims(srs, tmp_path, prec, R, n):
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **wl.config2_mesh_specs()[0])
    p = srs.default_parameters().set(T_STEP=2e-6, T_FINAL=2e-4, OUTPUT_STATES_INTERVAL=5e-5, INIT_RYR=4,
                                     RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    return [srs.Simulation(g, p, R, prec, srs.ENGINE_PLAIN, seeds=list(range(5, 5 + R))) for _ in range(n)]


def _same(a, b):
    for r in {0, a.R // 2, a.R - 1}:
        x, y = a.get_state(r), b.get_state(r)
        for k in x:
            assert np.array_equal(x[k], y[k]), (r, k)


# more shared memory than a block can have, and (768 blocks, five of them to an
# SM) than all blocks can have at once
@pytest.mark.parametrize("prec,R,nbytes", [(64, 1, 1 << 20), (32, 3, 1 << 20), (32, 16, 40960)])
def test_refused_launch(srs, tmp_path, prec, R, nbytes):
    a, b = _sims(srs, tmp_path, prec, R, 2)
    b.set_loop_reserve(nbytes)
    n0 = b.config()["kernel_launches"]
    for s in (a, b):
        s.explicit_step(3)
        s.explicit_step(70)
    assert b.config()["kernel_launches"] - n0 == 73  # one a step
    _same(a, b)
    for s in (a, b):
        s.reset()
    (rows, t, n), (rows_b, t_b, n_b) = a.run_simulation(), b.run_simulation()
    assert np.array_equal(t, t_b) and np.array_equal(n, n_b)
    assert all(np.array_equal(x, y) for x, y in zip(rows, rows_b))
    _same(a, b)


# 189 blocks a realization in FP64, 48 in FP32, 912 places on the device: both
# simulations fit at once, and neither leaves the other room
@pytest.mark.parametrize("prec,R", [(64, 1), (64, 4), (32, 1), (32, 16)])
def test_two_threads(srs, tmp_path, prec, R):
    a, b, ref = _sims(srs, tmp_path, prec, R, 3)
    errors = []

    def run(s):
        try:
            for _ in range(20):
                s.explicit_step(100)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(s,)) for s in (a, b)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for _ in range(20):
        ref.explicit_step(100)
    _same(a, ref)
    _same(b, ref)
