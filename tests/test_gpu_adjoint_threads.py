"""Threads of a reverse-sweep CTA: what the library chooses can be named too, the
result does not depend on it, and numbers outside the range are refused."""
import numpy as np
import pytest

from conftest import LINESCAN_DESC

pytestmark = pytest.mark.gpu


def test_thread_counts(srs, box_mesh):
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=24)
    R = 3
    sim = srs.Simulation(srs.Grid(p, box_mesh[0]), p, R, 32, srs.ENGINE_RESIDENT, seeds=list(range(1, R + 1)))
    sim.linescan_setup(**LINESCAN_DESC)
    _, f0 = sim.linescan()

    def run(threads):
        sim.reset()
        return sim.adjoint(n_steps=40, tick_every=10, f0=f0, grad_state=True, threads_per_cta=threads)

    loss, grad, gs = run(0)
    for threads in (64, 512, 544, 608, 640):
        x, y, z = run(threads)
        assert np.array_equal(x, loss) and np.array_equal(z, gs), threads
        assert np.allclose(y, grad, rtol=1e-5, atol=0), threads  # grouping of its FP32 partial sums
    for threads in (-32, 32, 100, 672):
        with pytest.raises(srs.SrsError) as e:
            run(threads)
        assert e.value.status == -1
