"""Line scans set up again and again: each takes the place of the one before, on
the device too, and gives what the only one of a simulation gives."""
import numpy as np
import pytest

from conftest import LINESCAN_DESC

pytestmark = pytest.mark.gpu


# tiled (R >= 16) and by sample; with the adjoint's own copies of the weights
@pytest.mark.parametrize("R,eng", [(16, 1), (32, 0), (4, 1)])
def test_set_up_again(srs, box_mesh, R, eng):
    import torch
    p = srs.default_parameters().set(T_STEP=9e-6, INIT_RYR=24)
    g = srs.Grid(p, box_mesh[0])
    seeds = list(range(1, R + 1))
    # about 1.3 M weights, 9 to 16 MB in either form
    descs = [dict(LINESCAN_DESC, res=0.003, offset1=0.01 * k) for k in range(2)]

    def measure(s, d, adjoint):
        s.linescan_setup(**d)
        s.reset()
        s.explicit_step(8)
        F, rest = s.linescan()
        out = [F, rest]
        if adjoint:
            out += list(s.adjoint(n_steps=8, tick_every=4, f0=rest)[:2])
        return out

    free = []
    sim = srs.Simulation(g, p, R, 32, eng, seeds=seeds)
    for k in range(12):
        got = measure(sim, descs[k % 2], k >= 2)
        if k >= 10:
            alone = measure(srs.Simulation(g, p, R, 32, eng, seeds=seeds), descs[k % 2], True)
            assert all(np.array_equal(x, y) for x, y in zip(got[:3], alone))
            # the resident sweep's blocks add their FP64 sums in any order
            assert np.allclose(got[3], alone[3], rtol=1e-12, atol=0)
        free.append(torch.cuda.mem_get_info()[0])
    # from the fourth on (the adjoint's buffers are there) nothing is added
    assert free[3] - free[9] < 4 << 20, [free[0] - f for f in free]
