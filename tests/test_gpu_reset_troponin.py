"""Reset of meshes whose troponin indicator is not 0 or 1 in some elements: the
equilibrium has troponin times the indicator there, at rest it counts once."""
import os
import shutil

import numpy as np
import pytest

from conftest import GOLDEN_MESH, params_from_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,eng,R", [(64, 0, 2), (32, 0, 3), (32, 1, 5)])
def test_reset_is_the_equilibrium(srs, tmp_path, prec, eng, R):
    d = os.path.dirname(GOLDEN_MESH)
    for f in os.listdir(d):
        shutil.copy(os.path.join(d, f), tmp_path)
    path = tmp_path / (os.path.basename(GOLDEN_MESH) + "_tet_properties.txt")
    lines = path.read_text().split("\n")
    for i, line in enumerate(lines[2:], 2):
        w = line.split()
        if len(w) == 8 and w[7] == "0" and i % 5 < 2:
            w[6] = str(2 + i % 5)
            lines[i] = " ".join(w)
    path.write_text("\n".join(lines))
    p, _ = params_from_golden(srs, "spark")
    g = srs.Grid(p, str(tmp_path / os.path.basename(GOLDEN_MESH)))
    assert set(g.elements()["tropc"]) >= {2, 3}
    want = g.initial_states(p)
    sim = srs.Simulation(g, p, R, prec, eng, seeds=list(range(1, R + 1)))
    for _ in range(2):
        for r in range(R):
            # FP32: one rounding of the deviation, which is below twice the value
            assert np.allclose(sim.get_state(r)["states"], want, rtol=2 ** -23 if prec == 32 else 0, atol=0)
        sim.explicit_step(3)
        sim.reset()
