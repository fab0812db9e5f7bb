"""Exchange of a realization's state with the device and explicit steps in
pieces, bit for bit: what is set is what is read (to the engines' rounding of
the deviation from rest, which is known exactly), through the staged and the
direct copy, and an odd number of steps, after which the engines' two state
buffers have changed places, leaves what the same steps leave in one call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENGINES = [(64, "PLAIN"), (32, "PLAIN"), (32, "RESIDENT")]


@pytest.fixture(scope="module")
def meshes(srs, tmp_path_factory):
    """Below and above the size at which the state is copied without staging (4 MB: 87,381 elements)."""
    out = {}
    for name, box in (("small", 0.5), ("large", 3.0)):
        base = str(tmp_path_factory.mktemp("state") / name)
        srs.write_box_mesh(base, box_x=box, box_y=box, box_z=min(box, 1.5), foot_half_x=0.1, foot_half_y=0.1,
                           n_foot_x=2, n_foot_y=3, n_out_x=(1 if name == "small" else 20),
                           n_out_y=(1 if name == "small" else 20), n_above_z=(3 if name == "small" else 10),
                           ryr_nx=3, ryr_ny=3, n_lcc=2, lcc_half=0.1)
        out[name] = base
    return out


def _params(srs):
    return srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)


@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("prec,engine", ENGINES)
def test_state_round_trip(srs, meshes, size, prec, engine):
    g = srs.Grid(_params(srs), meshes[size])
    N = g.n_ele
    assert (48 * N > 4 << 20) == (size == "large"), N
    if size == "large" and engine == "RESIDENT":
        pytest.skip("beyond the clusters' shared memory")
    sim = srs.Simulation(g, _params(srs), 3, prec, getattr(srs, "ENGINE_" + engine), seeds=[1, 2, 3])
    rest = sim.get_state(1)["states"]
    assert np.array_equal(rest, sim.get_state(2)["states"])
    rng = np.random.default_rng(5)
    # species an element does not hold rest at zero and stay there
    want = rest * (1 + 0.2 * rng.random(rest.shape))
    sim.set_state(1, want)
    got = sim.get_state(1)["states"]
    if prec == 32:
        want = rest + (want - rest).astype(np.float32).astype(np.float64)
    assert np.array_equal(got, want)
    assert np.array_equal(sim.get_state(0)["states"], rest)
    sim.explicit_step(3)
    sim.reset()
    for r in range(3):
        assert np.array_equal(sim.get_state(r)["states"], rest)


@pytest.mark.parametrize("fidelity", [0, 1])
@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("prec", [64, 32])
def test_explicit_steps_in_pieces(srs, meshes, prec, size, fidelity):
    p = _params(srs).set(FLAG_FIDELITY_SIM=fidelity)
    g = srs.Grid(p, meshes[size])
    R = 3 if size == "small" else 12  # the larger one beyond what one launch holds
    a, b = (srs.Simulation(g, p, R, prec, srs.ENGINE_PLAIN, seeds=list(range(R))) for _ in range(2))
    pieces = (1, 33, 34, 1, 0, 2, 35)
    for n in pieces:
        a.explicit_step(n)
    b.explicit_step(sum(pieces))
    for r in (0, R - 1):
        x, y = a.get_state(r), b.get_state(r)
        for k in ("states", "ryr", "lcc", "lccv", "residuals"):
            assert np.array_equal(x[k], y[k]), (r, k)
    assert np.array_equal(a.total_ca(), b.total_ca())


@pytest.mark.parametrize("prec", [64, 32])
def test_steps_after_the_end_of_a_run(srs, meshes, prec):
    """A finished realization takes no more steps: an odd number of them changes nothing."""
    p = _params(srs).set(T_FINAL=66e-6)
    g = srs.Grid(p, meshes["small"])
    sim = srs.Simulation(g, p, 3, prec, srs.ENGINE_PLAIN, seeds=[1, 2, 3])
    sim.run_simulation()
    end = [sim.get_state(r)["states"] for r in range(3)]
    for n in (1, 2, 5):
        sim.explicit_step(n)
        for r in range(3):
            assert np.array_equal(sim.get_state(r)["states"], end[r])
    sim.reset()
    sim.explicit_step(33)
    assert all(not np.array_equal(sim.get_state(r)["states"], end[r]) for r in range(3))


def test_state_gradient_in_chunks(srs, meshes):
    """dL/d(initial state) of more realizations than are converted at a time (64 MB)."""
    from conftest import LINESCAN_DESC
    p = _params(srs)
    g = srs.Grid(p, meshes["large"])
    R = 12
    assert R * 48 * g.n_ele > 64 << 20
    gs = []
    for seeds in (list(range(R)), [R - 1]):
        sim = srs.Simulation(g, p, len(seeds), 32, srs.ENGINE_PLAIN, seeds=seeds)
        n = sim.linescan_setup(**LINESCAN_DESC)
        f0 = sim.linescan()[1]
        assert n == len(f0)
        gs.append(sim.adjoint(4, 2, f0, grad_state=True)[2])
    assert np.abs(gs[0][-1]).max() > 0
    assert np.array_equal(gs[0][-1], gs[1][0])
