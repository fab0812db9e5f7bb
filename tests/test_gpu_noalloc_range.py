"""The allocation-free step on both sides of the size at which its update is dealt
to four warps a tile (912 tiles of 32 elements), called step by step and captured
into a graph, bit for bit with the regular FP64 engine."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 48, 49])
@pytest.mark.parametrize("capture", [0, 1])
def test_noalloc_sizes(srs, tmp_path, R, capture):
    import torch
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, box_x=0.5, box_y=0.5, box_z=0.5, foot_half_x=0.1, foot_half_y=0.1, n_foot_x=2,
                       n_foot_y=3, n_out_x=1, n_out_y=1, n_above_z=3, ryr_nx=3, ryr_ny=3, n_lcc=2, lcc_half=0.1)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3)
    g = srs.Grid(p, base)
    N = g.n_ele
    assert (N + 31) // 32 * 48 == 912
    seeds = np.arange(11, 11 + R, dtype=np.uint64)
    sim = srs.Simulation(g, p, R, 64, srs.ENGINE_PLAIN, seeds=list(seeds))
    st0 = [sim.get_state(r) for r in range(R)]
    steps = 4
    sim.explicit_step(steps)
    el, ch = g.elements(), g.channels()
    aij, nij, br = g.operator()
    reals = np.array(p.reals[:], np.float64)
    per = [[] for _ in range(N)]
    for kind, name in enumerate(("ryr_ele", "ryr_jsr", "lcc_ele")):
        for i, e in enumerate(ch[name]):
            per[e].append((kind, i))
    flags = (el["domain"] == 1).astype(np.int32) | (el["tropc"] != 0).astype(np.int32) << 1 | \
        np.array([4 if v else 0 for v in per], np.int32)
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    bufs = dict(aij=T(aij), nij=T(nij), br4=T(np.concatenate([br[k * N:(k + 1) * N] for k in (0, 1, 2, 5)])),
                v0=T(el["V0"]), bhi=T(el["TT"] * reals[27] / (el["V0"] * 1e-15)),
                blo=T(el["TT"] * reals[29] / (el["V0"] * 1e-15)), flags=T(flags),
                chan_ptr=T(np.cumsum([0] + [len(v) for v in per]).astype(np.int32)),
                chan_list=T(np.array([x for v in per for kc in v for x in kc], np.int32)),
                ryr_ele=T(ch["ryr_ele"]), ryr_jsr=T(ch["ryr_jsr"]), ryr_nb=T(ch["ryr_nb"]), lcc_ele=T(ch["lcc_ele"]))
    S = [T(np.concatenate([s["states"] for s in st0])), torch.zeros(R * 6 * N, dtype=torch.float64, device="cuda")]
    chan = {k: T(np.concatenate([s[n] for s in st0])) for k, n in
            (("ryr_states", "ryr"), ("lcc_states", "lcc"), ("lccv_states", "lccv"), ("residuals", "residuals"))}
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def step(k):
        d = srs.NoallocStep()
        d.n_ele, d.n_realizations, d.n_ryr, d.n_lcc = N, R, g.n_ryr, g.n_lcc
        for name, t in list(bufs.items()) + list(chan.items()):
            setattr(d, name, t.data_ptr())
        d.states_in, d.states_out, d.status = S[k % 2].data_ptr(), S[(k + 1) % 2].data_ptr(), status.data_ptr()
        d.reals = reals.ctypes.data_as(C.c_void_p).value
        d.seeds = seeds.ctypes.data_as(C.c_void_p).value
        d.step, d.v_m, d.ca_nsr, d.nogating = k, reals[15], reals[16], 0
        d.stream = torch.cuda.current_stream().cuda_stream
        srs.explicit_step_fp64_noalloc(d)

    if capture:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for k in range(steps):
                step(k)
        graph.replay()
    else:
        for k in range(steps):
            step(k)
    torch.cuda.synchronize()
    out = S[steps % 2].cpu().numpy().reshape(R, 6 * N)
    for r in range(R):
        want = sim.get_state(r)
        assert np.array_equal(out[r], want["states"]), r
        for k, n in (("ryr_states", "ryr"), ("lcc_states", "lcc"), ("lccv_states", "lccv"), ("residuals", "residuals")):
            assert np.array_equal(chan[k].cpu().numpy().reshape(R, -1)[r], want[n]), (r, n)
    assert int(status.item()) == 0
