"""Allocation-free steps of the small form keep nothing between calls: two
simulations stepped on two streams at once, with buffers of their own, and one
stepped alone afterwards, all bit for bit with the regular FP64 engine."""
import ctypes as C

import numpy as np
import pytest

from srs_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


class _Steps:
    def __init__(self, srs, g, p, seeds, nogating):
        import torch
        self.srs, self.nogating, R, N = srs, nogating, len(seeds), g.n_ele
        self.reals = np.array(p.reals[:], np.float64)
        self.seeds = np.array(seeds, np.uint64)
        el, ch = g.elements(), g.channels()
        aij, nij, br = g.operator()
        per = [[] for _ in range(N)]
        for kind, name in enumerate(("ryr_ele", "ryr_jsr", "lcc_ele")):
            for i, e in enumerate(ch[name]):
                per[e].append((kind, i))
        flags = (el["domain"] == 1).astype(np.int32) | (el["tropc"] != 0).astype(np.int32) << 1 | \
            np.array([4 if v else 0 for v in per], np.int32)
        sim = srs.Simulation(g, p, R, 64, srs.ENGINE_PLAIN, seeds=seeds)
        st0 = [sim.get_state(r) for r in range(R)]
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.t = dict(
            aij=T(aij), nij=T(nij), br4=T(np.concatenate([br[k * N:(k + 1) * N] for k in (0, 1, 2, 5)])),
            v0=T(el["V0"]), bhi=T(el["TT"] * self.reals[27] / (el["V0"] * 1e-15)),
            blo=T(el["TT"] * self.reals[29] / (el["V0"] * 1e-15)), flags=T(flags),
            chan_ptr=T(np.cumsum([0] + [len(v) for v in per]).astype(np.int32)),
            chan_list=T(np.array([x for v in per for kc in v for x in kc], np.int32)),
            ryr_ele=T(ch["ryr_ele"]), ryr_jsr=T(ch["ryr_jsr"]), ryr_nb=T(ch["ryr_nb"]), lcc_ele=T(ch["lcc_ele"]),
            ryr_states=T(np.concatenate([s["ryr"] for s in st0])),
            lcc_states=T(np.concatenate([s["lcc"] for s in st0])),
            lccv_states=T(np.concatenate([s["lccv"] for s in st0])),
            residuals=T(np.concatenate([s["residuals"] for s in st0])),
            status=torch.zeros(1, dtype=torch.int32, device="cuda"))
        self.S = [T(np.concatenate([s["states"] for s in st0])), T(np.zeros(R * 6 * N))]
        self.g, self.sim, self.k = g, sim, 0

    def step(self, stream):
        d = self.srs.NoallocStep()
        d.n_ele, d.n_realizations, d.n_ryr, d.n_lcc = self.g.n_ele, len(self.seeds), self.g.n_ryr, self.g.n_lcc
        for name, t in self.t.items():
            setattr(d, name, t.data_ptr())
        d.states_in, d.states_out = self.S[self.k % 2].data_ptr(), self.S[(self.k + 1) % 2].data_ptr()
        d.reals = self.reals.ctypes.data_as(C.c_void_p).value
        d.seeds = self.seeds.ctypes.data_as(C.c_void_p).value
        d.step, d.v_m, d.ca_nsr, d.nogating = self.k, self.reals[15], self.reals[16], self.nogating
        d.stream = stream.cuda_stream
        self.srs.explicit_step_fp64_noalloc(d)
        self.k += 1

    def check(self):
        self.sim.explicit_step(self.k)
        N6, R = 6 * self.g.n_ele, len(self.seeds)
        out = self.S[self.k % 2].cpu().numpy().reshape(R, N6)
        for r in range(R):
            want = self.sim.get_state(r)
            assert np.array_equal(out[r], want["states"]), r
            for k, n in (("ryr_states", "ryr"), ("lcc_states", "lcc"), ("lccv_states", "lccv"),
                         ("residuals", "residuals")):
                assert np.array_equal(self.t[k].cpu().numpy().reshape(R, -1)[r], want[n]), (r, n)
        assert int(self.t["status"].item()) == 0


# 12 tiles a realization: few blocks, several waves' worth, and coupled RyRs
@pytest.mark.parametrize("R,astar,nogating", [(3, 0.0, 0), (70, 0.0, 0), (5, 0.2, 0), (2, 0.0, 1)])
def test_overlapping_small_steps(srs, tmp_path, R, astar, nogating):
    import torch
    base = str(tmp_path / "m")
    srs.write_box_mesh(base, **wl.TINY_DYAD)
    p = srs.default_parameters().set(T_STEP=2e-6, INIT_RYR=4, RYR_K_PLUS=30.0, RYR_K_MINUS=4e3, RYR_A_STAR=astar,
                                     FLAG_NO_GATING=nogating)
    g = srs.Grid(p, base)
    a, b, alone = (_Steps(srs, g, p, list(range(s, s + R)), nogating) for s in (1, 1001, 2001))
    torch.cuda.synchronize()
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(30):
        a.step(sa)
        b.step(sb)
    torch.cuda.synchronize()
    for _ in range(3):
        alone.step(torch.cuda.current_stream())
    torch.cuda.synchronize()
    for s in (a, b, alone):
        s.check()
