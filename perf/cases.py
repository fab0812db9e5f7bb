"""What a user of this package has it do, as cases that can be timed.

Every case goes through the public Python entry points (srs_gb300): explicit
steps, whole RunSimulation ensembles, the allocation-free step on the caller's
own buffers, uneven multi-mesh batches, read-outs (line scan, total Ca, state)
and the adjoint.  Sizes are those of the package's workloads
(srs_gb300/workloads.py), tests and benchmark.  A parameter study is the usual
reason to run many ensembles, so the seed of a case sets the kinetic
parameters (a few per cent around DefaultSpark) and the realizations' random
streams.  Resident simulations leave cluster size and threads to the library.

`exact` is the same path in plain float64 torch.
"""
import ctypes
import functools
import math
import os
import random
import tempfile

import numpy as np
import torch

import srs_gb300 as srs
from srs_gb300 import workloads as wl

LINESCAN = dict(axis=0, offset1=0.0, offset2=0.1, x_min=-1.0, x_max=1.0, res=0.05, var_x=0.0289,
                var_y=0.1154, var_z=0.0289, r_thresh=1.0, f0_pad=0.0, pad_res=0.0, pad_min=0.0,
                pad_max=0.0, domain=(0, 0, 0, 0, 0, 0))
JITTERED = ("D_CA", "D_DYE", "V_RYR", "A_P", "K_ON_DYE", "K_OFF_DYE", "B_TOT_TRPN", "K_ON_CMDN")


def listed():
    return [
        # A host program that couples the step to its own code: one explicit
        # step per call, and the state back after a few (a 384-element mesh).
        dict(name="coupled-step", kind="step", mesh="tiny", prec=64, real=1, steps=1, calls=8),
        # A real-time loop on its own device buffers, one allocation-free
        # FP64 step per call, three realizations.
        dict(name="noalloc-loop", kind="noalloc", mesh="tiny", real=3, steps=64),
        # The plain single spark of the config mesh in FP64, with a line scan
        # at every grid-file step (the reference's own use).
        dict(name="spark-fp64", kind="spark", mesh="config", prec=64, engine="plain", real=1,
             steps=1536, frames=6),
        # A few FP32 realizations with Dirichlet faces, which only the plain
        # engine takes.
        dict(name="sparks-plain32-dirichlet", kind="spark", mesh="box", box=1.5, nf=6, no=2, na=8,
             ryr=10, prec=32, engine="plain", real=5, steps=1500, noflux=False),
        # The ensemble of the benchmark: 1024 realizations of the config mesh.
        dict(name="ensemble-1024", kind="spark", mesh="config", prec=32, engine="resident",
             real=1024, steps=1000),
        # A small odd ensemble on an odd mesh, clamped to 0 mV (LCC triggered).
        dict(name="ensemble-37-clamp", kind="spark", mesh="box", box=2.0, nf=8, no=3, na=11, ryr=25,
             prec=32, engine="resident", real=37, steps=1501, clamp=True),
        # The uneven multi-mesh batch: four meshes x two protocols x 32.
        dict(name="batch-uneven", kind="batch", real=32, steps=500),
        # The five-cluster release site at 50 nm cells (542,376 tets; the
        # benchmark's has 35 nm), 32 realizations, streamed.
        dict(name="site-32", kind="spark", mesh="site", h=0.05, prec=32, engine="plain", real=32,
             steps=64),
        # Sensitivities of the mean trace, whole trajectory kept (64 x config mesh).
        dict(name="adjoint-64", kind="adjoint", mesh="config", engine="resident", real=64,
             steps=512, tick=128, ckpt=0, mean=True),
        # The same with checkpoints, a loss per realization and dL/d(initial state).
        dict(name="adjoint-checkpointed", kind="adjoint", mesh="box", box=2.0, nf=8, no=3, na=11,
             ryr=25, engine="resident", real=21, steps=384, tick=32, ckpt=128, mean=False,
             grad_state=True),
        # The adjoint of a mesh that is streamed (69,696 tets).
        dict(name="adjoint-streamed", kind="adjoint", mesh="box", box=3.0, nf=10, no=6, na=22, ryr=49,
             engine="plain", real=8, steps=64, tick=16, ckpt=0, mean=True),
        # Reading an ensemble out: line scan, total Ca, some whole states.
        dict(name="readout-512", kind="readout", mesh="config", prec=32, engine="resident", real=512,
             steps=64),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _fills_clusters(n):
    """Whether n elements all but fill the shared memory (about 4,900 elements
    a block) of the smallest cluster that holds them; a program names the
    cluster there."""
    c = next(c for c in (1, 2, 3, 4, 5, 6, 8, 16) if n <= 5000 * c)
    return n > 4800 * (c - 0.13)


def _draw_mesh(rng, lo, hi):
    """A box dyad of between lo and hi tets (6 per hexahedron; one layer each in
    the cleft and the JSR), its cluster about as dense as the package's."""
    while True:
        nf, no, na = rng.randint(4, 11), rng.randint(1, 7), rng.randint(5, 24)
        n = 6 * (nf + 2 * no) ** 2 * (na + 2)
        if lo <= n <= hi and not _fills_clusters(n):
            break
    box = round(rng.uniform(1.5, 3.0), 2)
    return dict(mesh="box", box=box, nf=nf, no=no, na=na, ryr=rng.randint(8, 60))


def draw(rng):
    kind = rng.choice(["step", "noalloc", "spark64", "plain32", "ensemble", "ensemble", "ensemble",
                       "batch", "site", "adjoint", "adjoint-streamed", "readout"])
    if kind == "step":
        m = dict(mesh="tiny") if rng.random() < 0.5 else _draw_mesh(rng, 1500, 16000)
        return dict(kind="step", prec=rng.choice([32, 64]), real=rng.randint(1, 3),
                    steps=rng.randint(1, 5), calls=rng.randint(4, 12), **m)
    if kind == "noalloc":
        m = dict(mesh="tiny") if rng.random() < 0.5 else _draw_mesh(rng, 1500, 16000)
        return dict(kind="noalloc", real=rng.randint(1, 9), steps=rng.randint(16, 90), **m)
    if kind == "spark64":
        return dict(kind="spark", prec=64, engine="plain", real=_log_int(rng, 1, 8),
                    steps=_log_int(rng, 200, 1500), frames=rng.randint(0, 6),
                    **_draw_mesh(rng, 2000, 31000))
    if kind == "plain32":
        return dict(kind="spark", prec=32, engine="plain", real=_log_int(rng, 1, 24),
                    steps=_log_int(rng, 200, 1500), noflux=rng.random() < 0.5,
                    **_draw_mesh(rng, 2000, 60000))
    if kind == "ensemble":
        m = _draw_mesh(rng, 3000, 31000)
        real = _log_int(rng, 4, 900)
        return dict(kind="spark", prec=32, engine="resident", real=real,
                    steps=_log_int(rng, 200, 1200), clamp=rng.random() < 0.3, **m)
    if kind == "batch":
        return dict(kind="batch", real=rng.randint(9, 32), steps=rng.randint(150, 500))
    if kind == "site":
        return dict(kind="spark", mesh="site", h=round(rng.uniform(0.06, 0.09), 4), prec=32,
                    engine="plain", real=rng.randint(5, 32), steps=rng.randint(20, 64))
    if kind == "adjoint":
        return dict(kind="adjoint", engine="resident", real=_log_int(rng, 3, 64),
                    steps=rng.randint(128, 400), tick=rng.choice([16, 31, 64]),
                    ckpt=rng.choice([0, 0, 64, 100]), mean=rng.random() < 0.5,
                    grad_state=rng.random() < 0.3, **_draw_mesh(rng, 3000, 16000))
    if kind == "adjoint-streamed":
        return dict(kind="adjoint", engine="plain", real=rng.randint(2, 8), steps=rng.randint(32, 64),
                    tick=rng.choice([8, 16]), ckpt=rng.choice([0, 24]), mean=rng.random() < 0.5,
                    **_draw_mesh(rng, 30000, 72000))
    return dict(kind="readout", prec=32, engine=rng.choice(["resident", "plain"]),
                real=_log_int(rng, 8, 500), steps=rng.randint(16, 64), **_draw_mesh(rng, 3000, 16000))


# ---- inputs -------------------------------------------------------------------
_dir = None


@functools.lru_cache(maxsize=None)
def _mesh_files(key):
    """Writes a mesh once per process; (file base, max |a0|)."""
    global _dir
    if _dir is None:
        _dir = tempfile.mkdtemp(prefix="srs_cases_")
    m = dict(key)
    base = os.path.join(_dir, "_".join(str(v) for _, v in key).replace(".", "p"))
    if m["mesh"] == "tiny":
        rep = srs.write_box_mesh(base, **wl.TINY_DYAD)
    elif m["mesh"] == "config":
        rep = srs.write_box_mesh(base, **wl.CONFIG_DYAD)
    elif m["mesh"] == "config2":
        rep = srs.write_box_mesh(base, **wl.config2_mesh_specs()[m["index"]])
    elif m["mesh"] == "site":
        rep = srs.write_multisite_mesh(base, wl.config4_mesh_spec(h_fine=m["h"]))
    else:
        rad = 0.026 * math.sqrt(m["ryr"])
        rep = srs.write_box_mesh(base, box_x=m["box"], box_y=m["box"], box_z=m["box"],
                                 foot_half_x=rad + 0.05, foot_half_y=rad + 0.05, n_foot_x=m["nf"],
                                 n_foot_y=m["nf"], n_out_x=m["no"], n_out_y=m["no"], n_above_z=m["na"],
                                 ryr_mode=1, ryr_count=m["ryr"], ryr_radius=rad, ryr_pitch=0.030,
                                 n_lcc=max(1, round(m["ryr"] / 7)), lcc_half=rad + 0.05, seed=11,
                                 lcc_seed=21)
    return base, rep["max_a0"]


def _mesh_of(case):
    key = tuple((k, case[k]) for k in ("mesh", "box", "nf", "no", "na", "ryr", "h", "index") if k in case)
    return _mesh_files(key)


@functools.lru_cache(maxsize=None)
def _grid_noflux(base):
    return srs.Grid(srs.default_parameters(), base)


def _grid(case, p):
    """With no-flux boundaries the grid holds nothing of the parameters; with
    Dirichlet faces it holds their boundary sources."""
    base, _ = _mesh_of(case)
    return srs.Grid(p, base) if case.get("noflux") is False else _grid_noflux(base)


def _params(case, seed, max_a0, n_ryr):
    rng = random.Random(seed)
    p = wl.default_spark_params()
    for name in JITTERED:
        p.reals[srs.R[name]] *= math.exp(0.08 * max(-2.0, min(2.0, rng.gauss(0.0, 1.0))))
    p.set(T_STEP=wl.stable_dt(p, max_a0), INIT_RYR=min(24, n_ryr - 1), INIT_RYR_HOLD=10.0)
    if case.get("clamp"):
        p.set(INIT_RYR=-1, INIT_RYR_HOLD=0.0, FLAG_V_CLAMP=1, V_CLAMP=case.get("volt", 0.0), T_CLAMP=200.0)
    if case.get("noflux") is False:
        p.set(FLAG_NO_FLUX_BOUNDARY=0)
    if case["kind"] in ("spark", "batch"):
        dt = p.reals[srs.R["T_STEP"]]
        p.set(T_FINAL=(case["steps"] - 0.5) * dt, OUTPUT_STATES_INTERVAL=case["steps"] * dt / 3.5)
        if case.get("frames"):
            p.set(OUTPUT_GRID_FLAG=1, OUTPUT_GRID_INTERVAL=case["steps"] * dt / (case["frames"] + 0.5))
    return p


def _seeds(seed, n):
    first = random.Random(seed + 1).randrange(1, 1 << 40)
    return [first + r for r in range(n)]


def _problem(case, seed):
    """(grid, parameters, realization seeds) of one simulation."""
    base, a0 = _mesh_of(case)
    p = _params(case, seed, a0, _grid_noflux(base).n_ryr)
    return _grid(case, p), p, _seeds(seed, case["real"])


def _members(case, seed):
    """The members of an uneven batch: four meshes, leak and LCC-triggered.
    The third mesh all but fills clusters of six, so its cluster is named."""
    for k, cluster in enumerate((0, 0, 8, 0)):
        for j, volt in enumerate((-80.0, 0.0)):
            yield (dict(case, kind="batch", mesh="config2", index=k, clamp=True, volt=volt, cluster=cluster),
                   seed * 8 + 2 * k + j)


def _simulation(case, seed):
    g, p, seeds = _problem(case, seed)
    engine = srs.ENGINE_RESIDENT if case.get("engine", "plain") == "resident" else srs.ENGINE_PLAIN
    return srs.Simulation(g, p, case["real"], case.get("prec", 32), engine, seeds=seeds,
                          cluster_size=case.get("cluster", 0))


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "noalloc":
        return _prepare_noalloc(case, seed)
    if kind == "batch":
        sims = [_simulation(dict(c, engine="resident"), s) for c, s in _members(case, seed)]
        st.update(sims=sims, batch=srs.Batch(sims, steps_per_launch=250))
        return st
    sim = st["sim"] = _simulation(case, seed)
    if kind != "step":
        n = sim.linescan_setup(**LINESCAN)
    if kind == "readout":
        sim.explicit_step(case["steps"])
    if kind == "adjoint":
        st["f0"] = sim.linescan()[1]
        st["target"] = _target(case, seed, n)
    return st


def _target(case, seed, n):
    """A measured trace: a slow rise with noise."""
    r = np.random.RandomState(seed % (1 << 31))
    ticks = case["steps"] // case["tick"]
    shape = (ticks, n) if case["mean"] else (case["real"], ticks, n)
    rise = np.linspace(0.0, 1e-3, ticks)[:, None] * np.exp(-np.linspace(-2, 2, n) ** 2)
    return rise + 1e-4 * r.standard_normal(shape)


def _channel_lists(grid):
    N, ch = grid.n_ele, grid.channels()
    per = [[] for _ in range(N)]
    for kind, name in enumerate(("ryr_ele", "ryr_jsr", "lcc_ele")):
        for i, e in enumerate(ch[name]):
            per[e].append((kind, i))
    ptr = np.cumsum([0] + [len(x) for x in per]).astype(np.int32)
    return ptr, np.array([v for x in per for e in x for v in e], np.int32)


def _start_noalloc(case, seed, g, p):
    """Resting grid, the initial RyR open, fresh residuals."""
    r = np.random.RandomState(seed % (1 << 31))
    R = case["real"]
    S = np.tile(g.initial_states(p), (R, 1))
    ryr = np.zeros((R, g.n_ryr), np.int32)
    ryr[:, p.ints[srs.I["INIT_RYR"]]] = 1
    lcc, lccv = np.ones((R, g.n_lcc), np.int32), np.full((R, g.n_lcc), 2, np.int32)
    return S, ryr, lcc, lccv, np.log(r.uniform(1e-6, 1.0, (R, g.n_ryr + g.n_lcc)))


def _prepare_noalloc(case, seed):
    g, p, seeds = _problem(case, seed)
    N, R = g.n_ele, case["real"]
    aij, nij, br = g.operator()
    el, ch, reals = g.elements(), g.channels(), np.array(p.reals[:], np.float64)
    ptr, lst = _channel_lists(g)
    flags = (el["domain"] == 1) + 2 * (el["tropc"] != 0) + 4 * (np.diff(ptr) > 0)
    cap = el["TT"] / (el["V0"] * 1e-15)
    br = br.reshape(6, N)
    T = lambda a, t=None: torch.as_tensor(np.ascontiguousarray(a, dtype=t)).cuda()  # noqa: E731
    bufs = dict(aij=T(aij), nij=T(nij), br4=T(br[[0, 1, 2, 5]]), v0=T(el["V0"]),
                bhi=T(cap * reals[srs.R["B_TOT_SL_HI"]]), blo=T(cap * reals[srs.R["B_TOT_SL_LO"]]),
                flags=T(flags, np.int32), chan_ptr=T(ptr), chan_list=T(lst), ryr_ele=T(ch["ryr_ele"]),
                ryr_jsr=T(ch["ryr_jsr"]), ryr_nb=T(ch["ryr_nb"]), lcc_ele=T(ch["lcc_ele"]))
    start = [T(a) for a in _start_noalloc(case, seed, g, p)]
    S = [torch.zeros_like(start[0]) for _ in range(2)]
    live = [torch.zeros_like(a) for a in start[1:]]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sd = np.array(seeds, np.uint64)
    steps = []
    for k in range(2):
        d = srs.NoallocStep()
        d.n_ele, d.n_realizations, d.n_ryr, d.n_lcc = N, R, g.n_ryr, g.n_lcc
        for name, t in bufs.items():
            setattr(d, name, t.data_ptr())
        d.states_in, d.states_out = S[k].data_ptr(), S[1 - k].data_ptr()
        d.ryr_states, d.lcc_states, d.lccv_states, d.residuals = [t.data_ptr() for t in live]
        d.status = status.data_ptr()
        d.reals = reals.ctypes.data_as(ctypes.c_void_p).value
        d.seeds = sd.ctypes.data_as(ctypes.c_void_p).value
        d.v_m, d.ca_nsr = reals[srs.R["DEFAULT_VM"]], reals[srs.R["DEFAULT_CA_NSR"]]
        d.stream = torch.cuda.current_stream().cuda_stream
        steps.append(d)
    return dict(case=case, steps=steps, S=S, live=live, start=start, status=status,
                keep=(bufs, reals, sd))


# ---- one pass -------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        state["S"][0].copy_(state["start"][0])
        for a, b in zip(state["live"], state["start"][1:]):
            a.copy_(b)
        for k in range(case["steps"]):
            d = state["steps"][k % 2]
            d.step = k
            srs.explicit_step_fp64_noalloc(d)
        return [state["S"][case["steps"] % 2], *state["live"], state["status"]]
    if kind == "batch":
        for s in state["sims"]:
            s.reset()
        res = state["batch"].run_simulation(row_capacity=16)
        return [[np.stack(rows), t_end, n_steps] for rows, t_end, n_steps in res] + \
            [s.total_ca() for s in state["sims"]]
    sim = state["sim"]
    if kind == "readout":
        F, rest = sim.linescan()
        return [F, rest, sim.total_ca()] + [_state(sim, r) for r in (0, case["real"] // 2)]
    sim.reset()
    if kind == "step":
        for _ in range(case["calls"]):
            sim.explicit_step(case["steps"])
        return _state(sim, 0)
    if kind == "adjoint":
        loss, grad, gs = sim.adjoint(case["steps"], case["tick"], state["f0"], state["target"],
                                     checkpoint_every=case["ckpt"], grad_state=bool(case.get("grad_state")),
                                     flags=srs.ADJ_MEAN_TRACE if case["mean"] else 0)
        # the adjoint computes in FP32: its results at that precision
        out = [loss.astype(np.float32), grad.astype(np.float32)]
        return out if gs is None else out + [gs.astype(np.float32)]
    frames = []
    if case.get("frames"):
        res = sim.run_simulation(row_capacity=16, grid_callback=lambda n, t, done: frames.append(sim.linescan()[0]))
    else:
        res = sim.run_simulation(row_capacity=16)
    rows, t_end, n_steps = res
    out = [np.stack(rows), t_end, n_steps, sim.linescan()[0], sim.total_ca(), _state(sim, case["real"] - 1)]
    return out + [np.stack(frames)] if frames else out


def _state(sim, r):
    s = sim.get_state(r)
    return [s["states"], s["ryr"], s["lcc"], s["lccv"], s["residuals"]]


# ---- what a pass cannot do without ------------------------------------------------
def _element_steps(case):
    """[(elements, realizations, steps)]"""
    if case["kind"] == "batch":
        return [(_grid_noflux(_mesh_of(c)[0]).n_ele, case["real"], case["steps"]) for c, _ in _members(case, 0)]
    n = case["steps"] * case.get("calls", 1)
    return [(_grid_noflux(_mesh_of(case)[0]).n_ele, case["real"], 1 if case["kind"] == "readout" else n)]


def work(case):
    """Per element-step of a realization: the state read and written once
    (48 B in FP32, 96 B in FP64) and the geometry once for all realizations
    (44 / 68 B); the reverse step of the adjoint reads the recorded state,
    its rate and lambda and writes lambda (96 B)."""
    fp64 = case.get("prec") == 64 or case["kind"] == "noalloc"
    b = f = 0.0
    for N, R, n in _element_steps(case):
        es = float(N) * R * n
        if case["kind"] == "readout":
            b += es * 24
            f += es * 30
            continue
        b += es * ((96 + 68 / R) if fp64 else (48 + 44 / R))
        f += es * 150
        if case["kind"] == "adjoint":
            b += es * (96 + 44 / R)
            f += es * 300
    return dict(bytes=b, flops=f)


# ---- the same path in 64 bits -----------------------------------------------------
# Arrays are [element][realization]; species 0..5 = Ca, ATP, CMDN, TRPN, CSQN, dye.
THETA = ("D_CA", "D_DYE", "K_ON_CMDN", "K_OFF_CMDN", "K_ON_TRPN", "K_OFF_TRPN", "K_ON_CSQN",
         "K_OFF_CSQN", "K_ON_DYE", "K_OFF_DYE", "V_RYR", "A_P", "B_TOT_SL_HI", "K_D_SL_HI", "D_ATP",
         "D_CMDN", "K_ON_ATP", "K_OFF_ATP")


def _philox(c, key):
    """Philox4x32-10 (Salmon et al., SC'11) on uint64 columns."""
    c = [np.asarray(v, np.uint64) for v in c]
    k = [np.asarray(key & np.uint64(0xffffffff)), np.asarray(key >> np.uint64(32))]
    m32 = np.uint64(0xffffffff)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k[0], p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ k[1], p0 & m32]
        k = [(k[0] + np.uint64(0x9E3779B9)) & m32, (k[1] + np.uint64(0xBB67AE85)) & m32]
    return c


def _uniforms(seeds, channel, step, stream):
    z = np.zeros_like(seeds)
    o = _philox([z + np.uint64(step & 0xffffffff), z + np.uint64(step >> 32), channel.astype(np.uint64),
                 z + np.uint64(stream)], seeds)
    u = lambda a, b: (((a << np.uint64(20)) | (b >> np.uint64(12))).astype(np.float64) + 0.5) * 2.0 ** -52  # noqa: E731
    return u(o[0], o[1]), u(o[2], o[3])


class _Exact:
    def __init__(self, g, p, seeds):
        D = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a)).to("cuda", t)  # noqa: E731
        self.p = {k: p.reals[i] for k, i in srs.R.items()}
        self.i = {k: p.ints[i] for k, i in srs.I.items()}
        self.N, self.R, self.base = g.n_ele, len(seeds), g.mesh_base
        aij, nij, br = g.operator()
        self.a, self.nb = D(aij.reshape(-1, 5).T.copy()), D(nij.reshape(-1, 4).T.copy(), torch.int64)
        br = br.reshape(6, self.N)
        self.br = D(br)[:, :, None] if br.any() else [0.0] * 6
        el, ch = g.elements(), g.channels()
        self.order, self.dom = el["order"], el["domain"]
        self.V0, self.cap = D(el["V0"])[:, None], D(el["TT"] / (el["V0"] * 1e-15))[:, None]
        self.jsr, self.trop = D(el["domain"] == 1)[:, None], D(el["tropc"] != 0)[:, None]
        self.cl, self.js, self.le = (D(ch[k], torch.int64) for k in ("ryr_ele", "ryr_jsr", "lcc_ele"))
        self.NR, self.NL = g.n_ryr, g.n_lcc
        self.seeds = np.array(seeds, np.uint64)
        q = self.p
        rest = lambda b, s: q["C_0_CA"] * q[b] / (q["K_OFF_" + s] / q["K_ON_" + s] + q["C_0_CA"])  # noqa: E731
        cyt = 1.0 - self.jsr
        kd = q["K_OFF_CSQN"] / q["K_ON_CSQN"]
        self.rest = [q["C_0_CA"] * cyt + q["C_0_CA_JSR"] * self.jsr, rest("B_TOT_ATP", "ATP") * cyt,
                     rest("B_TOT_CMDN", "CMDN") * cyt, rest("B_TOT_TRPN", "TRPN") * cyt * self.trop,
                     q["C_0_CA_JSR"] * q["B_T_JSR"] / (kd + q["C_0_CA_JSR"]) * self.jsr,
                     rest("B_TOT_DYE", "DYE") * cyt]
        self.S = [v.expand(self.N, self.R).clone() for v in self.rest]
        self.ryr = torch.zeros(self.NR, self.R, dtype=torch.int64, device="cuda")
        self.lcc, self.lccv = (torch.full((self.NL, self.R), v, dtype=torch.int64, device="cuda") for v in (1, 2))
        if self.i["INIT_RYR"] >= 0:
            self.ryr[self.i["INIT_RYR"]] = 1
        nch = self.NR + self.NL
        sd = np.repeat(self.seeds, nch)
        u, _ = _uniforms(sd, np.tile(np.arange(nch), self.R), 0xffffffffffffffff, 2)
        self.res = D(np.log(u).reshape(self.R, nch).T)
        self.volt = q["V_CLAMP"] if self.i["FLAG_V_CLAMP"] else q["DEFAULT_VM"]
        self.step = 0

    def theta(self):
        return {k: torch.full((1, self.R), self.p[k], dtype=torch.float64, device="cuda") for k in THETA}

    def _lcc(self, V):
        V = 1e-6 if abs(V) < 1e-6 else V
        f = 96.5 / (310 * 8.314)
        E = math.exp(2 * V * f)
        return -(9.13e-13 * 1e12 * 1e-3) * V * 2 * f / (E - 1), E, 0.34 * self.p["CA_0"]

    def advance(self, S, ryr, lcc_open, th):
        """ExplicitStep of S under parameters th; the new state."""
        q = self.p
        ca, atp, cmdn, trpn, csqn, dye = S
        cyt = 1.0 - self.jsr

        def diffusion(s, c, d):
            acc = self.a[0][:, None] * c
            for k in range(4):
                acc = acc + self.a[k + 1][:, None] * c[self.nb[k]]
            return d * acc + self.br[s]
        r = [diffusion(0, ca, th["D_CA"]), diffusion(1, atp, th["D_ATP"]), diffusion(2, cmdn, th["D_CMDN"]),
             None, None, diffusion(5, dye, th["D_DYE"])]
        net = lambda b, tot, n: th["K_ON_" + n] * (tot - b) * ca - th["K_OFF_" + n] * b  # noqa: E731
        r[3] = net(trpn, q["B_TOT_TRPN"], "TRPN") * self.trop * cyt
        r[4] = net(csqn, q["B_T_JSR"], "CSQN") * self.jsr
        ki = (ca / q["K_D_i"]) ** 2
        ks = (q["DEFAULT_CA_NSR"] / q["K_D_SR"]) ** 2
        v = (ki * ki * 3.24873e12 + ki * (9.17846e6 - 11478.2 * ks) - 0.329904 * ks) / \
            (0.104217 + 17.923 * ks + ki * (1.75583e6 + ks * 7.61673e6) + ki * ki * (6.08463e11 + ks * 4.50544e11))
        rd, ra, rm = (net(b, q["B_TOT_" + n], n) * cyt for b, n in ((dye, "DYE"), (atp, "ATP"), (cmdn, "CMDN")))
        rc = r[0] - r[3] - r[4] - 2e-3 * v * th["A_P"] * self.trop * cyt - rd - ra - rm
        rc = rc + (q["DEFAULT_CA_NSR"] - ca) * q["V_REFILL"] * self.jsr
        J = ryr.to(torch.float64) * th["V_RYR"] * (ca[self.js] - ca[self.cl]) * q["V_CELL"]
        rc = rc.index_add(0, self.cl, J / self.V0[self.cl]).index_add(0, self.js, -J / self.V0[self.js])
        if self.NL:
            A, E, B = self._lcc(self.volt)
            rc = rc.index_add(0, self.le, lcc_open * A * (ca[self.le] * E - B) / self.V0[self.le])
        khi = th["K_D_SL_HI"]
        rc = rc / (1 + self.cap * th["B_TOT_SL_HI"] * khi / (khi + ca) ** 2)
        dt = q["T_STEP"]
        return [ca + dt * rc, atp + dt * (r[1] + ra), cmdn + dt * (r[2] + rm), trpn + dt * r[3],
                csqn + dt * r[4], dye + dt * (r[5] + rd)]

    def lcc_open(self):
        return (((self.lcc == 6) | (self.lcc == 12)) & (self.lccv == 2)).to(torch.float64)

    def gate(self):
        q, V, dt = self.p, self.volt, self.p["T_STEP"]
        ca = self.S[0]
        phi = 1.0 - (1000.0 / q["RYR_PHI_B"]) ** q["RYR_PHI_M"] + (ca[self.js] / q["RYR_PHI_B"]) ** q["RYR_PHI_M"]
        up = phi * q["RYR_K_PLUS"] * ca[self.cl] ** q["RYR_ETA"]
        rate = torch.where(self.ryr > 0, torch.full_like(up, q["RYR_K_MINUS"]), up)
        rates = [rate]
        if self.NL:
            al = 4.0 * 1.2 * 0.416 * math.exp(0.012 * (V - 35.0))
            be = 4.0 * 0.45 * 0.049 * math.exp(-0.05 * (V - 35.0))
            gm = 0.83 * 1.9 * 1.3 * 0.31 * 7.5 * 0.09233 / 1000.0 * ca[self.le]
            om, bL, aL = 0.83 * 2.0 * 1.3 * 0.01, 1.9356, 2.0
            W = torch.zeros(13, 3, self.NL, self.R, dtype=torch.float64, device="cuda")
            to = torch.zeros(13, 3, dtype=torch.int64, device="cuda")
            for s in range(1, 6):  # mode normal: back, forward, to mode Ca
                out = [(s - 1, (s - 1) * be), (s + 1, (5 - s) * al if s < 5 else 0.85), (s + 6, aL ** (s - 1) * gm)]
                for k, (t, w) in enumerate(out[1:] if s == 1 else out):
                    W[s, k], to[s, k] = w, t
                out = [(s + 5, (s - 1) * be / bL), (s, om / bL ** (s - 1)), (s + 7, (5 - s) * al * aL if s < 5 else 0.005)]
                for k, (t, w) in enumerate(out[1:] if s == 1 else out):
                    W[s + 6, k], to[s + 6, k] = w, t
            W[6, 0], to[6, 0] = 2.0, 5
            W[12, 0], to[12, 0] = 7.0, 11
            w = torch.gather(W.permute(1, 2, 3, 0), 3, self.lcc[None, :, :, None].expand(3, -1, -1, 1))[..., 0]
            yi = 0.4 / (1.0 + math.exp((V + 12.5) / 5.0)) + 0.6
            tau = 60.0 + 340.0 / (1.0 + math.exp((V + 30.0) / 12.0))
            wv = torch.where(self.lccv == 1, yi / tau, (1.0 - yi) / tau)
            rates.append(w.sum(0) + wv)
        self.res = self.res + torch.cat(rates) * dt
        hit = (self.res > 0).nonzero().cpu().numpy()
        for c, r in hit:
            u0, u1 = _uniforms(self.seeds[r:r + 1], np.array([c]), self.step, 0)
            self.res[c, r] = math.log(u0[0])
            if c < self.NR:
                self.ryr[c, r] = 1 - self.ryr[c, r]
                continue
            k = c - self.NR
            cum = torch.cumsum(w[:, k, r], 0).cpu().numpy()
            pick, s = u1[0] * float(rates[1][k, r]), int(self.lcc[k, r])
            j = int(np.searchsorted(cum, pick, side="right"))
            if j < 3:
                self.lcc[k, r] = to[s, j]
            else:
                self.lccv[k, r] = 3 - self.lccv[k, r]

    def one(self, th):
        self.S = self.advance(self.S, self.ryr, self.lcc_open(), th)
        if not self.i["FLAG_NO_GATING"]:
            self.gate()
        self.step += 1

    def weights(self):
        """PSF-weighted volumes of the line scan [samples][elements]."""
        nodes = np.loadtxt(self.base + ".node", skiprows=1, usecols=(1, 2, 3), comments="#")
        ele = np.loadtxt(self.base + ".ele", skiprows=1, usecols=(0, 1, 2, 3, 4), dtype=np.int64, comments="#")
        first = 0 if int(open(self.base + ".node").read(4000).split("\n")[1].split()[0]) == 0 else 1
        P = nodes[ele[:, 1:5] - first][self.order]
        cen = P.mean(1)
        vol = np.abs(np.einsum("ij,ij->i", P[:, 0] - P[:, 3], np.cross(P[:, 1] - P[:, 3], P[:, 2] - P[:, 3]))) / 6.0
        L = LINESCAN
        n = int((L["x_max"] - L["x_min"]) / L["res"])
        at = np.stack([L["x_min"] + L["res"] * np.arange(n), np.full(n, L["offset1"]), np.full(n, L["offset2"])], 1)
        var = np.array([L["var_x"], L["var_y"], L["var_z"]])
        W = np.zeros((n, len(vol)))
        for i in range(n):
            d = cen - at[i]
            near = (d * d).sum(1) < L["r_thresh"]
            W[i, near] = (vol * np.exp(-0.5 * (d * d / var).sum(1)))[near]
        return torch.as_tensor(W / ((2 * 3.14159) ** 1.5 * math.sqrt(var.prod()))).cuda()

    def row(self, t):
        q, ca = self.p, self.S[0]
        cur = 96485 * 2 * 1e-6
        ir = (self.ryr * q["V_RYR"] * (ca[self.js] - ca[self.cl]) * q["V_CELL"]).sum(0) * cur
        cols = [torch.full_like(ir, t), ir, self.ryr.sum(0)]
        if self.NL:
            A, E, B = self._lcc(self.volt)
            o = self.lcc_open()
            cols += [o.sum(0), (o * A * (ca[self.le] * E - B)).sum(0) * cur]
        else:
            cols += [torch.zeros_like(ir)] * 2
        cols += [ca[self.js].mean(0), ca[self.cl].mean(0)]
        return torch.stack([c.to(torch.float64) for c in cols], 1).cpu().numpy()

    def total(self):
        q, c = self.p, self.S[0]
        sl = self.cap * (q["B_TOT_SL_HI"] * c / (q["K_D_SL_HI"] + c) + q["B_TOT_SL_LO"] * c / (q["K_D_SL_LO"] + c))
        t = self.V0 * (sum(self.S) + sl)
        return torch.stack([(t * (1.0 - self.jsr)).sum(0), (t * self.jsr).sum(0)], 1).cpu().numpy()

    def state(self, r):
        order = (0, 1, 2, 3, 4, 5)
        return [np.concatenate([self.S[s][:, r].cpu().numpy() for s in order]), self.ryr[:, r].cpu().numpy(),
                self.lcc[:, r].cpu().numpy(), self.lccv[:, r].cpu().numpy(), self.res[:, r].cpu().numpy()]

    def simulate(self, on_frame=None):
        """RunSimulation: rows [R][n][7], t_end, steps."""
        q, th, dt = self.p, self.theta(), self.p["T_STEP"]
        rows, t, last = [self.row(0.0)], 0.0, 0.0
        due = lambda I: math.floor(t / I) > math.floor((t - last) / I)  # noqa: E731
        hold = self.i["INIT_RYR"]
        while t <= q["T_FINAL"]:
            if hold >= 0 and t < q["INIT_RYR_HOLD"]:
                self.ryr[hold] = 1
            if self.i["OUTPUT_GRID_FLAG"] and due(q["OUTPUT_GRID_INTERVAL"]):
                on_frame()
            if due(q["OUTPUT_STATES_INTERVAL"]):
                rows.append(self.row(t))
            self.one(th)
            t, last = t + dt, dt
        rows.append(self.row(t))
        return [np.stack(rows, 1), np.full(self.R, t), None]


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "adjoint":
            return _exact_adjoint(case, seed)
        if case["kind"] == "batch":
            ends = []
            for c, s in _members(case, seed):
                e = _Exact(*_problem(c, s))
                ends.append((e.simulate(), e.total()))
            return [x for x, _ in ends] + [x for _, x in ends]
        e = _Exact(*_problem(case, seed))
        if case["kind"] == "noalloc":
            S, ryr, lcc, lccv, res = _start_noalloc(case, seed, *_problem(case, seed)[:2])
            e.S = [torch.as_tensor(v.T.copy()).cuda() for v in S.reshape(e.R, 6, e.N).transpose(1, 0, 2)]
            e.res = torch.as_tensor(res.T.copy()).cuda()
        th = e.theta()
        if case["kind"] in ("step", "noalloc", "readout"):
            for _ in range(case["steps"] * case.get("calls", 1)):
                e.one(th)
        if case["kind"] == "step":
            return _floats(e.state(0))
        if case["kind"] == "noalloc":
            st = [e.state(r) for r in range(e.R)]
            return [np.stack([s[0] for s in st]), None, None, None, np.stack([s[4] for s in st]), None]
        W = e.weights()
        scan = lambda: (W @ e.S[5]).T.contiguous().cpu().numpy()  # noqa: E731
        if case["kind"] == "readout":
            rest = (W @ e.rest[5])[:, 0].cpu().numpy()
            return [scan(), rest, e.total()] + [_floats(e.state(r)) for r in (0, case["real"] // 2)]
        frames = []
        out = e.simulate(lambda: frames.append(scan()))
        out += [scan(), e.total(), _floats(e.state(case["real"] - 1))]
        return out + [np.stack(frames)] if frames else out


def _floats(state):
    return [state[0], None, None, None, state[4]]


def _exact_adjoint(case, seed):
    e = _Exact(*_problem(case, seed))
    W, tick, n = e.weights(), case["tick"], case["steps"]
    f0 = (W @ e.rest[5])[:, 0]
    target = torch.as_tensor(_target(case, seed, len(f0))).cuda()
    th, past = e.theta(), []
    for _ in range(n):
        past.append((e.S, e.ryr.clone(), e.lcc_open()))
        e.one(th)
    past.append((e.S, None, None))
    lam = [torch.zeros_like(v) for v in e.S]
    grad = torch.zeros(len(THETA), e.R, dtype=torch.float64, device="cuda")
    loss = torch.zeros(e.R, dtype=torch.float64, device="cuda")
    for t in range(n, 0, -1):
        if t % tick == 0:
            F = W @ past[t][0][5]
            k = t // tick - 1
            if case["mean"]:
                err = F.mean(1) / f0 - 1 - target[k]
                loss[0] += 0.5 * (err * err).sum()
                lam[5] += (W.T @ (err / f0))[:, None] / e.R
            else:
                err = F / f0[:, None] - 1 - target[:, k].T
                loss += 0.5 * (err * err).sum(0)
                lam[5] += W.T @ (err / f0[:, None])
        S, ryr, lo = past[t - 1]
        past[t] = None
        with torch.enable_grad():
            x = [v.detach().requires_grad_() for v in S]
            q = {k: v.detach().requires_grad_() for k, v in th.items()}
            y = e.advance(x, ryr, lo, q)
            got = torch.autograd.grad(y, x + [q[k] for k in THETA], lam)
        lam = list(got[:6])
        grad += torch.stack([v[0] for v in got[6:]])
    out = [loss.cpu().numpy(), grad.T.contiguous().cpu().numpy()]
    if case.get("grad_state"):
        cyt = 1.0 - e.jsr
        keep = [1.0, 1.0, 1.0, e.trop * cyt, e.jsr, 1.0]
        out.append(torch.stack([v * m for v, m in zip(lam, keep)]).permute(2, 0, 1).contiguous().cpu().numpy())
    return out
