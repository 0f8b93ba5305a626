"""The work that users of this package have it do, as measurable cases.

Five ways of using the library, each through its public entry points:

  solve    a whole small simulation: upload an initial field, RK steps, download
           (parameter studies, the driver's substeps between two snapshots)
  march    a large simulation that stays on the device: RK steps, then the
           state read in place through ``device_state`` (in-situ analysis)
  stream   fields that arrive and leave on the host: upload, one RK step and
           download of each, pipelined (``set_state_async``/``step_state_async``)
  batch    many independent FP32 problems of uneven size advanced together
  serve    solve requests admitted to a running server, results fetched
  rhs      one right-hand side in the caller's own device buffers

Orders, meshes and physics are those of ``3ddg_gb300/workloads.py``, the tests
and ``bench.py``, with odd and ragged meshes beside the round ones.
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

WATER = dict(C0=1.5, RHO0=1000.0, B_OVER_A=5.0, DIFF_CONST=4.3e-6)


def _single(name, kind, precision, order, ne, steps, blocks=(1, 1, 1), width=0.5, periodic=(0, 0, 0), sponge=2,
            source=False, nonlinear=True, diffusion=True):
    c = dict(kind=kind, precision=precision, order=order, ex=ne[0], ey=ne[1], ez=ne[2], bx=blocks[0], by=blocks[1],
             bz=blocks[2], width=width, px=periodic[0], py=periodic[1], pz=periodic[2], sponge=sponge,
             source=source, nonlinear=nonlinear, diffusion=diffusion, steps=steps)
    if name:
        c["name"] = name
    return c


def _many(name, kind, problems, least, most, steps):
    c = dict(kind=kind, problems=problems, least=least, most=most, steps=steps)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's own problem size (8^3 elements, N = 3), FP64: the
        # substeps between two snapshots; latency and launches count
        _single("solve_fp64_small", "solve", 64, 3, (8, 8, 8), 20, width=1.25),
        # the same in the FP32 form
        _single("solve_fp32_small", "solve", 32, 3, (8, 8, 8), 20, width=1.25),
        # a small ragged periodic box at a high order (the tests' periodic cases)
        _single("solve_fp64_ragged", "solve", 64, 5, (7, 5, 6), 10, periodic=(1, 0, 1), sponge=0),
        # the headline simulation: 64^3 elements at N = 4 in 2x2x2 blocks, FP64
        _single("march_fp64_large", "march", 64, 4, (32, 32, 32), 3, blocks=(2, 2, 2), sponge=3, source=True),
        # a mid-size FP64 run with a ragged mesh at the commonest order
        _single("march_fp64_n3", "march", 64, 3, (43, 37, 40), 5),
        # lossless linear propagation at a high order: no diffusion, no sponge
        _single("march_fp64_lossless", "march", 64, 6, (22, 19, 21), 3, periodic=(0, 1, 0), sponge=0,
                nonlinear=False, diffusion=False),
        # the headline mesh in the FP32 form
        _single("march_fp32_large", "march", 32, 4, (32, 32, 32), 8, blocks=(2, 2, 2), sponge=3, source=True),
        # an ordinary FP32 run that leaves part of the chip's memory idle
        _single("march_fp32_n3", "march", 32, 3, (25, 23, 24), 20),
        # uneven problems of every batch order (parameter sweep, data generation)
        _many("batch_uneven", "batch", 24, 4, 24, 100),
        # a few small problems together: launches and tails count
        _many("batch_small", "batch", 8, 4, 8, 60),
        # FP64 fields coming from and going back to the host every step
        _single("stream_fp64", "stream", 64, 4, (16, 16, 16), 4, blocks=(2, 2, 2), sponge=3, source=True),
        # solve requests served together, results copied back
        _many("serve_mix", "serve", 10, 4, 12, 60),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "march", "march", "march", "march", "stream", "batch", "serve", "rhs"])
    if kind in ("batch", "serve"):
        least = rng.randint(3, 6)
        problems = rng.randint(3, 24) if kind == "batch" else rng.randint(2, 12)
        most = least + rng.randint(1, 18 if kind == "batch" else 8)
        return _many(None, kind, problems, least, most, rng.randint(10, 70))
    order = rng.randint(1, 7)
    K3 = (order + 1) ** 3
    lo, hi = {"solve": (2e3, 2e5), "march": (1e5, 1.6e7), "stream": (1e5, 4e6), "rhs": (2e3, 9e5)}[kind]
    nodes = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = (nodes / K3) ** (1.0 / 3.0)
    ne = [max(2, round(side * rng.uniform(0.75, 1.3))) for _ in range(3)]
    while kind == "rhs" and ne[0] * ne[1] * ne[2] * ((K3 + 7) // 8 * 8) > 1000000:
        ne[ne.index(max(ne))] -= 1
    blocks = [1, 1, 1]
    if kind != "rhs" and rng.random() < 0.4:
        a = rng.randrange(3)
        blocks[a] = 2
        ne[a] = max(1, ne[a] // 2)
    periodic = [int(rng.random() < 0.25) for _ in range(3)]
    source = not periodic[2] and kind != "rhs" and rng.random() < 0.5
    total = ne[0] * ne[1] * ne[2] * blocks[0] * blocks[1] * blocks[2] * K3
    most = {"solve": 20, "march": 12, "stream": 4, "rhs": 1}[kind]
    steps = max(1, min(most, int(5e7 / total)))
    precision = 64 if kind in ("stream", "rhs") else rng.choice([64, 32])
    return _single(None, kind, precision, order, ne, steps, blocks, rng.choice([0.25, 0.5, 1.25]), periodic,
                   rng.randint(0, 3), source, rng.random() < 0.85, rng.random() < 0.85)


# ---------------------------------------------------------------- inputs
def _dt(order, c0, widths):
    return 0.5 / ((2 * order + 1) * c0 * sum(1.0 / w for w in widths))


def _config(case, seed):
    """Parameters of a single problem, in the parameter file's vocabulary."""
    rng = np.random.Generator(np.random.PCG64(seed))
    nb = [case["bx"], case["by"], case["bz"]]
    ne = [case["ex"], case["ey"], case["ez"]]
    w = case["width"]
    sp = [case["sponge"]] * 6
    for a, k in enumerate("xyz"):
        if case["p" + k]:
            sp[2 * a] = sp[2 * a + 1] = 0
    if case["source"]:
        sp[4] = 0
    cfg = dict(
        ORDER=case["order"], NUM_ELEMENTS=ne, NUM_BLOCKS=nb, ELEMENT_WIDTH=[w] * 3,
        STARTING_CORNER=[-0.5 * ne[0] * nb[0] * w, -0.5 * ne[1] * nb[1] * w, 0.0], EVALUATE_ADVECTION=1,
        EVALUATE_DIFFUSION=int(case["diffusion"]), EVALUATE_SPONGE=int(max(sp) > 0),
        BC_IS_PERIODIC=[case["px"], case["py"], case["pz"]], BC_SIGMA_MAX=0.5, BC_SPONGE_WIDTH=sp,
        PRECISION=case["precision"], **WATER)
    if not case["nonlinear"]:
        cfg["B_OVER_A"] = 0.0
    if case["source"]:
        cfg.update(SRC_FACE=4, SRC_AMPLITUDE=2.0, SRC_FREQUENCY=1.0, SRC_CYCLES=5.0,
                   SRC_PHASE=2.0 * math.pi * 0.005 * float(rng.uniform(-1.0, 1.0)), SRC_RADIUS=0.0)
    cfg["DT"] = _dt(case["order"], cfg["C0"], cfg["ELEMENT_WIDTH"])
    return cfg


def _configs(case, seed):
    """The problems of a batch or of a request stream: uneven meshes and
    orders, each with its own medium, tone burst, sponges and step count."""
    rng = np.random.Generator(np.random.PCG64(seed))
    # mesh sizes and orders go with the case, so that every seed is the same work
    shape = np.random.Generator(np.random.PCG64(1000003 * case["problems"] + 1009 * case["least"] + case["most"]))
    out = []
    for _ in range(case["problems"]):
        ne = [int(v) for v in shape.integers(case["least"], case["most"] + 1, size=3)]
        order = int(shape.integers(2, 6))
        steps = case["steps"] if case["kind"] == "batch" else int(shape.integers(case["steps"] // 2, case["steps"] + 1))
        c0 = float(rng.uniform(1.45, 1.60))
        sponge = int(rng.integers(2, 5))
        cfg = dict(
            ORDER=order, NUM_ELEMENTS=ne, NUM_BLOCKS=[1, 1, 1], ELEMENT_WIDTH=[0.25] * 3,
            STARTING_CORNER=[-0.125 * ne[0], -0.125 * ne[1], 0.0], EVALUATE_ADVECTION=1, EVALUATE_DIFFUSION=1,
            EVALUATE_SPONGE=1, BC_IS_PERIODIC=[0, 0, 0], BC_SIGMA_MAX=0.5,
            BC_SPONGE_WIDTH=[sponge, sponge, sponge, sponge, 0, sponge], SRC_FACE=4,
            SRC_AMPLITUDE=float(np.exp(rng.uniform(np.log(0.1), np.log(5.0)))),
            SRC_FREQUENCY=float(rng.uniform(0.5, 2.0)), SRC_CYCLES=5.0, SRC_PHASE=0.0, SRC_RADIUS=0.0, PRECISION=32,
            C0=c0, RHO0=WATER["RHO0"], B_OVER_A=WATER["B_OVER_A"], DIFF_CONST=WATER["DIFF_CONST"])
        cfg["DT"] = _dt(order, c0, cfg["ELEMENT_WIDTH"])
        # a batch steps as far as its caller asks; a request carries its count
        cfg["STEPS"] = steps if case["kind"] == "serve" else 1 << 30
        out.append(cfg)
    return out


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gll(K):
    """Gauss-Lobatto-Legendre points on [0, 1]."""
    leg = np.polynomial.legendre
    inner = np.real(leg.legroots(leg.legder([0.0] * (K - 1) + [1.0]))) if K > 2 else np.zeros(0)
    return (np.concatenate([[-1.0], np.sort(inner), [1.0]]) + 1.0) / 2.0


def _wave(cfg, seed, count):
    """``count`` wavefields in the download layout, [count][4][X][Y][Z]: sums
    of acoustic plane waves of 0.5 MPa in random directions, wavelengths of 3
    to 12 elements (whole numbers of them along periodic axes)."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    K = cfg["ORDER"] + 1
    E = [n * b for n, b in zip(cfg["NUM_ELEMENTS"], cfg["NUM_BLOCKS"])]
    w = cfg["ELEMENT_WIDTH"]
    z = _gll(K)
    dev = _device()
    x = [torch.tensor((np.arange(E[a])[:, None] + z[None, :]).reshape(-1) * w[a], dtype=torch.float64, device=dev)
         for a in range(3)]
    out = torch.zeros([count, 4] + [len(v) for v in x], dtype=torch.float64, device=dev)
    c0, r0 = cfg["C0"], cfg["RHO0"]
    for i in range(count):
        for _ in range(3):
            d = rng.normal(size=3)
            d /= np.linalg.norm(d)
            k = 2.0 * math.pi / (w[0] * rng.uniform(3.0, 12.0)) * d
            for a in range(3):
                if cfg["BC_IS_PERIODIC"][a]:
                    k[a] = 2.0 * math.pi / (E[a] * w[a]) * round(k[a] * E[a] * w[a] / (2.0 * math.pi))
            d = k / max(float(np.linalg.norm(k)), 1e-12)
            ph = (k[0] * x[0])[:, None, None] + (k[1] * x[1])[None, :, None] + (k[2] * x[2])[None, None, :]
            p = 0.5 * torch.cos(ph + float(rng.uniform(0, 2 * math.pi)))
            out[i, 0] += p / c0 ** 2
            for a in range(3):
                out[i, 1 + a] += float(d[a]) / (r0 * c0) * p
    return out


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _elements(cfg, grid):
    """[4][X][Y][Z] -> [4][elements][K^3] in the library's element order."""
    K, nb, ne = cfg["ORDER"] + 1, cfg["NUM_BLOCKS"], cfg["NUM_ELEMENTS"]
    v = grid.reshape([4] + [n for a in range(3) for n in (nb[a], ne[a], K)])
    return v.permute(0, 1, 4, 7, 2, 5, 8, 3, 6, 9).reshape(4, -1, K ** 3)


def _coords(cfg):
    """Global element coordinates of every element, in the library's order."""
    nb, ne = cfg["NUM_BLOCKS"], cfg["NUM_ELEMENTS"]
    g = np.indices([n * b for n, b in zip(ne, nb)])
    g = g.reshape([3] + [n for a in range(3) for n in (nb[a], ne[a])])
    return g.transpose(0, 1, 3, 5, 2, 4, 6).reshape(3, -1)


def _neighbours(cfg):
    """Face table [elements][6] of the rhs entry point (-1 - slot outside)."""
    E = [n * b for n, b in zip(cfg["NUM_ELEMENTS"], cfg["NUM_BLOCKS"])]
    g = _coords(cfg)
    index = np.empty(E, dtype=np.int64)
    index[g[0], g[1], g[2]] = np.arange(g.shape[1])
    nbr = np.empty((g.shape[1], 6), dtype=np.int32)
    slots = 0
    for a in range(3):
        for side in range(2):
            h = g.copy()
            h[a] += 1 if side else -1
            out = (h[a] < 0) | (h[a] >= E[a])
            h[a] %= E[a]
            code = index[h[0], h[1], h[2]]
            if not cfg["BC_IS_PERIODIC"][a]:
                n = int(out.sum())
                code[out] = -1 - (slots + np.arange(n))
                slots += n
            nbr[:, 2 * a + side] = code
    return nbr


def _sigma(cfg):
    """Sponge damping of every element: falls linearly from the nearest
    sponged face over that face's sponge width."""
    E = [n * b for n, b in zip(cfg["NUM_ELEMENTS"], cfg["NUM_BLOCKS"])]
    g, w, sp = _coords(cfg), cfg["ELEMENT_WIDTH"], cfg["BC_SPONGE_WIDTH"]
    if not cfg["EVALUATE_SPONGE"]:
        return np.zeros(g.shape[1])
    dist = np.full((6, g.shape[1]), 1e9)
    for a in range(3):
        if sp[2 * a]:
            dist[2 * a] = g[a] * w[a]
        if sp[2 * a + 1]:
            dist[2 * a + 1] = (E[a] - g[a] - 1) * w[a]
    edge = np.argmin(dist, axis=0)
    depth = np.array([max(1, sp[f]) * w[f // 2] for f in range(6)])[edge]
    sig = np.maximum(0.0, 1.0 - dist.min(axis=0) / depth) * cfg["BC_SIGMA_MAX"]
    return np.where(np.array(sp)[edge] == 0, 0.0, sig)


class _DeviceArray:
    """A device buffer of the library seen through the array interface; the
    tensors made of it keep it, and so the handle that owns the memory."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=typestr, data=(int(ptr), False),
                                             version=2)


def prepare(case, seed):
    dg = importlib.import_module("3ddg_gb300")
    kind = case["kind"]
    if kind == "batch":
        b = dg.Batch(_configs(case, seed))
        return dict(case=case, batch=b)
    if kind == "serve":
        return dict(case=case, server=dg.Server(8 << 30, keep_results=True), requests=_configs(case, seed))
    cfg = _config(case, seed)
    if kind == "rhs":
        K = case["order"] + 1
        K3, NP = K ** 3, (K ** 3 + 7) // 8 * 8
        el = _elements(cfg, _wave(cfg, seed, 1)[0])
        state = torch.zeros((4, el.shape[1], NP), dtype=torch.float64, device=el.device)
        state[:, :, :K3] = el
        ops = dg.line_operators(case["order"])
        dev = state.device
        return dict(case=case, lib=dg.lib(), params=dg.params_from_dict(cfg), mass=ops["mass"], stiff=ops["stiff"],
                    state=state, nbr=torch.from_numpy(_neighbours(cfg)).to(dev),
                    sigma=torch.from_numpy(_sigma(cfg)).to(dev), rhs=torch.zeros_like(state), K3=K3)
    s = dg.Solver(cfg)
    fields = _wave(cfg, seed, case["steps"] if kind == "stream" else 1)
    host = []
    for f in fields:
        a = _pinned(tuple(f.shape))
        torch.from_numpy(a).copy_(f)
        host.append(a)
    st = dict(case=case, solver=s, dt=cfg["DT"], fields=host)
    if kind == "march":
        s.set_state(host[0][0], host[0][1:])
        del st["fields"]
    else:
        st["out"] = [_pinned(host[0].shape) for _ in host]
    return st


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        s, f, o = state["solver"], state["fields"][0], state["out"][0]
        s.set_state(f[0], f[1:])
        s.step(state["dt"], case["steps"])
        s.state(o[0], o[1:])
        return o
    if kind == "march":
        s = state["solver"]
        s.step(state["dt"], case["steps"])
        base, stride, n = s.device_state()
        size, K3 = case["precision"] // 8, (case["order"] + 1) ** 3
        out = [torch.as_tensor(_DeviceArray(s, p, (n, K3), (stride * size, size), "<f%d" % size), device="cuda")
               for p in base]
        for t in out:
            t.owner = s
        return out
    if kind == "stream":
        s = state["solver"]
        for f, o in zip(state["fields"], state["out"]):
            s.set_state_async(f[0], f[1:])
            s.step_state_async(state["dt"], o[0], o[1:])
        s.synchronize()
        return state["out"]
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        return [v for i in range(case["problems"]) for v in b.state(i)]
    if kind == "serve":
        v = state["server"]
        ids = [v.submit(c) for c in state["requests"]]
        v.run()
        done = [v.result(i, state=True) for i in ids]
        return [r[k] for r in done for k in ("rho", "vel")]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    h = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    rc = state["lib"].dg_eval_rhs_noalloc(
        ctypes.byref(state["params"]), h(state["mass"]), h(state["stiff"]), p(state["state"]), p(state["nbr"]),
        p(state["sigma"]), p(state["rhs"]), state["state"].shape[1],
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError(state["lib"].dg_last_error().decode())
    return state["rhs"][:, :, :state["K3"]]


# ---------------------------------------------------------------- its cost
def _per_step(cfg):
    """(bytes, flops) of one RK step at least: every stage streams its input
    and its output once and, after the first, the step's initial state; line
    sums, face terms and the stage combination by the direct formulas."""
    K = cfg["ORDER"] + 1
    n = K ** 3
    for a in range(3):
        n *= cfg["NUM_ELEMENTS"][a] * cfg["NUM_BLOCKS"][a]
    size = cfg["PRECISION"] // 8
    diff = cfg["EVALUATE_DIFFUSION"]
    stage = 7 + 3 * 2 * 2 * (K + 2) + 6 / K * 21 + 14 + (diff and 3 * 2 * (K + 2) + 3 + 6 / K * 5)
    return (8 + 12 + 12) * size * n, 3.0 * stage * n


def work(case):
    if case["kind"] in ("batch", "serve"):
        b = f = 0.0
        for c in _configs(case, 0):
            sb, sf = _per_step(c)
            n = case["steps"] if case["kind"] == "batch" else c["STEPS"]
            b, f = b + n * sb, f + n * sf
        return {"bytes": b, "flops": f}
    b, f = _per_step(_config(case, 0))
    if case["kind"] == "rhs":
        return {"bytes": b / 4, "flops": f / 3}
    return {"bytes": b * case["steps"], "flops": f * case["steps"]}


# ---------------------------------------------------------------- in 64 bits
class _Plain:
    """The semi-discrete scheme and its SSP-RK3 step in plain 64-bit torch,
    on fields [X elements][Y][Z][K][K][K]."""

    def __init__(self, cfg):
        self.cfg = cfg
        self.K = K = cfg["ORDER"] + 1
        self.E = [n * b for n, b in zip(cfg["NUM_ELEMENTS"], cfg["NUM_BLOCKS"])]
        dev = _device()
        leg = np.polynomial.legendre
        # Lagrange basis on the nodes, M and S by Gauss quadrature on [0, 1]
        z = _gll(K)
        q, wq = leg.leggauss(K + 2)
        q, wq = (q + 1) / 2, wq / 2
        V = np.linalg.inv(leg.legvander(2 * z - 1, K - 1))
        ell = leg.legvander(2 * q - 1, K - 1) @ V
        der = np.stack([leg.legval(2 * q - 1, leg.legder(np.eye(K)[i])) * 2 for i in range(K)], axis=1) @ V
        M = ell.T @ (wq[:, None] * ell)
        S = der.T @ (wq[:, None] * ell)
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        self.D = t(np.linalg.solve(M, S))
        self.L = [t(np.linalg.solve(M, np.eye(K)[:, i])) for i in (0, K - 1)]
        g = _coords(cfg)
        sig = np.zeros(self.E)
        sig[g[0], g[1], g[2]] = _sigma(cfg)
        self.sigma = t(sig)[..., None, None, None]

    def burst(self, t):
        c = self.cfg
        if "SRC_FACE" not in c:
            return 0.0
        T = c["SRC_CYCLES"] / c["SRC_FREQUENCY"]
        if t < 0 or t > T:
            return 0.0
        return c["SRC_AMPLITUDE"] * math.sin(math.pi * t / T) ** 2 * math.sin(
            2 * math.pi * c["SRC_FREQUENCY"] * t + c["SRC_PHASE"])

    def along(self, v, a):
        return torch.movedim(torch.movedim(v, 3 + a, -1) @ self.D.T, -1, 3 + a)

    def others(self, v, a, outside):
        """Values across the two faces of axis a: (left neighbour's last node,
        right neighbour's first node), ``outside`` beyond the domain."""
        lo, hi = v.select(3 + a, 0), v.select(3 + a, self.K - 1)
        left, right = torch.roll(hi, 1, a), torch.roll(lo, -1, a)
        if not self.cfg["BC_IS_PERIODIC"][a]:
            left.select(a, 0).fill_(outside[0])
            right.select(a, self.E[a] - 1).fill_(outside[1])
        return lo, hi, left, right

    def lift(self, g0, gN, a):
        shape = [1] * 6
        shape[3 + a] = self.K
        return self.L[0].view(shape) * g0.unsqueeze(3 + a) + self.L[1].view(shape) * gN.unsqueeze(3 + a)

    def rhs(self, u, t):
        c = self.cfg
        c0, r0, ba, Dc = c["C0"], c["RHO0"], c["B_OVER_A"], c["DIFF_CONST"]
        p = self.burst(t)
        rho = u[0]
        mom = lambda d: c0 * c0 / r0 * (d + ba / (2 * r0) * d * d)  # noqa: E731
        mass = lambda v, d: v * r0 if ba == 0 else v * (d + r0)  # noqa: E731
        out = [torch.zeros_like(rho)]
        for a in range(3):
            w = c["ELEMENT_WIDTH"][a]
            src = [p if c.get("SRC_FACE", -1) == 2 * a + s else 0.0 for s in (0, 1)]
            ro = [v / c0 ** 2 for v in src]
            uo = [src[0] / (r0 * c0), -src[1] / (r0 * c0)]
            fm, fa = mom(rho), mass(u[1 + a], rho)
            m0, mN, ml, mr = self.others(fm, a, [mom(v) for v in ro])
            a0, aN, al, ar = self.others(fa, a, [mass(v, d) for v, d in zip(uo, ro)])
            k = c0 / (2 * r0)
            out.append((self.along(fm, a) + self.lift(0.5 * (ml + m0) + k * (al - a0),
                                                      -(0.5 * (mr + mN) + k * (aN - ar)), a)) / w)
            k = r0 / (2 * c0)
            f = self.along(fa, a) + self.lift(0.5 * (al + a0) + k * (ml - m0),
                                              -(0.5 * (ar + aN) + k * (mN - mr)), a)
            if c["EVALUATE_DIFFUSION"]:
                d0, dN, dl, dr = self.others(rho, a, ro)
                G = (self.along(rho, a) + self.lift(0.5 * (dl + d0), -0.5 * (dr + dN), a)) * (Dc / w)
                q0, qN, ql, qr = self.others(G, a, [0.0, 0.0])
                f = f + self.along(G, a) + self.lift(0.5 * (ql + q0), -0.5 * (qr + qN), a)
            out[0] = out[0] + f / w
        return torch.stack(out) - self.sigma * u

    def step(self, u, t):
        dt = self.cfg["DT"]
        w23, w13 = float(np.float32(2.0 / 3.0)), float(np.float32(1.0 / 3.0))  # the reference's weights
        a = u + dt * self.rhs(u, t)
        a = 0.75 * u + 0.25 * (a + dt * self.rhs(a, t + dt))
        return w13 * u + w23 * a + dt * 2.0 / 3.0 * self.rhs(a, t + 0.5 * dt)

    def split(self, grid):
        v = grid.reshape([4] + [n for a in range(3) for n in (self.E[a], self.K)])
        return v.permute(0, 1, 3, 5, 2, 4, 6).contiguous()

    def grid(self, u):
        return u.permute(0, 1, 4, 2, 5, 3, 6).reshape([4] + [e * self.K for e in self.E])

    def steps(self, u, n, t=0.0):
        for _ in range(n):
            u = self.step(u, t)
            t += self.cfg["DT"]
        return u


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        out = []
        for c in _configs(case, seed):
            s = _Plain(c)
            zero = torch.zeros([4] + s.E + [s.K] * 3, dtype=torch.float64, device=_device())
            n = case["steps"] if kind == "batch" else c["STEPS"]
            g = s.grid(s.steps(zero, n)).cpu()
            out += [g[0], g[1:]]
        return out
    cfg = _config(case, seed)
    s = _Plain(cfg)
    fields = _wave(cfg, seed, case["steps"] if kind == "stream" else 1)
    if kind == "stream":
        out = []
        for i, f in enumerate(fields):
            out.append(s.grid(s.step(s.split(f), i * cfg["DT"])).cpu())
        return out
    if kind == "rhs":
        return _elements(cfg, s.grid(s.rhs(s.split(fields[0]), 0.0)))
    g = s.grid(s.steps(s.split(fields[0]), case["steps"]))
    return g if kind == "solve" else list(_elements(cfg, g))
