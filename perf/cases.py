"""The workloads the solver's speed is measured on, through its public entry points.

A case is a dict of plain values; `kind` names the entry point:

    step      Fluid.update: one SPH step of a scene whose state a program holds on the GPU
    host      Fluid.update_host: upload, step and read back from pinned host memory in one call
    batch     Batch.step: one step of many independent scenes of uneven sizes
    rollout   local.rollout: judged cycles of one SPH step and K - 1 extrapolated steps
    train     Surrogate.sample + forward_backward: one training sample of the message-passing net
    predict   the same sample without the backward pass, and its predictions
    gemm      wc_nn_gemm: one layer of that network on the tensor cores
    surface   Surface.extract: the colour field and marching cubes of a fluid

`exact` restates each of them in 64 bits with plain torch operations (the surface apart: its
triangles follow discrete decisions on an explicitly rounded field).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from watercube_gb300 import _abi as A
from watercube_gb300 import batch as B
from watercube_gb300 import fluid as F
from watercube_gb300 import local as L
from watercube_gb300 import surface as S
from watercube_gb300 import surrogate as M
from watercube_gb300.train_surrogate import DEFAULT_WEIGHTS as MP_WEIGHTS

H16K, DT1M = 0.0457, 2.5e-4  # the dam break's kernel radius at 16,384 particles, its dt at 1,048,576


def listed():
    return [
        # the smallest workload configured: a 16,384-particle dam break, where launches count
        {"name": "step_16k", "kind": "step", "preset": "dam", "n": 16384, "settled": 0.0},
        # the reference application's own scene: 80,000 particles, its equation of state, wall and
        # mouse terms, with the particle ids and neighbour counts a test or an exporter reads
        {"name": "step_80k_reference", "kind": "step", "preset": "reference", "n": 80000, "settled": 0.0},
        # the benchmark's scene at its start: 1,048,576 particles at the rest spacing
        {"name": "step_1m", "kind": "step", "preset": "dam", "n": 1048576, "settled": 0.0},
        # the same scene late in the benchmark's window: a fifth of the particles compressed to
        # 5.7 times the rest density
        {"name": "step_1m_settled", "kind": "step", "preset": "dam", "n": 1048576, "settled": 0.2},
        # a renderer or controller on the host: state in, one step, state out; a ragged count
        {"name": "host_200k", "kind": "host", "preset": "dam", "n": 200003, "settled": 0.0},
        # the batched workload: 512 scenes, log-uniform in 4,096 .. 65,536 particles
        {"name": "batch_512", "kind": "batch", "scenes": 512, "n_min": 4096, "n_max": 65536, "scene_draw": 0},
        # the learned rollout: two cycles of K = 4 at 1,048,576 particles
        {"name": "rollout_1m_network", "kind": "rollout", "n": 1048576, "mode": "network", "ages": 3, "cycles": 2},
        # one training sample of the 8-layer message-passing network (a middling training scene)
        {"name": "train_16k", "kind": "train", "n": 16384},
        # inference on one large scene of the training draw
        {"name": "predict_65k", "kind": "predict", "n": 65536},
        # that network's widest layers: the first edge layer with its gathered node rows, and the
        # weight gradient of an edge layer (split over a ragged number of edges)
        {"name": "gemm_edge", "kind": "gemm", "form": "gather", "rows": 460000, "k": 128},
        {"name": "gemm_wgrad", "kind": "gemm", "form": "wgrad", "rows": 459213, "k": 128},
        # a surface mesh for export of a scene in motion
        {"name": "surface_128", "kind": "surface", "n": 262144, "grid": 128},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "step", "host", "batch", "rollout", "rollout", "train", "predict",
                       "gemm", "gemm", "surface"])
    if kind == "step":
        return {"kind": kind, "preset": rng.choice(["dam", "dam", "reference"]), "n": log(2000, 1048576),
                "settled": rng.choice([0.0, rng.uniform(0.02, 0.2)])}
    if kind == "host":
        return {"kind": kind, "preset": "dam", "n": log(4096, 1048576), "settled": 0.0}
    if kind == "batch":
        return {"kind": kind, "scenes": log(2, 256), "n_min": log(1000, 4096), "n_max": log(8192, 65536),
                "scene_draw": rng.randrange(1 << 16)}
    if kind == "rollout":
        return {"kind": kind, "n": log(16384, 1048576), "mode": rng.choice(["stale", "taylor", "network"]),
                "ages": rng.choice([3, 4, 5]), "cycles": rng.choice([1, 2])}
    if kind == "train":
        return {"kind": kind, "n": log(2048, 16384)}
    if kind == "predict":
        return {"kind": kind, "n": log(2048, 65536)}
    if kind == "gemm":
        form = rng.choice(["layer", "gather", "layernorm", "concat", "wgrad"])
        k = 256 if form == "concat" else rng.choice([16, 32, 128, 384]) if form == "layer" else 128
        return {"kind": kind, "form": form, "rows": log(4000, 460000), "k": k}
    return {"kind": kind, "n": log(8192, 262144), "grid": rng.randrange(33, 129)}


# ---- inputs -----------------------------------------------------------------------------------------


def _params(case):
    if case.get("preset") == "reference":
        p = F.reference_params()
        p.num_particles = case["n"]
        # the reference's scene at n particles: its lattice fills the same part of the box
        p.particle_radius = 0.01 * (80000 / case["n"]) ** (1 / 3)
        p.grid_res = max(1, int(21 * (case["n"] / 80000) ** (1 / 3)))
        p.particle_mass = 0.08 * (80000 / case["n"])
        p.flags |= A.WC_FLAG_TRACK_IDS | A.WC_FLAG_NEIGHBOR_COUNTS
    else:
        p = F.dam_break_params(case["n"])
        if case["kind"] == "rollout":
            p.flags |= A.WC_FLAG_TRACK_IDS
    return F.finalize(p)


def _dt(n):
    return DT1M * (1048576 / n) ** (1 / 3)


def _scene(case, p, seed):
    """A scene in motion: the preset's jittered lattice (part of it settled to a denser one at the
    floor), falling, spreading and stirred."""
    n, h = case["n"], p.kernel_radius
    rng = np.random.default_rng(seed)
    if case.get("preset") == "reference":
        st = F.generate_reference_lattice(p, seed)
    else:
        st = F.generate_dam_break(p, seed)
        low = int(n * case.get("settled", 0.0))
        if low:
            side = max(1, int(0.4 / (0.28 * h)))
            q = np.arange(low)
            base = np.stack([q % side, q // (side * side), (q // side) % side], 1)
            top = (base[-1, 1] + 1) * 0.28 * h
            st["position"][:low] = (base + 0.5) * 0.28 * h + rng.uniform(-0.03, 0.03, (low, 3)) * h
            side = max(1, int(0.4 / (0.5 * h)))
            q = np.arange(n - low)
            up = np.stack([q % side, q // (side * side), (q // side) % side], 1)
            st["position"][low:] = (up + 0.5) * 0.5 * h + rng.uniform(-0.01, 0.01, (n - low, 3)) * h
            st["position"][low:, 1] += top
    x = st["position"]
    st["velocity"] = x * np.float32([0.5, -0.8, 0.3]) + rng.standard_normal((n, 3), dtype=np.float32) * 0.05
    # in the order that the step before left: by the cells the particles come from
    c = ((x - st["velocity"] * np.float32(2 * _dt(n))) / p.bin_size).astype(np.int64).clip(0, p.grid_res - 1)
    st = st[np.argsort((c[:, 2] * p.grid_res + c[:, 1]) * p.grid_res + c[:, 0], kind="stable")]
    return st


class _Device:
    """A buffer of the solver as an array that torch can view; a view keeps its owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 3}


def _view(owner, ptr, shape, typestr="<f4"):
    return torch.as_tensor(_Device(owner, ptr, shape, typestr), device="cuda")


def _pinned(n):
    return torch.zeros(32 * n, dtype=torch.uint8, pin_memory=True).numpy().view(A.PARTICLE_DTYPE)


def _resident(state, handle, st):
    """The handle's state buffers as tensors, the scene to start from beside them on the GPU."""
    b, n = handle.device_buffers(), st.shape[0]
    state["stream"] = torch.cuda.ExternalStream(b.stream)
    state["pos"], state["vel"] = (
        _view(handle, q, (n, 4)) for q in (b.state_pos_density, b.state_vel_pressure))
    both = torch.from_numpy(st.view(np.float32).reshape(n, 8)).cuda()
    state["pos0"], state["vel0"] = both[:, :4].contiguous(), both[:, 4:].contiguous()
    state["out"] = _columns(state["pos"], state["vel"])
    return b


def _columns(pos, vel):
    return {"position": pos[:, :3], "density": pos[:, 3], "velocity": vel[:, :3], "pressure": vel[:, 3]}


def _batch_inputs(case, seed):
    specs = B.batch_specs(case["scenes"], case["n_min"], case["n_max"], case["scene_draw"])
    for k, s in enumerate(specs):
        s.seed = (seed * 1000003 + k) & 0xFFFFFFFF
    params = [B.scene_params(s) for s in specs]
    return params, [B.scene_particles(s, p) for s, p in zip(specs, params)]


def _sample_inputs(case, seed):
    p = _params(case)
    st = _scene(case, p, seed)
    rng = np.random.default_rng(seed + 1)
    n, dt = case["n"], 1e-3 * (16384 / case["n"]) ** (1 / 3)
    acc = np.float32([0, -9.81, 0]) + 6 * np.sin(9 * st["position"][:, [1, 2, 0]] + rng.uniform(0, 6, 3).astype(np.float32))
    acc += rng.standard_normal((n, 3), dtype=np.float32) * 0.3
    hist, target = np.zeros((5, n, 4), np.float32), np.zeros((n, 4), np.float32)
    for k in range(5):
        hist[k, :, :3] = st["velocity"] - acc * np.float32(k * dt) + rng.standard_normal((n, 3), dtype=np.float32) * 0.002
    hist[0, :, :3] = st["velocity"]
    target[:, :3] = acc
    return p, st, hist, target, dt


def _gemm_inputs(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    rows, k, form = case["rows"], case["k"], case["form"]

    def bf(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()

    t = {"a": bf(rows, 128 if form == "concat" else k), "bias": torch.randn(128, generator=g, device="cuda")}
    if form == "wgrad":
        t["b"] = bf(rows, 128, scale=1e-3)
    else:
        t["b"] = bf(128, k, scale=k ** -0.5)
    if form == "concat":
        t["a2"] = bf(rows, 128)
    if form == "gather":  # rows sorted by receiver, 28 of them to a node; senders nearby
        nodes = rows // 28 + 1
        t["recv"] = (torch.arange(rows, device="cuda") // 28).int()
        near = torch.randint(-600, 601, (rows,), generator=g, device="cuda")
        t["send"] = (t["recv"] + near).clamp(0, nodes - 1).int()
        t["add1"], t["add2"] = bf(nodes, 128), bf(nodes, 128)
    if form == "layernorm":
        t["resid"] = bf(rows, 128)
        t["gamma"] = 1 + 0.1 * torch.randn(128, generator=g, device="cuda")
        t["beta"] = 0.1 * torch.randn(128, generator=g, device="cuda")
    return t


def prepare(case, seed):
    kind, state = case["kind"], {"case": case}
    if kind in ("step", "rollout", "host", "surface"):
        p = _params(case)
        st = _scene(case, p, seed)
        f = F.Fluid.create(kind, p).setup(st)
        state["fluid"] = f
        state["time"] = 1 / 60 if case.get("preset") == "reference" else _dt(case["n"])
        if kind == "host":
            state["in"], state["out"] = _pinned(case["n"]), _pinned(case["n"])
            state["in"][:] = st
        elif kind == "surface":
            state["surface"] = S.Surface(case["grid"])
            # where the mesh goes: page-locked, with room for the splashes of a scene in motion
            room = torch.zeros(24 * case["grid"] ** 2, 3, 3, pin_memory=True)
            state["out"] = room.numpy()
        else:
            b = _resident(state, f, st)
            if case.get("preset") == "reference":
                state["out"]["ids"] = _view(f, b.particle_ids, (case["n"],), "<i4")
                state["out"]["neighbours"] = _view(f, b.neighbor_counts, (case["n"],), "<i4")
        if kind == "rollout":
            state["ids"], state["ids0"] = _view(f, b.particle_ids, (case["n"],), "<i4"), torch.arange(case["n"], dtype=torch.int32, device="cuda")
            state["mode"] = {"stale": A.WC_LOCAL_STALE, "taylor": A.WC_LOCAL_TAYLOR, "network": A.WC_LOCAL_NETWORK}[case["mode"]]
            state["net"] = L.load_weights(L.DEFAULT_WEIGHTS.with_name(f"local_k{case['ages'] + 1}.npz"), capacity=1)
    elif kind == "batch":
        params, initial = _batch_inputs(case, seed)
        state["batch"] = B.Batch(params, initial)
        _resident(state, state["batch"], np.concatenate(initial))
    elif kind in ("train", "predict"):
        p, st, state["hist"], state["target"], state["dt"] = _sample_inputs(case, seed)
        state["fluid"] = F.Fluid.create(kind, p).setup(st)
        z = np.load(MP_WEIGHTS)
        state["net"] = M.Surrogate(layers=8)
        state["net"].set_params(z["params"])
    elif kind == "gemm":
        state["t"] = t = _gemm_inputs(case, seed)
        rows, k, form = case["rows"], case["k"], case["form"]
        g = state["desc"] = A.GemmDesc()
        state["err"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        if form == "wgrad":
            # split over the rows as the training step splits it: at least 1,024 rows, 257 parts
            chunk = max(1024, (rows // 256 + 63) // 64 * 64)
            parts = -(-rows // chunk)
            out = torch.zeros(parts, k, 128, device="cuda")
            g.m, g.n, g.k, g.k_chunk = k, 128, rows, chunk
            g.a, g.lda, g.a_transposed = t["a"].data_ptr(), k, 1
            g.b, g.ldb, g.b_rowmajor = t["b"].data_ptr(), 128, 1
            g.c_f32, g.ldc, g.split_stride = out.data_ptr(), 128, k * 128
        else:
            out = torch.zeros(rows, 128, dtype=torch.bfloat16, device="cuda")
            g.m, g.n, g.k, g.k_chunk = rows, 128, k, -(-k // 64) * 64
            g.a, g.lda, g.b, g.ldb = t["a"].data_ptr(), t["a"].shape[1], t["b"].data_ptr(), k
            g.bias, g.relu, g.c_bf16, g.ldc = t["bias"].data_ptr(), int(form != "layernorm"), out.data_ptr(), 128
            if form == "concat":
                g.a2, g.lda2, g.k_split = t["a2"].data_ptr(), 128, 128
            if form == "gather":
                g.add1, g.add1_idx, g.add2, g.add2_idx, g.ld_add = (
                    t["add1"].data_ptr(), t["recv"].data_ptr(), t["add2"].data_ptr(), t["send"].data_ptr(), 128)
            if form == "layernorm":
                g.ln_gamma, g.ln_beta, g.ln_resid = t["gamma"].data_ptr(), t["beta"].data_ptr(), t["resid"].data_ptr()
        state["out"] = out
    torch.cuda.synchronize()
    return state


# ---- one pass --------------------------------------------------------------------------------------------


def _restart(s):
    with torch.cuda.stream(s["stream"]):
        s["pos"].copy_(s["pos0"], non_blocking=True)
        s["vel"].copy_(s["vel0"], non_blocking=True)
        if "ids0" in s:
            s["ids"].copy_(s["ids0"], non_blocking=True)


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "step":
        _restart(s)
        s["fluid"].update(s["time"])
        return s["out"]
    if kind == "batch":
        _restart(s)
        s["batch"].step(1e-3)
        return s["out"]
    if kind == "host":
        s["fluid"].update_host(s["time"], s["in"], s["out"])
        return {k: s["out"][k] for k in ("position", "density", "velocity", "pressure")}
    if kind == "rollout":
        _restart(s)
        ages = s["case"]["ages"]
        stats = L.rollout(s["fluid"], s["time"], (ages + 1) * s["case"]["cycles"], ages=ages, net=s["net"], mode=s["mode"])
        with torch.cuda.stream(s["stream"]):  # trajectories by particle
            ids = s["ids"].long()
            pos, vel = (torch.empty_like(x).index_copy_(0, ids, x) for x in (s["pos"], s["vel"]))
        return dict(_columns(pos, vel), reverted=int(stats["reverted"]))
    if kind == "train":
        s["net"].sample(s["fluid"], s["dt"], s["hist"], s["target"])
        s["net"].zero_grads()
        return {"loss": s["net"].forward_backward(True), "grads": s["net"].grads()}
    if kind == "predict":
        s["net"].sample(s["fluid"], s["dt"], s["hist"])
        s["net"].forward_backward(False)
        return s["net"].predictions()
    if kind == "gemm":
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        A.check(A.lib().wc_nn_gemm(C.byref(s["desc"]), s["err"].data_ptr(), stream), "wc_nn_gemm")
        return s["out"]
    count = s["surface"].extract(s["fluid"])
    if count > len(s["out"]):
        raise RuntimeError(f"{count} triangles, room for {len(s['out'])}")
    A.check(A.lib().wc_surface_get_triangles(s["surface"]._h, A._ptr(s["out"]), count), "wc_surface_get_triangles")
    return {"triangles": count, "mesh": s["out"]}


# ---- what a pass cannot do without ------------------------------------------------------------------------


def _neighbours(case):
    """Mean particles within h of one, itself included."""
    if case.get("preset") == "reference":
        return 4.19 * (4 / 1.75) ** 3
    x = case.get("settled", 0.0)
    return 4.19 * (8 * (1 - x) + x / 0.28 ** 3)


def work(case):
    kind = case["kind"]
    if kind in ("step", "host", "rollout", "surface"):
        n, nb = case["n"], _neighbours(case)
        if kind == "rollout":  # per cycle a step, then ages integrations of 12 operations
            return {"bytes": 64.0 * n, "flops": case["cycles"] * n * (nb * 80.0 + 36.0 * case["ages"])}
        if kind == "surface":  # the field's vertices inside the fluid see 33 particles each
            v = case["grid"] ** 3
            return {"bytes": 32.0 * n + 36.0 * 6 * v ** (2 / 3), "flops": 0.13 * v * 33 * 11.0}
        return {"bytes": 64.0 * n, "flops": n * nb * 45.0}
    if kind == "batch":
        a, b = case["n_min"], case["n_max"]
        n = case["scenes"] * (b - a) / math.log(b / a)
        return {"bytes": 64.0 * n, "flops": n * 33 * 45.0}
    if kind in ("train", "predict"):
        n, e = case["n"], 28.0 * case["n"]
        layer = 2.0 * 128 * 128
        flops = e * (16 * 256 + layer) + n * (32 * 256 + layer) + 8 * (e * 2 * layer + n * 5 * layer) + n * layer * 1.1
        if kind == "train":
            return {"bytes": n * 128.0 + 4.0 * 984208 * 2, "flops": 3 * flops}
        return {"bytes": n * 128.0 + 4.0 * 984208, "flops": flops}
    rows, k, form = case["rows"], case["k"], case["form"]
    if form == "wgrad":
        parts = -(-rows // max(1024, (rows // 256 + 63) // 64 * 64))
        return {"bytes": rows * (k + 128) * 2.0 + parts * k * 128 * 4.0, "flops": 2.0 * rows * k * 128}
    extra = {"layernorm": 256.0, "gather": 8.0 + 512 / 28}.get(form, 0.0)
    return {"bytes": rows * ((k + 128) * 2.0 + extra), "flops": 2.0 * rows * k * 128}


# ---- the same in 64 bits --------------------------------------------------------------------------------


class _Sph64:
    """The SPH step's equations in float64, particles in the order given. `c`: the constants, as
    floats or as one value per particle (a batch, whose scenes lie `off` cells apart)."""

    def __init__(self, c, off=0, cells=None):
        self.c = {k: torch.as_tensor(v, dtype=torch.float64, device="cuda") for k, v in c.items()}
        self.R = torch.as_tensor(c["R"], dtype=torch.int64, device="cuda")
        self.off, self.cells = off, cells or int(c["R"]) ** 3

    def at(self, name, i):
        v = self.c[name]
        return v[i] if v.ndim else v

    def col(self, name):
        v = self.c[name]
        return v[:, None] if v.ndim else v

    def on(self, flag):
        return (self.c["flags"].long() & flag != 0).any().item()

    def pairs(self, x, most=1 << 25):
        """Chunks (i, j) of the ordered pairs with |x_i - x_j| < h, i = j included."""
        R = self.R
        c = torch.minimum((x / self.col("bin")).long().clamp(min=0), (R[:, None] if R.ndim else R) - 1)
        key = self.off + (c[:, 2] * R + c[:, 1]) * R + c[:, 0]
        order = torch.argsort(key)
        start = torch.zeros(self.cells + 1, dtype=torch.int64, device="cuda")
        start[1:] = torch.cumsum(torch.bincount(key, minlength=self.cells), 0)
        lo, hi = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                y, z = c[:, 1] + dy, c[:, 2] + dz
                ok = (y >= 0) & (y < R) & (z >= 0) & (z < R)
                row = self.off + (z * R + y) * R
                a = torch.where(ok, row + (c[:, 0] - 1).clamp(min=0), 0)
                b = torch.where(ok, row + torch.minimum(c[:, 0] + 1, R - 1) + 1, 0)
                lo.append(start[a])
                hi.append(torch.where(ok, start[b], start[a]))
        lo, cnt = torch.stack(lo, 1), torch.stack(hi, 1) - torch.stack(lo, 1)
        done = torch.cumsum(cnt.sum(1), 0)
        first, n = 0, x.shape[0]
        while first < n:
            base = int(done[first - 1]) if first else 0
            last = max(first + 1, int(torch.searchsorted(done, base + most, right=True)))
            m = cnt[first:last].reshape(-1)
            rep = torch.repeat_interleave(torch.arange(m.numel(), device="cuda"), m)
            j = order[lo[first:last].reshape(-1)[rep] + torch.arange(rep.numel(), device="cuda") - (torch.cumsum(m, 0) - m)[rep]]
            i = first + rep // 9
            d2 = (x[i] - x[j]).square().sum(1)
            hit = d2 < self.at("h", i) ** 2
            yield i[hit], j[hit]
            first = last

    def forces(self, x, v, rates=False):
        """Density, pressure and acceleration; with `rates` also the density rate and J = da/dt of
        the pressure term."""
        n, c = x.shape[0], self.c
        s, q = torch.zeros(n, dtype=x.dtype, device="cuda"), torch.zeros(n, dtype=x.dtype, device="cuda")
        for i, j in self.pairs(x):
            r = x[i] - x[j]
            w = self.at("h", i) ** 2 - r.square().sum(1)
            s.index_add_(0, i, w ** 3)
            if rates:
                q.index_add_(0, i, w ** 2 * (r * (v[i] - v[j])).sum(1))
        rho = c["m"] * c["c6"] * s
        rhodot = -6 * c["m"] * c["c6"] * q
        if int(c["eos"].reshape(-1)[0]) == A.WC_EOS_LINEAR:
            p, pdot = c["p0"] + c["k"] * (rho - c["rho0"]), c["k"] * rhodot
        else:
            y = rho / c["rho0"]
            p, pdot = c["p0"] + c["k"] * (y ** 3 - 1), 3 * c["k"] * y ** 2 / c["rho0"] * rhodot
        if self.on(A.WC_FLAG_WALL_DENSITY):
            rho = rho + self.wall_density(x)
        f, g, jf = (torch.zeros_like(x) for _ in range(3))
        for i, j in self.pairs(x):
            r, u, h = x[i] - x[j], v[i] - v[j], self.at("h", i)
            d = r.square().sum(1).sqrt()
            rj, hd, inv = rho[j], h - d, torch.where(d > 0, 1 / d, 0.0)
            pres = ((p[i] + p[j]) / (2 * rj)).clamp(min=0)
            f.index_add_(0, i, (pres * hd ** 2 * inv)[:, None] * r)
            g.index_add_(0, i, (-hd / rj)[:, None] * u)
            if rates:
                k = hd ** 2 * inv
                dpres = torch.where(pres > 0, (pdot[i] + pdot[j]) / (2 * rj) - pres * rhodot[j] / rj, 0.0)
                rate = dpres * k - pres * hd * inv * (2 + hd * inv) * (r * u).sum(1) * inv
                jf.index_add_(0, i, rate[:, None] * r + (pres * k)[:, None] * u)
        fp, fv, inv = -self.col("m") * self.col("cs"), self.col("m") * self.col("cv") * self.col("mu"), 1 / (rho[:, None] + 1e-16)
        grav = torch.stack([c["gx"].expand(n), c["gy"].expand(n), c["gz"].expand(n)], 1)
        ext = grav * rho[:, None]
        if self.on(A.WC_FLAG_WALL_FORCE):  # the reference's: the length of a 3-vector taken as 3
            near = torch.where(x < c["h"], -x, torch.where(x > c["size"] - c["h"], c["size"] - x, 0.0))
            ext = ext + 0.01 * (c["h"] - 3) ** 2 * near / 3 * c["cs"]
        acc = (fp * f + fv * g + ext) * inv
        return rho, p, acc, rhodot, -rhodot[:, None] * inv * fp * f * inv + fp * jf * inv

    def wall_density(self, x):
        c = self.c

        def w(r):
            return c["m"] * (c["h"] ** 2 - r ** 2) ** 3 * c["c6"]

        h, s, tot = c["h"], c["size"], 0.0
        for a in range(3):  # the reference's z branch tests y
            far = x[:, 1] if a == 2 else x[:, a]
            tot = tot + torch.where(x[:, a] < h, w(x[:, a]), torch.where(far > s - h, w(s - x[:, a]), 0.0))
        return 4 * tot

    def move(self, x, v, a, dt):
        v = v + a * dt
        if self.on(A.WC_FLAG_SPEED_CLAMP):
            v = torch.minimum(torch.maximum(v, -self.col("max_speed")), self.col("max_speed"))
        x, lo, hi = x + v * dt, self.col("border"), self.col("size") - self.col("border")
        out = (x < lo) | (x > hi)
        return torch.minimum(torch.maximum(x, lo), hi), torch.where(out, -self.col("damping") * v, v)


def _consts(p):
    g = list(p.gravity)
    return {"R": p.grid_res, "bin": p.bin_size, "h": p.kernel_radius, "m": p.particle_mass, "rho0": p.rest_density,
            "p0": p.rest_pressure, "k": p.stiffness, "mu": p.viscosity, "c6": p.poly6_const, "cs": p.spiky_const,
            "cv": p.visc_const, "size": p.size, "border": p.wall_border, "damping": p.wall_damping, "gx": g[0], "gy": g[1],
            "gz": g[2], "eos": p.eos, "flags": p.flags, "max_speed": p.max_speed}


def _sorted_order(x, bin_, R, off=0):
    """The cell sort's order: keys in single precision, ties in the input's order."""
    # divided by a tensor: by a scalar torch multiplies with the reciprocal
    bin_ = torch.as_tensor(bin_, dtype=torch.float32, device="cuda")
    c = torch.minimum((x / bin_).long().clamp(min=0), (R[:, None] if torch.is_tensor(R) else torch.tensor(R, device="cuda")) - 1)
    return torch.sort(off + (c[:, 2] * R + c[:, 1]) * R + c[:, 0], stable=True)[1]


def _state64(st):
    both = torch.from_numpy(st.view(np.float32).reshape(-1, 8).copy()).cuda()
    return both[:, :3].contiguous(), both[:, 4:7].contiguous()


def _exact_step(sph, x32, v32, dt, order):
    x, v = x32.double(), v32.double()
    rho, p, acc, _, _ = sph.forces(x, v)
    x, v = sph.move(x, v, acc, dt)
    return {"position": x[order], "density": rho[order], "velocity": v[order], "pressure": p[order]}


def _exact_rollout(case, p, sph, x, v, dt):
    ages, net = case["ages"], None
    if case["mode"] == "network":
        z = np.load(L.DEFAULT_WEIGHTS.with_name(f"local_k{ages + 1}.npz"))
        w = torch.from_numpy(z["params"]).double().cuda()
        a_s, v_s = float(z["accel_scale"]), float(z["velocity_scale"])
        sizes = [(32, 64), (64,), (64, 64), (64,), (64, 16), (16,)]
        net = [t.reshape(s) for t, s in zip(torch.split(w, [math.prod(s) for s in sizes]), sizes)]
    for _ in range(case["cycles"]):
        rho, pr, acc, rhodot, J = sph.forces(x, v, rates=True)
        change = torch.zeros(x.shape[0], ages, 3, dtype=x.dtype, device="cuda")
        if case["mode"] != "stale":
            change += J[:, None] * dt * torch.arange(1, ages + 1, device="cuda")[None, :, None]
        if net:
            h, k = p.kernel_radius, p.stiffness
            wall = torch.stack([x[:, 0], p.size - x[:, 0], x[:, 1], p.size - x[:, 1], x[:, 2], p.size - x[:, 2]], 1)
            y = torch.cat([acc / a_s, J * 1e-3 / a_s, 0.1 * (rhodot / rho)[:, None], v / v_s, (rho / p.rest_density - 1)[:, None],
                           (pr / (k * p.rest_density))[:, None], (wall / h).clamp(0, 1),
                           torch.full_like(x[:, :1], 100 * k / p.rest_density), torch.zeros_like(x[:, :1]).expand(-1, 13)], 1)
            y = torch.relu(torch.relu(y @ net[0] + net[1]) @ net[2] + net[3]) @ net[4] + net[5]
            y = y[:, :3 * ages] * (a_s * (dt / 1e-3) ** 2)
            change += (y - y.mean(0)).reshape(-1, ages, 3)
        x, v = kept = sph.move(x, v, acc, dt)
        for a in range(ages):
            x, v = sph.move(x, v, acc + change[:, a], dt)
        rho = rho + (ages + 1) * dt * rhodot
        pr = p.rest_pressure + p.stiffness * (rho - p.rest_density)
        # the judge: the carried densities against SPH's, plain steps instead where they are over 1 % off
        if float((rho / sph.forces(x, v)[0] - 1).abs().mean()) > 0.01:
            x, v = kept
            for _ in range(ages):
                rho, pr, acc, _, _ = sph.forces(x, v)
                x, v = sph.move(x, v, acc, dt)
    return {"position": x, "density": rho, "velocity": v, "pressure": pr, "reverted": None}


def _exact_net(case, p, st, hist, target, dt, train):
    """The message-passing network in float64; gradients by autograd. Its features and weights
    are held in 16 bits, so they are rounded here too; what is computed from them is not."""
    x32, _ = _state64(st)
    n, h = case["n"], p.kernel_radius
    x, sph = x32.double(), _Sph64(_consts(p))
    both = [(i[i != j], j[i != j]) for i, j in sph.pairs(x)]
    recv, send = torch.cat([b[0] for b in both]), torch.cat([b[1] for b in both])
    v = torch.from_numpy(hist[:, :, :3]).double().cuda()
    a_s = 10.0
    wall = torch.stack([x[:, 0], p.size - x[:, 0], x[:, 1], p.size - x[:, 1], x[:, 2], p.size - x[:, 2]], 1)
    xn = torch.cat([v[0]] + [(v[k - 1] - v[k]) / (dt * a_s) for k in range(1, 5)] +
                   [(wall / h).clamp(0, 1), torch.full_like(x[:, :1], p.stiffness / p.rest_density * 200),
                    torch.zeros(n, 10, dtype=x.dtype, device="cuda")], 1)
    d = (x[recv] - x[send]) / h
    xe = torch.cat([d, d.norm(dim=1, keepdim=True), torch.zeros(d.shape[0], 12, dtype=x.dtype, device="cuda")], 1)
    xn, xe = xn.bfloat16().double(), xe.bfloat16().double()
    flat = torch.from_numpy(np.load(MP_WEIGHTS)["params"]).double().cuda().requires_grad_(train)
    at = 0

    def take(*shape):
        nonlocal at
        at += math.prod(shape)
        return flat[at - math.prod(shape):at].reshape(shape)

    def linear(k, m=128, bias=True):
        w = take(k, m)
        return w + (w.bfloat16().double() - w).detach(), take(m) if bias else 0.0

    def norm(y):
        g, b = take(128), take(128)
        return torch.nn.functional.layer_norm(y, (128,), g, b, 1e-5)

    def mlp(z):
        w, b = linear(z.shape[1])
        z = torch.relu(z @ w + b)
        w, b = linear(128)
        return norm(z @ w + b)

    with torch.set_grad_enabled(train):
        hn, e = mlp(xn), mlp(xe)
        for _ in range(8):
            (we, be), (wi, _), (ws, _) = linear(128), linear(128, bias=False), linear(128, bias=False)
            z = torch.relu(e @ we + be + (hn @ wi)[recv] + (hn @ ws)[send])
            w, b = linear(128)
            e = e + norm(z @ w + b)
            agg = torch.zeros_like(hn).index_add(0, recv, e)
            hn = hn + mlp(torch.cat([hn, agg], 1))
        w, b = linear(128)
        z = torch.relu(hn @ w + b)
        w, b = linear(128, 16)
        y = (z @ w + b)[:, :3]
        if not train:
            return torch.cat([y * a_s, torch.zeros_like(y[:, :1])], 1)
        loss = (y - torch.from_numpy(target[:, :3]).double().cuda() / a_s).square().mean()
        loss.backward()
    return {"loss": loss.detach(), "grads": flat.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "host"):
        p = _params(case)
        x, v = _state64(_scene(case, p, seed))
        dt = np.float32(1 / 60) * np.float32(p.time_scale) if case.get("preset") == "reference" else np.float32(_dt(case["n"]))
        out = _exact_step(_Sph64(_consts(p)), x, v, float(dt), _sorted_order(x, p.bin_size, p.grid_res))
        if case.get("preset") == "reference":
            out.update(ids=None, neighbours=None)
        return out
    if kind == "rollout":
        p = _params(case)
        x, v = _state64(_scene(case, p, seed))
        return _exact_rollout(case, p, _Sph64(_consts(p)), x.double(), v.double(), float(np.float32(_dt(case["n"]))))
    if kind == "batch":
        params, initial = _batch_inputs(case, seed)
        count = torch.tensor([len(s) for s in initial], device="cuda")
        each = [_consts(p) for p in params]
        off = np.concatenate([[0], np.cumsum([c["R"] ** 3 for c in each])])
        c = {k: torch.repeat_interleave(torch.tensor([e[k] for e in each], dtype=torch.float64, device="cuda"), count) for k in each[0]}
        offs = torch.repeat_interleave(torch.from_numpy(off[:-1]).cuda(), count)
        x, v = _state64(np.concatenate(initial))
        order = _sorted_order(x, c["bin"].float()[:, None], c["R"].long(), offs)
        return _exact_step(_Sph64(c, offs, int(off[-1])), x, v, float(np.float32(1e-3)), order)
    if kind in ("train", "predict"):
        p, st, hist, target, dt = _sample_inputs(case, seed)
        return _exact_net(case, p, st, hist, target, float(np.float32(dt)), kind == "train")
    if kind == "gemm":
        t = {k: v.double() if v.is_floating_point() else v for k, v in _gemm_inputs(case, seed).items()}
        if case["form"] == "wgrad":
            chunk = max(1024, (case["rows"] // 256 + 63) // 64 * 64)
            return torch.stack([a.T @ b for a, b in zip(t["a"].split(chunk), t["b"].split(chunk))])
        a = torch.cat([t["a"], t["a2"]], 1) if case["form"] == "concat" else t["a"]
        y = a @ t["b"].T + t["bias"]
        if case["form"] == "layernorm":
            return torch.nn.functional.layer_norm(y, (128,), t["gamma"], t["beta"], 1e-5) + t["resid"]
        if case["form"] == "gather":
            y = y + t["add1"][t["recv"].long()] + t["add2"][t["send"].long()]
        return torch.relu(y)
    return None
