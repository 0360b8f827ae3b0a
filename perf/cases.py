"""The work a user has this framework do, as cases to time: power flows and N-1 batches through ``SecurityAnalysis``,
``BatchContext``, ``ConcurrentBatch`` and ``MultiGridAnalysis``, the batched linear solve on device buffers, and the
learned warm start's network (training step, inference).  The grids are the synthetic 118- to 9,241-bus ones.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` makes what a
program has in hand before the call, ``run(state)`` is one pass, ``work(case)`` counts the bytes and operations a pass
cannot do without, ``tolerance(case)`` says how far two correct implementations may differ and ``exact(case, seed)``
gives the results in 64 bits from plain torch and numpy.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

if "olf-gpu_b200" not in sys.path:
    sys.path.insert(0, os.path.abspath("olf-gpu_b200"))      # the working folder is the repository's root

from olfgpu import native, packing, synthetic  # noqa: E402
from olfgpu.gnn import FEAT_IN, GraphData, WarmStartNet, init_params  # noqa: E402
from olfgpu.learned_start import LearnedStart  # noqa: E402
from olfgpu.security_analysis import ConcurrentBatch, MultiGridAnalysis, SecurityAnalysis  # noqa: E402

TOL = 1e-8
SCHEDULE = (native.LEVELS_SHARED_ALL, 0, 256)      # what SecurityAnalysis and the JNI layer set on their contexts
CHECKPOINT = os.path.join("olf-gpu_b200", "checkpoints", "warmstart_grid9241.npz")
LOADING = {"grid118": (0.9, 1.0), "grid300": (0.9, 1.0), "grid2000": (0.95, 1.0), "grid2000q": (0.95, 1.0),
           "grid9241": (0.95, 1.0)}
# per bus: Jacobian non-zeros (scalars), factor blocks and 2x2 block updates of a factorization
SHAPE = {"grid118": (118, 15.5, 5.6, 6.5), "grid300": (300, 15.4, 6.1, 7.9), "grid2000": (2000, 15.3, 6.8, 12.5),
         "grid2000q": (2000, 15.3, 6.8, 12.5), "grid9241": (9241, 16.0, 7.7, 22.4)}


def listed():
    return [
        # one AC power flow from a flat start: the smallest call, all latency
        {"name": "flow_118", "kind": "flow", "grid": "grid118", "count": 1},
        # a mid-size grid's contingencies with the generators' reactive limits (the outer loop switches PV to PQ)
        {"name": "n1_300_limits", "kind": "n1", "grid": "grid300", "count": 1000, "limits": True, "mixed": False},
        # as many outages as the 2,000-bus grid has non-bridge branches, as one uniform batch
        {"name": "n1_2000_all", "kind": "n1", "grid": "grid2000", "count": 2235, "limits": False, "mixed": False},
        # a ragged batch in mixed precision (FP32 factors, FP64 refinement near convergence)
        {"name": "n1_2000_mixed", "kind": "n1", "grid": "grid2000", "count": 501, "limits": False, "mixed": True},
        # a short list of critical contingencies of a large grid, as an operator's re-check asks for
        {"name": "n1_9241_few", "kind": "n1", "grid": "grid9241", "count": 17, "limits": False, "mixed": False},
        # the benchmark's batch on the plain FP64 engine, as one chunk of a security analysis
        {"name": "n1_9241", "kind": "n1", "grid": "grid9241", "count": 500, "limits": False, "mixed": False},
        # the benchmark's own path: learned start, mixed precision (FP64 near convergence), eight concurrent parts
        {"name": "learned_9241", "kind": "learned", "grid": "grid9241", "count": 500, "parts": 8},
        # grids of uneven size in one launch, reactive limits where the grid has them
        {"name": "uneven", "kind": "uneven", "count300": 301, "count2000": 257, "count9241": 64},
        # the linear solve alone, on device buffers of a caller that does not allocate
        {"name": "linear_2000", "kind": "linear", "grid": "grid2000", "count": 48, "mixed": False},
        # one optimiser step of the warm-start network at the batch the training uses
        {"name": "train_9241", "kind": "train", "grid": "grid9241", "count": 32},
        # the network's predictions for a batch of outages of the 2,000-bus grid
        {"name": "infer_2000", "kind": "infer", "grid": "grid2000", "count": 67},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["flow", "n1", "n1", "n1", "n1", "learned", "uneven", "linear", "train", "infer"])
    if kind == "flow":
        return {"kind": kind, "grid": rng.choice(["grid118", "grid300", "grid2000", "grid9241"]), "count": 1,
                "start": rng.randrange(1 << 16)}
    if kind == "n1":
        grid = rng.choice(["grid118", "grid300", "grid2000", "grid2000q", "grid9241"])
        top = {"grid118": 1000, "grid300": 1000, "grid2000": 2235, "grid2000q": 1000, "grid9241": 500}[grid]
        limits = grid in ("grid300", "grid2000q") and rng.random() < 0.6
        return {"kind": kind, "grid": grid, "count": _log(rng, 2, top), "limits": limits,
                "mixed": not limits and rng.random() < 0.35}
    if kind == "learned":
        return {"kind": kind, "grid": "grid9241", "count": _log(rng, 40, 500), "parts": rng.choice([4, 8])}
    if kind == "uneven":
        return {"kind": kind, "count300": _log(rng, 8, 301), "count2000": _log(rng, 8, 257),
                "count9241": _log(rng, 3, 64)}
    if kind == "linear":
        return {"kind": kind, "grid": rng.choice(["grid118", "grid300", "grid2000"]), "count": _log(rng, 1, 60),
                "mixed": rng.random() < 0.3}
    if kind == "train":
        return {"kind": kind, "grid": rng.choice(["grid300", "grid2000", "grid9241"]), "count": _log(rng, 4, 32)}
    return {"kind": kind, "grid": rng.choice(["grid300", "grid2000"]), "count": _log(rng, 4, 128)}


# ---------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=24)
def _case_grid(name, seed):
    """The named grid at a loading drawn from the seed, with its base case solved on the host."""
    g0 = synthetic.build(name)
    rng = np.random.default_rng([seed, g0.n_bus])
    g = g0.scaled(float(rng.uniform(*LOADING[name])))
    ok, _, vm, va = synthetic.newton_polar(g, g0.base_vm, g0.base_va)
    if not ok:
        raise RuntimeError(f"{name}: the base case does not converge")
    g.base_vm, g.base_va = vm, va
    return g


@functools.lru_cache(maxsize=16)
def _candidates(name, limits):
    """The outages that have a solution at the heaviest loading: a state that never converges follows rounding, so two
    correct implementations end anywhere, and a contingency list keeps such outages apart."""
    p = packing.pack(synthetic.build(name), with_reactive_limits=limits)
    cand = synthetic.outage_candidates(synthetic.build(name))
    sa = SecurityAnalysis(p, reactive_limits=limits)
    r = sa.solve_n1(cand, chunk=min(512, cand.shape[0]), tol=TOL)
    sa.close()
    return cand[(r.status == native.CONVERGED) & (r.iterations <= 5) & (r.total_iterations <= 20)]


def _outages(name, count, seed, limits=False):
    cand = _candidates(name, limits)
    rng = np.random.default_rng([seed, count])
    return np.sort(rng.choice(cand, size=count, replace=count > cand.shape[0]))


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _systems(name, count, seed):
    """Jacobians near the base state as CSR values, their pattern and right-hand sides, through the engine's fill."""
    g = _case_grid(name, seed)
    p = packing.pack(g, with_reactive_limits=False)
    rng = np.random.default_rng([seed, 7])
    x = np.tile(p.x_base, (count, 1))
    x[:, 0::2] += rng.uniform(-0.02, 0.02, (count, p.n_bus))
    x[:, 1::2] += rng.uniform(-0.02, 0.02, (count, p.n_bus))
    s = native.Structure(p, native.PLAN_DEFAULT)
    ctx = native.BatchContext(s, count)
    J, _ = ctx.debug_fill(x, p.target, p.base_row_mode, np.zeros((count, p.n_elements), np.uint8))
    return p, s, ctx, J, rng.standard_normal((count, p.n))


def _net_inputs(case, seed):
    """Node inputs, outaged branches and targets of a batch of samples: base-case features normalised over the buses,
    the outage's endpoint flag and flows, sparse normalised state changes."""
    g = _case_grid(case["grid"], seed)
    p = packing.pack(g, with_reactive_limits=False)
    from olfgpu.learned_start import branch_flows, node_features
    f = node_features(p, p.x_base)
    f[:, :4] = (f[:, :4] - f[:, :4].mean(0)) / np.maximum(f[:, :4].std(0), 1e-6)
    p1, q1 = branch_flows(g, p.x_base)
    scale = max(float(np.std([p1, q1])), 1e-6)
    B, nb = case["count"], g.n_bus
    outs = _outages(case["grid"], B, seed).astype(np.int32)
    x0 = np.zeros((B, nb, FEAT_IN), np.float32)
    x0[:, :, :7] = f
    rows = np.arange(B)
    for end, sign in ((g.f[outs], 1.0), (g.t[outs], -1.0)):
        x0[rows, end, 7] = 1.0
        x0[rows, end, 8] = sign * p1[outs] / scale
        x0[rows, end, 9] = sign * q1[outs] / scale
    rng = np.random.default_rng([seed, 11])
    target = rng.standard_normal((B * nb, 2)).astype(np.float32)
    return g, x0.reshape(B * nb, FEAT_IN), outs, target


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("flow", "n1", "learned"):
        g = _case_grid(case["grid"], seed)
        limits = bool(case.get("limits"))
        p = packing.pack(g, with_reactive_limits=limits)
    if kind == "flow":
        s = native.Structure(p, native.PLAN_DEFAULT)
        ctx = native.BatchContext(s, 1)
        ctx.set_schedule(*SCHEDULE)
        return {"kind": kind, "p": p, "ctx": ctx, "none": np.zeros((1, p.n_elements), np.uint8)}
    if kind == "n1":
        sa = SecurityAnalysis(p, precision=native.MIXED if case["mixed"] else native.FP64,
                              refinement_steps=3 if case["mixed"] else 1, reactive_limits=limits)
        return {"kind": kind, "sa": sa, "outages": _outages(case["grid"], case["count"], seed, limits)}
    if kind == "learned":
        outs = _outages(case["grid"], case["count"], seed)
        ls = LearnedStart.load(CHECKPOINT, synthetic.build(case["grid"]))
        s = native.Structure(p, native.PLAN_DEFAULT)
        cb = ConcurrentBatch(s, case["count"], case["parts"], native.MIXED, 3, native.MIXED_FP64_NEAR, SCHEDULE)
        start = torch.empty((case["count"], p.n), dtype=torch.float64, device="cuda")
        cb.set_device_start(start)
        return {"kind": kind, "p": p, "ls": ls, "cb": cb, "start": start, "outages": outs, "s": s,
                "x0": _pinned(p.x_base), "target": _pinned(p.target), "mode": _pinned(p.base_row_mode),
                "masks": _pinned(p.outage_masks(outs)), "out": _pinned(np.zeros((case["count"], p.n + 3)))}
    if kind == "uneven":
        names = ("grid300", "grid2000q", "grid9241")
        counts = (case["count300"], case["count2000"], case["count9241"])
        packs = [packing.pack(_case_grid(n, seed)) for n in names]
        ma = MultiGridAnalysis(packs, counts, schedule=(0, 0, 0), ordering=native.PLAN_DEFAULT, member_schedule=SCHEDULE)
        return {"kind": kind, "ma": ma, "outages": [_outages(n, c, seed, n != "grid9241") for n, c in zip(names, counts)]}
    if kind == "linear":
        p, s, ctx, J, rhs = _systems(case["grid"], case["count"], seed)
        return {"kind": kind, "s": s, "ctx": ctx, "count": case["count"],
                "precision": native.MIXED if case["mixed"] else native.FP64, "J": torch.from_numpy(J).cuda(),
                "rhs": torch.from_numpy(rhs).cuda(),
                "out": torch.zeros((case["count"], p.n), dtype=torch.float64, device="cuda")}
    g, x0, outs, target = _net_inputs(case, seed)
    net = WarmStartNet(GraphData.from_grid(g), 4, params=init_params(4, seed % 1000))
    return {"kind": kind, "net": net, "x0": torch.from_numpy(x0).cuda().to(torch.bfloat16),
            "outages": torch.from_numpy(outs).cuda(), "target": torch.from_numpy(target).cuda()}


# ---------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------
def _rows(out, n):
    """Result rows [x(n), iterations, ||F||inf, status] without the residual: at convergence it is rounding noise."""
    return {"x": out[:, :n], "iterations": out[:, n], "status": out[:, n + 2]}


def _result(r):
    return {"x": r.x, "iterations": r.iterations, "status": r.status}


def run(state):
    kind = state["kind"]
    if kind == "flow":
        p = state["p"]
        return _rows(state["ctx"].solve(p.x_flat, p.target, p.base_row_mode, state["none"], tol=TOL), p.n)
    if kind == "n1":
        return _result(state["sa"].solve_n1(state["outages"], tol=TOL))
    if kind == "learned":
        p = state["p"]
        state["ls"].predict_device(p, state["x0"], state["outages"], out=state["start"])
        torch.cuda.current_stream().synchronize()       # the engine reads the start on its own streams
        out, _ = state["cb"].solve(state["x0"], state["target"], state["mode"], state["masks"], tol=TOL,
                                   out=state["out"])
        return {"x": out[:, :p.n], "status": out[:, p.n + 2]}
    if kind == "uneven":
        return [_result(r) for r in state["ma"].solve(state["outages"], tol=TOL)[0]]
    if kind == "linear":
        state["s"].linear_solve_noalloc(state["count"], state["J"].data_ptr(), state["rhs"].data_ptr(),
                                        state["out"].data_ptr(), state["precision"],
                                        torch.cuda.current_stream().cuda_stream)
        return state["out"]
    net = state["net"]
    if kind == "train":
        loss = net.loss_and_grad(state["x0"], state["outages"], state["target"])
        net.adam(0.0)          # a rate of zero: the moments move, the weights stay, so a pass can be repeated
        return {"loss": loss, "gradients": net.grad}
    return net.forward(state["x0"], state["outages"])[:, :2]


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without, and what it may differ by
# ---------------------------------------------------------------------------------------------------------------
def _solve_work(grid, count, iterations):
    """Inputs (base vectors, outage list) and result rows; per iteration and scenario the Jacobian's and the 2x2 block
    factorization's and substitutions' operations (16 per block update, 8 per factor block)."""
    nb, nnz, blocks, updates = SHAPE[grid]
    flops = nb * (nnz * 6 + updates * 16 + blocks * 8)
    return {"bytes": count * (2 * nb + 3) * 8 + 6 * nb * 8 + count * 4, "flops": count * iterations * flops}


def work(case):
    kind = case["kind"]
    if kind in ("flow", "n1", "learned"):
        return _solve_work(case["grid"], case["count"], 5 if kind == "flow" else 6 if case.get("limits") else 3)
    if kind == "uneven":
        parts = [_solve_work("grid300", case["count300"], 6), _solve_work("grid2000q", case["count2000"], 6),
                 _solve_work("grid9241", case["count9241"], 3)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if kind == "linear":
        nb, nnz, blocks, updates = SHAPE[case["grid"]]
        return {"bytes": case["count"] * nb * (nnz + 4) * 8, "flops": case["count"] * nb * (updates * 16 + blocks * 8)}
    nb = SHAPE[case["grid"]][0]
    rows, edges = case["count"] * nb, case["count"] * nb * 3.4
    dense = 2 * rows * (16 * 64 + 4 * (64 * 128 + 128 * 64) + 64 * 16)
    forward = {"bytes": rows * (FEAT_IN * 2 + 8), "flops": dense + 4 * edges * 64 * 4}
    if kind == "infer":
        return forward
    return {"bytes": forward["bytes"] + rows * 8 + 51000 * 4 * 6, "flops": 3 * forward["flops"]}


def tolerance(case):
    """About four times what the path differs from its 64-bit results by (see exact)."""
    kind = case["kind"]
    if kind in ("train", "infer"):
        return {"rel": 4e-2}          # bf16 weights and activations through four layers: 1e-2 seen
    if kind == "linear":
        return {"rel": 2e-3} if case["mixed"] else {"rel": 1e-11}
    if kind == "learned" or case.get("mixed"):
        # a scenario may stop anywhere inside the 1e-8 mismatch ball (its first steps are FP32, or its start comes from
        # a bf16 network): 6.5e-10 seen
        return {"rel": 1e-8, "max": 1e-6, "differ": 0.0}
    return {"rel": 1e-10, "max": 1e-8, "differ": 0.0}


# ---------------------------------------------------------------------------------------------------------------
# The results in 64 bits: plain torch, no code of this package beyond the input data
# ---------------------------------------------------------------------------------------------------------------
class _Network:
    """The grid's complex admittance equations for a batch of lanes: V is [buses, lanes]."""

    def __init__(self, g, outages, device):
        self.nb, self.dev = g.n_bus, device
        t = lambda a: torch.as_tensor(np.asarray(a), device=device)  # noqa: E731
        ys = 1.0 / (g.r + 1j * g.x)
        sh = 0.5j * g.b
        yff, yft, ytt = g.ratio ** 2 * (ys + sh), -g.ratio * ys, ys + sh
        diag = np.zeros(g.n_bus, complex)
        np.add.at(diag, g.shunt_bus, g.shunt_g + 1j * g.shunt_b)
        if g.open_bus.shape[0]:
            yo, far = 1.0 / (g.open_r + 1j * g.open_x), 0.5j * g.open_b
            np.add.at(diag, g.open_bus, far + yo * far / (yo + far))
        idx = np.arange(g.n_bus)
        self.Y = torch.sparse_coo_tensor(
            t(np.stack([np.concatenate([g.f, g.f, g.t, g.t, idx]), np.concatenate([g.f, g.t, g.f, g.t, idx])])),
            t(np.concatenate([yff, yft, yft, ytt, diag])), (g.n_bus, g.n_bus)).coalesce().to_sparse_csr()
        self.f, self.t = (t(g.f[outages]), t(g.t[outages])) if outages is not None else (None, None)
        if outages is not None:
            self.out = t(np.stack([yff[outages], yft[outages], ytt[outages]]))
        spec = np.zeros(g.n_bus, complex)
        np.add.at(spec, g.gen_bus, g.gen_p + 0j)
        np.add.at(spec, g.load_bus, -(g.load_p + 1j * g.load_q))
        self.spec = t(spec)[:, None]
        pv = np.zeros(g.n_bus, bool)
        pv[g.gen_bus] = True
        vset = np.zeros(g.n_bus)
        vset[g.gen_bus] = g.gen_vset
        self.fixed_v, self.vset, self.slack = t(pv)[:, None], t(vset)[:, None], int(g.slack)

    def current(self, V):
        """Y V with each lane's outaged branch taken out."""
        c = self.Y @ V
        if self.f is not None and V.shape[1] == self.f.shape[0]:
            k = torch.arange(V.shape[1], device=self.dev)
            vf, vt = V[self.f, k], V[self.t, k]
            c[self.f, k] -= self.out[0] * vf + self.out[1] * vt
            c[self.t, k] -= self.out[1] * vf + self.out[2] * vt
        return c

    def rows(self, s, dth, dvm):
        """Stacked rows [2 buses, lanes] (2b: P or slack angle, 2b + 1: Q or voltage) of powers s and identities."""
        out = torch.empty((2 * self.nb, s.shape[1]), dtype=torch.float64, device=self.dev)
        out[0::2], out[1::2] = s.real, torch.where(self.fixed_v, dvm, s.imag)
        out[2 * self.slack] = dth[self.slack]
        return out

    def mismatch(self, x):
        th, vm = x[0::2], x[1::2]
        V = vm * torch.exp(1j * th)
        return self.rows(V * self.current(V).conj() - self.spec, th, vm - self.vset)

    def tangent(self, x, d):
        """J(x) d for directions d [2 buses, lanes]; x has one column or as many as d."""
        th, vm, dth, dvm = x[0::2], x[1::2], d[0::2], d[1::2]
        e = torch.exp(1j * th)
        V = vm * e
        dV = e * (dvm + 1j * vm * dth)
        return self.rows(dV * self.current(V).conj() + V * self.current(dV).conj(), dth, dvm)

    def jacobian(self, x):
        """The dense Jacobian of one lane's state [2 buses, 1], without outages."""
        n = 2 * self.nb
        J = torch.empty((n, n), dtype=torch.float64, device=self.dev)
        for a in range(0, n, 512):
            b = min(n, a + 512)
            d = torch.zeros((n, b - a), dtype=torch.float64, device=self.dev)
            d[torch.arange(a, b), torch.arange(b - a)] = 1.0
            J[:, a:b] = self.tangent(x, d)
        return J


def _newton(g, outages, x0, extra=0):
    """Newton's iterations of every lane from x0 [n] at the engine's stopping rule; each step solved to rounding by
    refinement, preconditioned with the base state's inverse corrected for the lane's outage.  Lanes that meet the rule
    stay, `extra` more steps excepted.  Returns (x [lanes, n], iterations) or None when a lane does not converge."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    base = _Network(g, None, dev)
    net = _Network(g, outages, dev)
    n, lanes = 2 * g.n_bus, 1 if outages is None else len(outages)
    xb = torch.as_tensor(x0, device=dev)[:, None]
    inv = None
    if outages is not None:
        inv = torch.linalg.inv(base.jacobian(xb))
        f, t = net.f, net.t
        idx = torch.stack([2 * f, 2 * f + 1, 2 * t, 2 * t + 1])                       # [4, lanes]
        k = torch.arange(lanes, device=dev)
        xt = xb.expand(n, lanes)
        D = torch.empty((lanes, 4, 4), dtype=torch.float64, device=dev)             # the outage's change of J, [row, col]
        for c in range(4):
            d = torch.zeros((n, lanes), dtype=torch.float64, device=dev)
            d[idx[c], k] = 1.0
            D[:, :, c] = (net.tangent(xt, d) - base.tangent(xt, d))[idx, k].T
        W = inv[:, idx.reshape(-1)].reshape(n, 4, lanes)                               # inv E
        small = W[idx[:, None, :], torch.arange(4, device=dev)[None, :, None], k].permute(2, 0, 1)
        cap = torch.linalg.inv(torch.eye(4, dtype=torch.float64, device=dev) + D @ small) @ D

    def solve(x, r):
        if inv is None:
            return torch.linalg.solve(net.jacobian(x), r)
        d = torch.zeros_like(r)
        res = r
        for _ in range(40):
            z = inv @ res
            z = z - torch.einsum("ncl,cl->nl", W, torch.einsum("lcd,dl->cl", cap, z[idx, k]))
            d = d + z
            res = r - net.tangent(x, d)
            if float(res.abs().max()) <= 1e-14 * float(r.abs().max()):
                break
        bad = torch.nonzero(~(res.abs().amax(0) <= 1e-12 * r.abs().amax(0))).flatten().tolist()
        for l in bad if n <= 4000 else []:          # the correction did not contract: this lane's own dense solve
            one = _Network(g, np.asarray(outages)[l:l + 1], dev)
            A = base.jacobian(x[:, l:l + 1])
            for c in range(4):
                e = torch.zeros((n, 1), dtype=torch.float64, device=dev)
                e[idx[c, l]] = 1.0
                A[:, idx[c, l]] = one.tangent(x[:, l:l + 1], e)[:, 0]
            d[:, l] = torch.linalg.solve(A, r[:, l])
        return d
    x = xb.expand(n, lanes).clone()
    its = torch.zeros(lanes, dtype=torch.int64, device=dev)
    left = torch.full((lanes,), extra, dtype=torch.int64, device=dev)
    for _ in range(15 + extra):
        F = net.mismatch(x)
        done = (F.abs().amax(0) < TOL) & (its > 0) & (left <= 0)
        left = torch.where((F.abs().amax(0) < TOL) & (its > 0), left - 1, left)
        if bool(done.all()):
            return x.T.contiguous().cpu().numpy(), its.cpu().numpy()
        step = solve(x, -F)
        go = ~done
        x = torch.where(go, x + step, x)
        its = its + go.to(torch.int64)
    return None


def _net_exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g, x0, outs, target = _net_inputs(case, seed)
    host = init_params(4, seed % 1000)
    B, nb, grad = case["count"], g.n_bus, case["kind"] == "train"
    par = {}
    for name, v in host.items():
        w = torch.from_numpy(v).to(dev)
        if name.startswith("w_") and not name.startswith("w_e"):
            w = w.to(torch.bfloat16)                                     # the weights the matrix products read
        par[name] = w.double().requires_grad_(grad)
    feats = np.stack([g.r, g.x, g.b, g.ratio], axis=1)
    feats = (feats - feats.mean(0)) / np.maximum(feats.std(0), 1e-9)
    es = torch.from_numpy(np.concatenate([feats, feats]).astype(np.float32)).to(dev).double()
    src = torch.as_tensor(np.concatenate([g.f, g.t]), device=dev).long()
    dst = torch.as_tensor(np.concatenate([g.t, g.f]), device=dev).long()
    branch = np.concatenate([np.arange(g.f.shape[0])] * 2)
    keep = torch.as_tensor(branch[None, :] != outs[:, None], device=dev)[..., None]
    h = torch.relu(torch.from_numpy(x0).to(dev).to(torch.bfloat16).double() @ par["w_in"] + par["b_in"])
    for l in range(4):
        pq = (h @ par[f"w_pq{l}"]).reshape(B, nb, 128)
        msg = torch.relu(pq[:, src, :64] + pq[:, dst, 64:] + (es @ par[f"w_e{l}"] + par[f"b_msg{l}"])) * keep
        agg = torch.zeros((B, nb, 64), dtype=torch.float64, device=dev).index_add(1, dst, msg).reshape(B * nb, 64)
        h = h + torch.relu(torch.cat([h, agg], dim=1) @ par[f"w_upd{l}"] + par[f"b_upd{l}"])
    out = (h @ par["w_out"] + par["b_out"])[:, :2]
    if not grad:
        return out
    loss = ((out - torch.from_numpy(target).to(dev).double()) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "gradients": {k: v.grad for k, v in par.items()}}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "infer"):
        return _net_exact(case, seed)
    if kind == "linear":
        p, s, ctx, J, rhs = _systems(case["grid"], case["count"], seed)
        e = s.export()
        rows = np.repeat(np.arange(p.n), np.diff(e["row_ptr"]))
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        out = []
        for k in range(case["count"]):
            A = torch.zeros((p.n, p.n), dtype=torch.float64, device=dev)
            A[torch.as_tensor(rows, device=dev), torch.as_tensor(e["col_idx"], device=dev).long()] = \
                torch.as_tensor(J[k], device=dev)
            out.append(torch.linalg.solve(A, torch.as_tensor(rhs[k], device=dev)))
        return torch.stack(out)
    if kind == "uneven" or case.get("limits"):
        return None                                  # the reactive-limit loop has no plain 64-bit counterpart here
    g = _case_grid(case["grid"], seed)
    p = packing.pack(g, with_reactive_limits=False)
    if kind == "flow":
        r = _newton(g, None, p.x_flat) if g.n_bus <= 2000 else None
    else:
        r = _newton(g, _outages(case["grid"], case["count"], seed), p.x_base, extra=2 if kind == "learned" else 0)
    if r is None:
        return None
    x, its = r
    if kind == "learned":
        return {"x": x, "status": np.zeros(x.shape[0])}
    its = its.astype(np.float64) if kind == "flow" else its
    return {"x": x, "iterations": its, "status": np.zeros_like(its)}
