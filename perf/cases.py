"""The solve path's work as its users run it: one dict per case, through the package's public entry points.

A program keeps the network and its factor and solves for new right-hand sides, injections or
outages, so the network of a case is fixed by its sizes (seeded grids, `ybus_b200.grids`) and the
seed of `prepare` draws what the program would be given: right-hand sides, injections, outages,
weights. The handles (uploaded factor, DC network, adjoint) are made anew by each `prepare`. All
device work runs on the library's own stream of one `Gpu`.

Kinds and ranges (sizes log-uniform, odd ones included):

- solve: B' of a grid of 500 to 10,000 buses (1.35 branches a bus), 1 to 13,499 right-hand sides
  (unit injections or branch columns), FP64 or FP32 with FP64 refinement, device or host arrays;
- jacobian: the Newton-Raphson Jacobian's LU of 500 to 10,000 buses, 1 to 4,096 right-hand sides,
  plain or transposed, FP64, device arrays;
- columns: PTDF or LODF columns of 500 to 10,000 buses, 1 to 1,024 columns, to host arrays;
- n1: N-1 screening, 1,000 to 10,000 buses, 8 to 500 outages of up to 64 scenarios, pinned host
  injections, FP64 or FP32 with refinement;
- adjoint: the flow loss forward and backward, 500 to 10,000 buses, 1 to 1,024 scenarios, pinned
  host arrays;
- complex: 1 to 16 Ybus LU factors of 500 to 46,293 buses (1.3 branches a bus), 1 to 128 complex
  right-hand sides each, complex128 or complex64 with refinement, device arrays.
"""
import functools
import math

import numpy as np
import torch

from ybus_b200 import FP32, FP64, Gpu, GpuFactor, configs, grids, host, solve_batch_complex
from ybus_b200.dc import DcNetwork, FlowLoss

MAX_STEPS, TOLERANCE = 3, 1e-10  # the refined solve's corrections at most and its relative residual
MARGIN = 0.8                     # the flow loss's share of the limit
DENSE_COMPLEX = 16000            # networks up to this order are checked against a dense 64-bit solve
COMPLEX_SIZES = [int(n) for n in configs.complex_sizes()]  # the 16 networks of the complex batch, largest first


def listed():
    return [
        # One injection on a 2,000-bus grid: an interactive what-if, where latency counts
        {"name": "solve_2k_one", "kind": "solve", "buses": 2000, "extra": 700, "count": 1, "rhs": "units",
         "precision": "fp64", "host": False},
        # 256 unit injections on the 2,000-bus grid from and to the caller's host arrays
        {"name": "solve_2k_host", "kind": "solve", "buses": 2000, "extra": 700, "count": 256, "rhs": "units",
         "precision": "fp64", "host": True},
        # A ragged block of sensitivity columns of the 10,000-bus grid
        {"name": "solve_10k_block", "kind": "solve", "buses": 10000, "extra": 3500, "count": 999, "rhs": "branches",
         "precision": "fp64", "host": False},
        # Every branch's column of the 10,000-bus grid: the whole PTDF block in one call
        {"name": "solve_10k_ptdf", "kind": "solve", "buses": 10000, "extra": 3500, "count": 13499, "rhs": "branches",
         "precision": "fp64", "host": False},
        # A small block through FP32 substitution with FP64 refinement
        {"name": "refined_10k_block", "kind": "solve", "buses": 10000, "extra": 3500, "count": 256, "rhs": "branches",
         "precision": "refined", "host": False},
        # The whole PTDF block through FP32 substitution with FP64 refinement
        {"name": "refined_10k_ptdf", "kind": "solve", "buses": 10000, "extra": 3500, "count": 13499, "rhs": "branches",
         "precision": "refined", "host": False},
        # A power flow's Jacobian solved for many mismatches (batched Newton steps, AC sensitivities)
        {"name": "jacobian_10k", "kind": "jacobian", "buses": 10000, "count": 4096, "transposed": False},
        # A block of PTDF columns handed to the caller as flows per branch
        {"name": "ptdf_columns_10k", "kind": "columns", "buses": 10000, "extra": 3500, "count": 1000, "what": "ptdf"},
        # Security screening: outages under many injection scenarios, the largest loading of each
        {"name": "n1_10k", "kind": "n1", "buses": 10000, "extra": 3500, "outages": 300, "scenarios": 64,
         "precision": "fp64"},
        # A training step through the flow loss: gradients by injection and by susceptance
        {"name": "adjoint_10k", "kind": "adjoint", "buses": 10000, "extra": 3500, "scenarios": 1024},
        # 16 admittance networks of uneven sizes in one launch, complex128
        {"name": "complex_16", "kind": "complex", "networks": 16, "largest": COMPLEX_SIZES[0],
         "smallest": COMPLEX_SIZES[-1], "count": 128, "precision": "fp64"},
        # The same batch through complex64 substitution with complex128 refinement
        {"name": "complex_16_refined", "kind": "complex", "networks": 16, "largest": COMPLEX_SIZES[0],
         "smallest": COMPLEX_SIZES[-1], "count": 128, "precision": "refined"},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "jacobian", "columns", "n1", "adjoint", "complex", "complex"])
    if kind == "complex":
        largest = log(500, 46293)
        return {"kind": kind, "networks": rng.randint(1, 16), "largest": largest, "smallest": log(500, largest),
                "count": log(1, 128), "precision": rng.choice(["fp64", "refined"])}
    buses = log(1000 if kind == "n1" else 500, 10000)
    if kind == "jacobian":
        return {"kind": kind, "buses": buses, "count": log(1, 4096), "transposed": rng.random() < 0.5}
    case = {"kind": kind, "buses": buses, "extra": int(0.35 * buses)}
    if kind == "solve":
        host_arrays = rng.random() < 0.25
        case.update(count=log(1, 2048 if host_arrays else 13499), rhs=rng.choice(["units", "branches"]),
                    precision="fp64" if host_arrays else rng.choice(["fp64", "fp64", "refined"]), host=host_arrays)
    elif kind == "columns":
        case.update(count=log(1, 1024), what=rng.choice(["ptdf", "lodf"]))
    elif kind == "n1":
        case.update(outages=log(8, 300), scenarios=rng.randint(1, 64), precision=rng.choice(["fp64", "refined"]))
    else:
        case.update(scenarios=log(1, 1024))
    return case


# ---- networks and inputs ----------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def gpu():
    return Gpu.new(0)


@functools.lru_cache(maxsize=8)
def grid(buses, extra):
    return grids.make_grid(buses, extra, grids.SEED_BASE + buses)


@functools.lru_cache(maxsize=4)
def jacobian(buses):
    return configs.jacobian_system(buses, 1, grids.SEED_BASE + buses)


@functools.lru_cache(maxsize=64)
def admittance(buses, index):
    """Network `index` of a batch: its Ybus (CSC) and COLAMD LU."""
    g = grids.make_complex_grid(buses, grids.SEED_BASE + 60 + index)
    r, c, v = grids.ybus_triplets(g)
    a = host.Matrix.from_triplets(buses, buses, r, c, v, by_rows=False)
    return a, host.lu(a, host.COLAMD), (r, c, v)


def complex_buses(case):
    """The batch's orders, evenly spread in logarithm between the largest and the smallest; the
    workload's own 16 where its ends are given."""
    k, lo, hi = case["networks"], case["smallest"], case["largest"]
    if (k, hi, lo) == (len(COMPLEX_SIZES), COMPLEX_SIZES[0], COMPLEX_SIZES[-1]):
        return COMPLEX_SIZES
    return [int(round(hi * (lo / hi) ** (i / max(k - 1, 1)))) for i in range(k)]


def randoms(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def branch_ends(g):
    """Branch ends as unknowns (bus - 1; bus 0 is the slack: -1) and susceptances, on the GPU."""
    return (torch.from_numpy(g.frm - 1).cuda(), torch.from_numpy(g.to - 1).cuda(),
            torch.from_numpy(1.0 / g.x).cuda())


def right_hand_sides(case, seed):
    """(count, buses - 1): unit injections at random buses, or the columns of random branches
    (each branch at most once in a round over all of them)."""
    g = grid(case["buses"], case["extra"])
    n, count, r = g.n_bus - 1, case["count"], randoms(seed)
    b = torch.zeros(count, n, dtype=torch.float64, device="cuda")
    rows = torch.arange(count, device="cuda")
    if case["rhs"] == "units":
        b[rows, torch.randint(0, n, (count,), generator=r, device="cuda")] = 1.0
        return b
    rounds = -(-count // g.n_branch)
    k = torch.cat([torch.randperm(g.n_branch, generator=r, device="cuda") for _ in range(rounds)])[:count]
    f, t, y = (e[k] for e in branch_ends(g))
    for end, value in ((f, y), (t, -y)):
        keep = end >= 0
        b[rows[keep], end[keep]] += value[keep]
    return b


def jacobian_rhs(case, seed):
    n = jacobian(case["buses"]).lu.n
    return torch.randn(case["count"], n, dtype=torch.float64, device="cuda", generator=randoms(seed))


def pinned(t):
    """The values of a GPU tensor in pinned host memory, as a numpy array."""
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def injections(buses, count, r):
    """(count, buses) N(0, 0.1) injections, the slack (bus 0) taking the balance."""
    p = 0.1 * torch.randn(count, buses, dtype=torch.float64, device="cuda", generator=r)
    p[:, 0] = -p[:, 1:].sum(1)
    return p


def outage_inputs(case, seed):
    """(outaged, scenario_ptr, injections on the GPU, weights) of an N-1 screening."""
    g = grid(case["buses"], case["extra"])
    rng = np.random.default_rng(seed)
    outaged = rng.choice(np.flatnonzero(~bridges(case["buses"], case["extra"])), case["outages"], replace=False)
    counts = np.random.default_rng(case["outages"]).integers(1, case["scenarios"] + 1, outaged.size)  # U[1, scenarios]
    ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    return outaged, ptr, injections(g.n_bus, int(ptr[-1]), randoms(seed)), 1.0 / rng.uniform(0.5, 2.0, g.n_branch)


@functools.lru_cache(maxsize=8)
def bridges(buses, extra):
    return DcNetwork.from_grid(gpu(), grid(buses, extra)).bridges()


def adjoint_inputs(case, seed):
    g = grid(case["buses"], case["extra"])
    r = randoms(seed)
    p = injections(g.n_bus, case["scenarios"], r)
    return p, 0.5 + 1.5 * torch.rand(g.n_branch, dtype=torch.float64, device="cuda", generator=r)


def column_ids(case, seed):
    g = grid(case["buses"], case["extra"])
    rng = np.random.default_rng(seed)
    return rng.integers(0, g.n_bus if case["what"] == "ptdf" else g.n_branch, case["count"])


def complex_rhs(case, seed):
    """Per network (count, buses) complex128 on the GPU, N(0, 1) + i N(0, 1)."""
    r = randoms(seed)
    return [torch.complex(*(torch.randn(case["count"], n, dtype=torch.float64, device="cuda", generator=r)
                            for _ in range(2))) for n in complex_buses(case)]


# ---- what a program has in hand, and its call ---------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "solve":
        bp = configs.bprime(grid(case["buses"], case["extra"]))
        f = GpuFactor.from_cholesky(gpu(), host.cholesky(bp))
        if case["precision"] == "refined":
            f.attach_matrix(bp)
        b = right_hand_sides(case, seed)
        if case["host"]:
            b = b.cpu().numpy()
        else:
            state["x"] = torch.empty_like(b)
        state.update(factor=f, b=b)
    elif kind == "jacobian":
        lu = jacobian(case["buses"]).lu
        make = GpuFactor.from_lu_transposed if case["transposed"] else GpuFactor.from_lu
        b = jacobian_rhs(case, seed)
        state.update(factor=make(gpu(), lu), b=b, x=torch.empty_like(b))
    elif kind == "columns":
        state.update(net=DcNetwork.from_grid(gpu(), grid(case["buses"], case["extra"])), ids=column_ids(case, seed))
    elif kind == "n1":
        outaged, ptr, inj, weights = outage_inputs(case, seed)
        state.update(net=DcNetwork.from_grid(gpu(), grid(case["buses"], case["extra"])), outaged=outaged, ptr=ptr,
                     injections=pinned(inj), weights=weights)
    elif kind == "adjoint":
        p, limits = adjoint_inputs(case, seed)
        net = DcNetwork.from_grid(gpu(), grid(case["buses"], case["extra"]))
        state.update(loss=FlowLoss(net, case["scenarios"]), p=pinned(p), limits=limits.cpu().numpy(),
                     grad_p=pinned(torch.zeros_like(p)), grad_b=np.zeros(net.n_branch))
    else:
        state["factors"] = []
        for i, n in enumerate(complex_buses(case)):
            a, lu, _ = admittance(n, i)
            f = GpuFactor.from_lu_complex(gpu(), lu)
            f.attach_matrix_complex(a)
            state["factors"].append(f)
        state["b"] = complex_rhs(case, seed)
        state["x"] = [torch.empty_like(b) for b in state["b"]]
    torch.cuda.synchronize()  # the inputs are there before the library's stream reads them
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("solve", "jacobian"):
        f, b = state["factor"], state["b"]
        if case.get("host"):
            return f.solve_many(b)
        x = state["x"]
        if case.get("precision") == "refined":
            f.solve_many_refined_device(b.data_ptr(), x.data_ptr(), case["count"], MAX_STEPS, TOLERANCE)
        else:
            f.solve_many_device(b.data_ptr(), x.data_ptr(), case["count"], FP64)
        return x
    if kind == "columns":
        return (state["net"].ptdf_columns if case["what"] == "ptdf" else state["net"].lodf_columns)(state["ids"])
    if kind == "n1":
        return state["net"].outage_loadings_batch(state["outaged"], state["ptr"], state["injections"],
                                                  state["weights"], FP64 if case["precision"] == "fp64" else FP32)
    if kind == "adjoint":
        loss = state["loss"].forward(state["p"], state["limits"], MARGIN)
        return (np.float64(loss),) + state["loss"].backward(state["grad_p"], state["grad_b"])
    solve_batch_complex(state["factors"], [b.data_ptr() for b in state["b"]], [x.data_ptr() for x in state["x"]],
                        [case["count"]] * case["networks"], FP64 if case["precision"] == "fp64" else FP32, MAX_STEPS,
                        TOLERANCE)
    return state["x"]


# ---- the least a pass must move and compute ------------------------------------------------------------

def work(case):
    """Right-hand sides in, results out and the factor once; two operations per factor entry and
    right-hand side (eight for complex values)."""
    kind = case["kind"]
    if kind == "complex":
        lus = [admittance(n, i)[1] for i, n in enumerate(complex_buses(case))]
        entries = sum(lu.l.idx.size + lu.u.idx.size for lu in lus)
        return {"bytes": 32 * case["count"] * sum(lu.n for lu in lus) + 20 * entries,
                "flops": 8 * entries * case["count"]}
    if kind == "jacobian":
        lu = jacobian(case["buses"]).lu
        entries = lu.l.idx.size + lu.u.idx.size
        return {"bytes": 16 * lu.n * case["count"] + 12 * entries, "flops": 2 * entries * case["count"]}
    g = grid(case["buses"], case["extra"])
    entries, n, m = host.cholesky(configs.bprime(g)).l.idx.size, g.n_bus - 1, g.n_branch
    if kind == "solve":
        return {"bytes": 16 * n * case["count"] + 12 * entries, "flops": 4 * entries * case["count"]}
    if kind == "columns":  # pairs in, flows out
        return {"bytes": 8 * m * case["count"] + 12 * entries, "flops": (4 * entries + 3 * m) * case["count"]}
    if kind == "n1":  # injections in, one loading a scenario out
        scenarios = case["outages"] * (case["scenarios"] + 1) // 2
        return {"bytes": 8 * g.n_bus * scenarios + 12 * entries, "flops": (4 * entries + 9 * m) * scenarios}
    count = case["scenarios"]  # injections in, their gradient out, two solves
    return {"bytes": 16 * g.n_bus * count + 12 * entries, "flops": (8 * entries + 20 * m) * count}


# ---- the same results in plain 64-bit torch ------------------------------------------------------------

def dense_bprime(g):
    f, t, y = branch_ends(g)
    a = torch.zeros(g.n_bus, g.n_bus, dtype=torch.float64, device="cuda")
    f, t = f + 1, t + 1
    for i, j, v in ((f, f, y), (t, t, y), (f, t, -y), (t, f, -y)):
        a.index_put_((i, j), v, accumulate=True)
    return a[1:, 1:].contiguous()


class Dense:
    """A's solve by a dense factor, with one correction: rows of `b` to rows of the result."""

    def __init__(self, a, spd):
        self.a, self.spd = a, spd
        self.factor = torch.linalg.cholesky(a) if spd else torch.linalg.lu_factor(a)

    def once(self, b):
        return torch.cholesky_solve(b, self.factor) if self.spd else torch.linalg.lu_solve(*self.factor, b)

    def __call__(self, rows):
        b = rows.T
        x = self.once(b)
        return (x + self.once(b - self.a @ x)).T.contiguous()


def flows_of(g, theta):
    """(scenarios, branches) flows of angles over the unknowns."""
    f, t, y = branch_ends(g)
    full = torch.nn.functional.pad(theta, (1, 0))
    return y * (full[:, f + 1] - full[:, t + 1])


def exact(case, seed):
    kind = case["kind"]
    if kind == "jacobian":
        p, i, v = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in jacobian(case["buses"]).jacobian.arrays())
        n = p.numel() - 1
        a = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        a[i, torch.repeat_interleave(torch.arange(n, device="cuda"), p.diff())] = v  # CSC
        return Dense(a.T.contiguous() if case["transposed"] else a, False)(jacobian_rhs(case, seed))
    if kind == "complex":
        out = []
        for k, (n, b) in enumerate(zip(complex_buses(case), complex_rhs(case, seed))):
            if n > DENSE_COMPLEX:  # a dense factor of it takes too long
                out.append(None)
                continue
            r, c, v = (torch.from_numpy(x).cuda() for x in admittance(n, k)[2])
            a = torch.zeros(n, n, dtype=torch.complex128, device="cuda").index_put_((r, c), v, accumulate=True)
            out.append(Dense(a, False)(b))
        return out
    g = grid(case["buses"], case["extra"])
    solve = Dense(dense_bprime(g), True)
    f, t, y = branch_ends(g)
    if kind == "solve":
        return solve(right_hand_sides(case, seed))

    def pairs(plus, minus):
        e = torch.zeros(plus.numel(), g.n_bus - 1, dtype=torch.float64, device="cuda")
        rows = torch.arange(plus.numel(), device="cuda")
        for end, value in ((plus, 1.0), (minus, -1.0)):
            keep = end >= 0
            e[rows[keep], end[keep]] += value
        return e

    if kind == "columns":
        ids = torch.from_numpy(column_ids(case, seed)).cuda()
        if case["what"] == "ptdf":
            return flows_of(g, solve(pairs(ids - 1, torch.full_like(ids, -1))))
        h = flows_of(g, solve(pairs(f[ids], t[ids])))
        rows = torch.arange(ids.numel(), device="cuda")
        h = h / (1.0 - h[rows, ids])[:, None]
        h[rows, ids] = -1.0
        h[torch.from_numpy(bridges(case["buses"], case["extra"])).cuda()[ids]] = float("nan")
        return h
    if kind == "n1":
        outaged, ptr, p, weights = outage_inputs(case, seed)
        k = torch.from_numpy(outaged).cuda()
        of = torch.repeat_interleave(torch.arange(k.numel(), device="cuda"), torch.from_numpy(np.diff(ptr)).cuda())
        yk = solve(pairs(f[k], t[k]))
        rows = torch.arange(k.numel(), device="cuda")
        across = flows_of(g, yk)[rows, k] / y[k]          # c'y of each outage
        theta = solve(p[:, 1:])
        out = torch.empty(p.shape[0], dtype=torch.float64, device="cuda")
        w = torch.from_numpy(weights).cuda()
        for lo in range(0, p.shape[0], 2048):
            s = slice(lo, min(lo + 2048, p.shape[0]))
            th, c = theta[s], of[s]
            mine = torch.arange(th.shape[0], device="cuda")
            z = flows_of(g, th)[mine, k[c]] / y[k[c]] / (1.0 / y[k[c]] - across[c])
            fl = flows_of(g, th + z[:, None] * yk[c])
            fl[mine, k[c]] = 0.0
            out[s] = (fl.abs() * w).amax(1)
        return None, out, None, None
    p, limits = adjoint_inputs(case, seed)
    theta = solve(p[:, 1:])
    fl = flows_of(g, theta)
    u = fl.abs() - MARGIN * limits
    soft = torch.nn.functional.softplus(u, threshold=1e9)
    d = 2.0 * soft * torch.sigmoid(u) * fl.sign()       # dL/df
    q = torch.zeros(theta.shape[0], g.n_bus, dtype=torch.float64, device="cuda")
    q.index_add_(1, f + 1, d * y).index_add_(1, t + 1, -d * y)
    lam = solve(q[:, 1:])
    across, back = fl / y, flows_of(g, lam) / y
    return soft.square().sum(), torch.nn.functional.pad(lam, (1, 0)), ((d - back) * across).sum(0)
