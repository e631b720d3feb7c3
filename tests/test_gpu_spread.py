"""The spread solve (the automatic choice of the plain solves): counts around a group's 32 and a
block's four groups, factors with and without a top, long chains, many partial sums, Cholesky and
LU, FP32 with one and two right-hand sides per lane, batches of complex LU, against the oracle at
the bars of the other solves; leading dimensions, two streams at once, and replay under capture."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import random_spd, random_square, right_hand_sides, star_spd, worst_relative_difference
from ybus_b200 import FP32, FP64, CudaError, GpuFactor, Pair, PairUpdate, configs, grids, host, solve_batch_complex
from ybus_b200.dc import DcNetwork, FlowLoss

pytestmark = pytest.mark.gpu

BARS = ((FP64, 1e-12), (FP32, 1e-4))


def path(n):
    """A path graph's matrix: one chain, rows of one entry."""
    k = np.arange(n - 1)
    r = np.concatenate([np.arange(n), k, k + 1])
    c = np.concatenate([np.arange(n), k + 1, k])
    v = np.concatenate([np.full(n, 2.5), np.full(2 * n - 2, -1.0)])
    return host.Matrix.from_triplets(n, n, r, c, v)


FACTORS = {
    "two": lambda: host.cholesky(random_spd(2, 1, 7)),
    "three": lambda: host.cholesky(random_spd(3, 1, 7)),
    "path": lambda: host.cholesky(path(997)),
    "sparse": lambda: host.cholesky(random_spd(200, 3, 7)),
    "dense": lambda: host.cholesky(random_spd(60, 60, 7)),
    "star": lambda: host.cholesky(star_spd(200)),
    "grid": lambda: host.cholesky(configs.bprime(grids.make_grid(1500, 520, 11))),
    "lu": lambda: host.lu(random_square(120, 3, 3)),
    "jacobian": lambda: configs.jacobian_system(400, 1, 5).lu,
}


def upload(gpu, f):
    return GpuFactor.from_lu(gpu, f) if isinstance(f, host.HostLu) else GpuFactor.from_cholesky(gpu, f)


def solve(gpu, factor, rhs, prec, ldb=0, ldx=0, stream=None):
    import torch
    n = rhs.shape[1]
    b = torch.full((rhs.shape[0], n + ldb), 3.0, dtype=torch.float64, device="cuda")
    b[:, :n] = torch.from_numpy(rhs).cuda()
    x = torch.full((rhs.shape[0], n + ldx), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), rhs.shape[0], prec, stream, ldb=n + ldb, ldx=n + ldx)
    gpu.synchronize(stream)
    x = x.cpu().numpy()
    assert np.all(x[:, n:] == 7.0), "rows past n are not written"
    return x[:, :n]


@pytest.mark.parametrize("name", sorted(FACTORS))
def test_spread_solve_matches_the_cpu(gpu, name):
    f = FACTORS[name]()
    factor = upload(gpu, f)
    for count in (1, 31, 32, 33, 128, 129, 300, 2048, 2113):
        info = factor.spread_info(FP64, count)
        assert info["slots"] <= 64 and info["top"] <= f.n
        rhs = right_hand_sides(f.n, count, 11)
        sample = np.unique(np.r_[0, count // 2, count - 1, np.arange(0, count, 37)])
        cpu = orc.solve_many(f, rhs[sample], threads=8)
        for prec, bar in BARS:
            d = worst_relative_difference(solve(gpu, factor, rhs, prec, ldb=3, ldx=5)[sample], cpu)
            assert d < bar, f"{name} count {count} precision {prec}: {d:e}"


def test_a_shape_or_threshold_takes_the_automatic_choice_to_the_other_solves(gpu):
    chol = FACTORS["grid"]()
    factor = upload(gpu, chol)
    rhs = right_hand_sides(chol.n, 40, 3)
    first = solve(gpu, factor, rhs, FP64)
    factor.set_lane_min_count(FP64, 1)
    with pytest.raises(CudaError):
        factor.spread_info(FP64, 40)
    assert worst_relative_difference(solve(gpu, factor, rhs, FP64), first) < 1e-12


def test_repeats_and_two_streams_at_once_give_the_same_bits(gpu):
    import torch
    chol = FACTORS["grid"]()
    factor = upload(gpu, chol)
    streams = [torch.cuda.Stream() for _ in range(6)]  # more than the workspaces a factor keeps
    bs = [torch.from_numpy(right_hand_sides(chol.n, 700 - 60 * k, k + 1)).cuda() for k in range(6)]
    alone = [torch.from_numpy(solve(gpu, factor, b.cpu().numpy(), FP64)).cuda() for b in bs]
    xs = [torch.zeros_like(b) for b in bs]
    torch.cuda.synchronize()
    for _ in range(20):
        for b, x, s in zip(bs, xs, streams):
            factor.solve_many_device(b.data_ptr(), x.data_ptr(), b.shape[0], FP64, s.cuda_stream)
    torch.cuda.synchronize()
    for x, a in zip(xs, alone):
        assert torch.equal(x, a)


def test_a_solve_that_has_run_can_be_captured(gpu):
    import torch
    chol = FACTORS["grid"]()
    factor = upload(gpu, chol)
    stream = torch.cuda.Stream()
    b = torch.from_numpy(right_hand_sides(chol.n, 96, 5)).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 1, FP64, stream.cuda_stream)  # another count
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        factor.solve_many_device(b.data_ptr(), x.data_ptr(), 96, FP64, stream.cuda_stream)
    for seed in (6, 7):
        rhs = right_hand_sides(chol.n, 96, seed)
        b.copy_(torch.from_numpy(rhs))
        graph.replay()
        torch.cuda.synchronize()
        assert worst_relative_difference(x.cpu().numpy(), orc.solve_many(chol, rhs, threads=8)) < 1e-12


def complex_lu(r, c, v):
    a = host.Matrix.from_triplets(max(r) + 1, max(r) + 1, r, c, v, by_rows=False)
    return a, host.lu(a, host.COLAMD)


def complex_two():
    return complex_lu([0, 1, 0, 1], [0, 1, 1, 0], [4 + 1j, 3 - 2j, 1j, 0.5])


def complex_path(n):
    k = list(range(n - 1))
    return complex_lu(list(range(n)) + k + [i + 1 for i in k], list(range(n)) + [i + 1 for i in k] + k,
                      [2.5 + 0.5j] * n + [-1 + 0.25j] * (n - 1) + [-1 - 0.5j] * (n - 1))


def complex_dense(n):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3 * n * np.eye(n)
    r, c = np.indices((n, n)).reshape(2, -1)
    return complex_lu(r.tolist(), c.tolist(), v.ravel())


def complex_star(n):
    """One column of n entries: more pairs of a row than one packet of the sweeps holds."""
    k = list(range(1, n))
    return complex_lu([0] + k + k + [0] * (n - 1), [0] + k + [0] * (n - 1) + k,
                      [3.0 * n] + [2 + 1j] * (n - 1) + [-1j] * (n - 1) + [1 + 0j] * (n - 1))


@pytest.mark.parametrize("prec,bar", BARS)
@pytest.mark.parametrize("counts", [(1, 32, 33, 129), (0, 31, 300, 2), (64, 0, 1, 0)])
def test_a_complex_batch_matches_the_cpu(gpu, counts, prec, bar):
    """Every second network's arrays lie on an 8-byte boundary that is no 16-byte one; x after its
    last value is not written. Without corrections FP32 is complex64."""
    import torch
    lus, factors = [], []
    for a, lu in (complex_two(), complex_path(997), complex_dense(60), complex_star(300)):
        lus.append(lu)
        factors.append(GpuFactor.from_lu_complex(gpu, lu))
        factors[-1].attach_matrix_complex(a)
    rng = np.random.default_rng(5)
    rhs = [rng.standard_normal((c, lu.n)) + 1j * rng.standard_normal((c, lu.n)) for lu, c in zip(lus, counts)]
    for shift in (0, 1):
        bs, xs = [], []
        for i, b in enumerate(rhs):
            off = shift * (i % 2)
            t = torch.zeros(2 * b.size + 4, dtype=torch.float64)
            t[off:off + 2 * b.size] = torch.from_numpy(b.view(np.float64).ravel().copy())
            bs.append((t.cuda(), off))
            xs.append((torch.full((2 * b.size + 4,), 7.0, dtype=torch.float64, device="cuda"), off))
        torch.cuda.synchronize()
        solve_batch_complex(factors, [t.data_ptr() + 8 * o for t, o in bs], [t.data_ptr() + 8 * o for t, o in xs],
                            counts, prec, max_steps=0)
        gpu.synchronize()
        for lu, b, (t, off) in zip(lus, rhs, xs):
            x = t.cpu().numpy()
            assert np.all(x[:off] == 7.0) and np.all(x[off + 2 * b.size:] == 7.0)
            if len(b):
                sol = x[off:off + 2 * b.size].view(np.complex128).reshape(b.shape)
                assert worst_relative_difference(sol, orc.solve_many_lu(lu, b)) < bar


DOMAIN = 4


@pytest.mark.parametrize("kind", [None, DOMAIN], ids=["spread", "domain"])
@pytest.mark.parametrize("count", [1, 31, 33, 300])
@pytest.mark.parametrize("name", ["grid", "lu"])
def test_refined_solve(gpu, name, count, kind):
    """Leading dimensions, and x in b's place (the automatic choice leaves that to the domain solve)."""
    import torch
    if name == "grid":
        a = configs.bprime(grids.make_grid(1500, 520, 11))
    else:
        a = random_square(120, 3, 3)
    f = host.cholesky(a) if name == "grid" else host.lu(a)
    factor = upload(gpu, f)
    factor.attach_matrix(a)
    if kind is not None:
        factor.set_tile_kind(FP32, kind)
    n = f.n
    rhs = right_hand_sides(n, count, 11)
    cpu = orc.solve_many(f, rhs, threads=8)
    p, i, v = a.to_csr().arrays()
    for inplace in (False, True):
        b = torch.full((count, n + 3), 3.0, dtype=torch.float64, device="cuda")
        b[:, :n] = torch.from_numpy(rhs).cuda()
        x = b if inplace else torch.full((count, n + 5), 7.0, dtype=torch.float64, device="cuda")
        ratio = torch.empty(count, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), count, 4, 1e-10, ratio.data_ptr(),
                                         ldb=n + 3, ldx=x.shape[1])
        gpu.synchronize()
        xs = x.cpu().numpy()
        assert np.all(xs[:, n:] == (3.0 if inplace else 7.0)), "rows past n are not written"
        assert worst_relative_difference(xs[:, :n], cpu) < 1e-8
        assert max(orc.relative_residual(p, i, v, xs[k, :n], rhs[k]) for k in range(0, count, 7)) <= 1.05e-10
        assert ratio.cpu().numpy().max() <= 1e-10


@pytest.mark.parametrize("count", [1, 31, 33, 300])
@pytest.mark.parametrize("name", ["two", "path", "star", "grid"])
def test_pairs_and_their_updates(gpu, name, count):
    """Pairs with one end, both or none, against the CPU, and the updates bit for bit from them."""
    f = FACTORS[name]()
    factor = upload(gpu, f)
    factor.set_block_width(300)
    rng = np.random.default_rng(count)
    plus, minus = rng.integers(-1, f.n, count), rng.integers(-1, f.n, count)
    minus[minus == plus] = -1
    pairs = [Pair(None if p < 0 else int(p), None if m < 0 else int(m)) for p, m in zip(plus, minus)]
    rhs = np.zeros((count, f.n))
    for k in range(count):
        if plus[k] >= 0:
            rhs[k, plus[k]] = 1.0
        if minus[k] >= 0:
            rhs[k, minus[k]] = -1.0
    ys = factor.pair_solves(pairs).solutions()
    cpu = orc.solve_many(f, rhs, threads=8)
    some = np.abs(cpu).max(axis=1) > 0
    assert worst_relative_difference(ys[some], cpu[some]) < 1e-12 and not ys[~some].any()
    base, alpha, weight = rng.standard_normal(f.n), rng.standard_normal(count), 2.0 + rng.random(count)
    out = factor.pair_updates(base, [PairUpdate(q, a, w) for q, a, w in zip(pairs, alpha, weight)]).solutions()
    for k in range(0, count, 7):
        exact, _ = orc.pair_update(base, ys[k], pairs[k].plus, pairs[k].minus, alpha[k], weight[k])
        assert np.array_equal(out[k], exact)


@pytest.mark.parametrize("slack", [0, 7, 299])
@pytest.mark.parametrize("count", [1, 7, 33])
def test_adjoint_of_any_slack(gpu, slack, count):
    g = grids.make_grid(300, 100, 3)
    rng = np.random.default_rng(count)
    p, limits = rng.normal(0.0, 0.1, (count, g.n_bus)), rng.uniform(0.5, 2.0, g.n_branch)
    net = DcNetwork.from_grid(gpu, g, slack)
    loss_fn = FlowLoss(net, count)
    loss = loss_fn.forward(p, limits)
    gp, gb = loss_fn.backward()
    r, c, v = grids.bbus_triplets(g)
    keep = np.delete(np.arange(g.n_bus), slack)
    chol = host.cholesky(host.Matrix.from_triplets(g.n_bus, g.n_bus, r, c, v).select(keep, keep))
    position = -np.ones(g.n_bus, np.int64)
    position[keep] = np.arange(keep.size)
    loss_c, gp_c, gb_c = orc.flow_loss_and_gradient(chol, g.n_bus, g.frm, g.to, 1.0 / g.x, position, p, limits)
    assert abs(loss - loss_c) <= 1e-12 * abs(loss_c)
    assert np.abs(gp - gp_c).max() <= 1e-10 * np.abs(gp_c).max()
    assert np.abs(gb - gb_c).max() <= 1e-10 * np.abs(gb_c).max()
    assert (gp[:, slack] == 0.0).all()


@pytest.mark.parametrize("name", ["cholesky", "lu", "complex"])
@pytest.mark.parametrize("count", [1, 40, 2100])
def test_a_value_not_finite_stays_in_its_island_and_column(gpu, name, count):
    """Two networks without a coupling in one factor; the second's solutions and the other columns' come out
    as without the spoiled entry."""
    import torch
    n = 700
    k = np.arange(n)
    j = (k // 2 * 2 + 37 * (1 + k % 5)) % n  # neighbours of a parity: even rows and odd rows are islands
    j = np.where((j + k) % 2 == 0, j, (j + 1) % n)
    r, c = np.r_[k, k, j], np.r_[k, j, k]
    keep = r != c
    keep[:n] = True
    w = 1.0 + (k % 7) / 7.0
    v = np.r_[np.full(n, 30.0), -w, -w][keep]
    r, c = r[keep], c[keep]
    rng = np.random.default_rng(count)
    b = rng.standard_normal((count, n))
    spoiled = b.copy()
    spoiled[count // 2, 10] = np.nan
    if name == "complex":
        a = host.Matrix.from_triplets(n, n, r, c, v * (1 + 0.25j), by_rows=False)
        factor = GpuFactor.from_lu_complex(gpu, host.lu(a, host.COLAMD))
        xs = []
        for rhs in (b, spoiled):
            t = torch.from_numpy(rhs.astype(np.complex128).view(np.float64).copy()).cuda()
            x = torch.empty_like(t)
            torch.cuda.synchronize()
            solve_batch_complex([factor], [t.data_ptr()], [x.data_ptr()], [count], FP64)
            gpu.synchronize()
            xs.append(x.cpu().numpy().view(np.complex128))
    else:
        a = host.Matrix.from_triplets(n, n, r, c, v, by_rows=name == "cholesky")
        factor = upload(gpu, host.cholesky(a) if name == "cholesky" else host.lu(a))
        xs = [solve(gpu, factor, rhs, FP64) for rhs in (b, spoiled)]
    clean, x = xs
    others = np.arange(count) != count // 2
    assert np.array_equal(x[others], clean[others])
    assert np.isnan(x[count // 2, 10])
    assert worst_relative_difference(x[[count // 2], 1::2], clean[[count // 2], 1::2]) < 1e-12


def test_a_refined_solve_that_has_run_can_be_captured(gpu):
    """Beside a plain FP32 layout of the captured size, which holds no matrix."""
    import torch
    a = configs.bprime(grids.make_grid(1500, 520, 11))
    chol = host.cholesky(a)
    factor = GpuFactor.from_cholesky(gpu, chol)
    factor.attach_matrix(a)
    stream = torch.cuda.Stream()
    b = torch.from_numpy(right_hand_sides(chol.n, 300, 5)).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 64, FP32, stream.cuda_stream)
    factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), 300, 4, 1e-10, stream=stream.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), 64, 4, 1e-10, stream=stream.cuda_stream)
    rhs = right_hand_sides(chol.n, 64, 6)
    b[:64].copy_(torch.from_numpy(rhs))
    x.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert worst_relative_difference(x[:64].cpu().numpy(), orc.solve_many(chol, rhs, threads=8)) < 1e-8
