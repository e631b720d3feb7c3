"""Captured solves and several streams: a graph that holds a solve keeps giving the oracle's solutions
whatever is solved between its replays and beside them, for any count once the factor has solved
something, and gives its working arrays back when it is destroyed."""
import threading
import time

import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import right_hand_sides, worst_relative_difference
from ybus_b200 import FP32, FP64, GpuFactor, configs, grids, host, solve_batch_complex

pytestmark = pytest.mark.gpu

BARS = {FP64: 1e-12, FP32: 1e-4}


@pytest.fixture(scope="module")
def grid():
    a = configs.bprime(grids.make_grid(1500, 520, 11))
    return a, host.cholesky(a)


def columns(n, count, seed):
    import torch
    return torch.from_numpy(right_hand_sides(n, count, seed)).cuda()


def capture(stream, enqueue):
    import torch
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        enqueue()
    return graph


def agrees(x, chol, rhs, bar):
    return worst_relative_difference(x.cpu().numpy(), orc.solve_many(chol, rhs.cpu().numpy(), threads=8)) < bar


@pytest.mark.parametrize("prec", [FP64, FP32])
def test_a_captured_solve_outlives_larger_and_smaller_ones(gpu, grid, prec):
    """On the captured stream, which the workspaces are kept by: 5,000 columns need a larger work array, one
    column a layout with more partial sums."""
    import torch
    chol = grid[1]
    factor = GpuFactor.from_cholesky(gpu, chol)
    stream = torch.cuda.Stream()
    b, x = columns(chol.n, 96, 5), torch.zeros(96, chol.n, dtype=torch.float64, device="cuda")
    many, out = columns(chol.n, 5000, 7), torch.zeros(5000, chol.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 96, prec, stream.cuda_stream)
    graph = capture(stream, lambda: factor.solve_many_device(b.data_ptr(), x.data_ptr(), 96, prec, stream.cuda_stream))
    for seed, count in ((8, 5000), (9, 1), (10, 1500), (11, 33)):
        factor.solve_many_device(many.data_ptr(), out.data_ptr(), count, prec, stream.cuda_stream)
        b.copy_(columns(chol.n, 96, seed))
        x.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert agrees(x, chol, b, BARS[prec])


def test_replays_beside_eager_solves_on_other_streams(gpu, grid):
    import torch
    chol = grid[1]
    factor = GpuFactor.from_cholesky(gpu, chol)
    capturing, other = torch.cuda.Stream(), torch.cuda.Stream()
    b, c = columns(chol.n, 300, 5), columns(chol.n, 280, 6)
    x, y = torch.zeros_like(b), torch.zeros_like(c)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 300, FP64, capturing.cuda_stream)
    factor.solve_many_device(c.data_ptr(), y.data_ptr(), 280, FP64, other.cuda_stream)
    graph = capture(capturing, lambda: factor.solve_many_device(b.data_ptr(), x.data_ptr(), 300, FP64,
                                                                capturing.cuda_stream))
    alone_x, alone_y = x.clone(), y.clone()
    x.zero_(), y.zero_()
    torch.cuda.synchronize()
    for _ in range(30):
        graph.replay()  # on the current stream
        factor.solve_many_device(c.data_ptr(), y.data_ptr(), 280, FP64, other.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(x, alone_x) and torch.equal(y, alone_y)
    assert agrees(x, chol, b, BARS[FP64])


def test_any_count_can_be_captured_and_two_in_one_graph(gpu, grid):
    import torch
    chol = grid[1]
    factor = GpuFactor.from_cholesky(gpu, chol)
    stream = torch.cuda.Stream()
    b = columns(chol.n, 2600, 5)
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 1, FP64, stream.cuda_stream)
    row = 8 * chol.n

    def both():
        factor.solve_many_device(b.data_ptr(), x.data_ptr(), 600, FP64, stream.cuda_stream)
        factor.solve_many_device(b.data_ptr() + 600 * row, x.data_ptr() + 600 * row, 2000, FP64, stream.cuda_stream)

    graph = capture(stream, both)
    for seed in (6, 7):
        b.copy_(columns(chol.n, 2600, seed))
        x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert agrees(x[::37], chol, b[::37], BARS[FP64])


def test_a_destroyed_graph_gives_its_arrays_back(gpu, grid):
    import torch
    chol = grid[1]
    factor = GpuFactor.from_cholesky(gpu, chol)
    stream = torch.cuda.Stream()
    b = columns(chol.n, 3000, 5)
    x = torch.zeros_like(b)

    def solve():
        factor.solve_many_device(b.data_ptr(), x.data_ptr(), 3000, FP64, stream.cuda_stream)

    torch.cuda.synchronize()
    solve()
    for _ in range(2):  # the first makes what torch keeps for its graphs
        graph = capture(stream, solve)
        graph.replay()
        torch.cuda.synchronize()
        held = torch.cuda.mem_get_info()[0]
        del graph
        for _ in range(100):  # the driver tells of a graph's end from a thread of its own
            solve()
            torch.cuda.synchronize()
            back = torch.cuda.mem_get_info()[0] - held
            if back > 0:
                break
            time.sleep(0.1)
    assert back >= 8 * 3000 * chol.n, back


def refined(factor, b, x, count, stream, ratio=None):
    factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), count, 4, 1e-10,
                                     None if ratio is None else ratio.data_ptr(), stream=stream.cuda_stream)


@pytest.mark.parametrize("kind", [None, 4, 5], ids=["spread", "domain", "lane"])
def test_a_captured_refined_solve_outlives_larger_ones(gpu, grid, kind):
    """More columns than the solve that ran before it, and larger ones between its replays."""
    import torch
    a, chol = grid
    factor = GpuFactor.from_cholesky(gpu, chol)
    factor.attach_matrix(a)
    if kind is not None:
        factor.set_tile_kind(FP32, kind)
    stream = torch.cuda.Stream()
    b, x = columns(chol.n, 96, 5), torch.zeros(96, chol.n, dtype=torch.float64, device="cuda")
    many, out = columns(chol.n, 5000, 7), torch.zeros(5000, chol.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    refined(factor, many, out, 40, stream)
    graph = capture(stream, lambda: refined(factor, b, x, 96, stream))
    for seed, count in ((8, 5000), (9, 1)):
        refined(factor, many, out, count, stream)
        b.copy_(columns(chol.n, 96, seed))
        x.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert agrees(x, chol, b, 1e-8)


@pytest.mark.parametrize("kind", [None, 4], ids=["spread", "domain"])
def test_refined_solves_on_several_streams_at_once(gpu, grid, kind):
    import torch
    a, chol = grid
    factor = GpuFactor.from_cholesky(gpu, chol)
    factor.attach_matrix(a)
    if kind is not None:
        factor.set_tile_kind(FP32, kind)
    streams = [torch.cuda.Stream() for _ in range(6)]
    bs = [columns(chol.n, 700 - 60 * k, k + 1) for k in range(6)]
    xs = [torch.zeros_like(b) for b in bs]
    ratios = [torch.zeros(b.shape[0], dtype=torch.float64, device="cuda") for b in bs]
    torch.cuda.synchronize()
    alone = []
    for b, x, r in zip(bs, xs, ratios):
        refined(factor, b, x, b.shape[0], streams[0], r)
        torch.cuda.synchronize()
        alone.append((x.clone(), r.clone()))
    torch.cuda.synchronize()
    for _ in range(10):
        for b, x, s, r in zip(bs, xs, streams, ratios):
            refined(factor, b, x, b.shape[0], s, r)
    torch.cuda.synchronize()
    for x, r, (xa, ra) in zip(xs, ratios, alone):
        assert torch.equal(x, xa) and torch.equal(r, ra)


def complex_batch(gpu, sizes, counts, seed):
    import torch
    lus, factors, bs = [], [], []
    rng = np.random.default_rng(seed)
    for k, (n, count) in enumerate(zip(sizes, counts)):
        r, c, v = grids.ybus_triplets(grids.make_complex_grid(n, grids.SEED_BASE + 70 + seed + k))
        lus.append(host.lu(host.Matrix.from_triplets(n, n, r, c, v, by_rows=False), host.COLAMD))
        factors.append(GpuFactor.from_lu_complex(gpu, lus[-1]))
        bs.append(torch.from_numpy(rng.standard_normal((count, 2 * n))).cuda())
    return lus, factors, bs


@pytest.mark.parametrize("threads", [False, True], ids=["one thread", "threads"])
def test_complex_batches_on_two_streams_at_once(gpu, threads):
    """Other networks and counts on each stream, the lists of blocks among what a batch uploads."""
    import torch
    batches = [complex_batch(gpu, (900, 400), (70, 129), 1), complex_batch(gpu, (300, 700, 500), (64, 33, 260), 9)]
    streams = [torch.cuda.Stream() for _ in batches]
    xs = [[torch.zeros_like(b) for b in bs] for _, _, bs in batches]
    torch.cuda.synchronize()

    def solve(k):
        _, factors, bs = batches[k]
        solve_batch_complex(factors, [b.data_ptr() for b in bs], [x.data_ptr() for x in xs[k]],
                            [b.shape[0] for b in bs], FP64, stream=streams[k].cuda_stream)

    for k in range(2):
        for _ in range(8):
            solve(k)
    torch.cuda.synchronize()
    alone = [[x.clone() for x in some] for some in xs]
    torch.cuda.synchronize()
    if threads:
        work = [threading.Thread(target=lambda k=k: [solve(k) for _ in range(20)]) for k in range(2)]
        for t in work:
            t.start()
        for t in work:
            t.join()
    else:
        for _ in range(20):
            solve(0), solve(1)
    torch.cuda.synchronize()
    for some, was, (lus, _, bs) in zip(xs, alone, batches):
        for x, a, lu, b in zip(some, was, lus, bs):
            assert torch.equal(x, a)
            cpu = orc.solve_many_lu(lu, b[::9].cpu().numpy().view(np.complex128))
            assert worst_relative_difference(x[::9].cpu().numpy().view(np.complex128), cpu) < 1e-12
