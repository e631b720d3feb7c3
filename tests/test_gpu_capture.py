"""Captured solves and several streams: a graph that holds a solve keeps giving the oracle's solutions
whatever is solved between its replays and beside them, for any count once the factor has solved
something, and gives its working arrays back when it is destroyed."""
import time

import pytest

import oracle.oracle as orc
from fixtures import right_hand_sides, worst_relative_difference
from ybus_b200 import FP32, FP64, GpuFactor, configs, grids, host

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
