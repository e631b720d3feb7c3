"""The spread solve (the automatic choice of the plain solves): counts around a group's 32 and a
block's four groups, factors with and without a top, long chains, many partial sums, Cholesky and
LU, FP32 with one and two right-hand sides per lane, against the oracle at the bars of the other
solves; leading dimensions, two streams at once, and replay under capture."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import random_spd, random_square, right_hand_sides, star_spd, worst_relative_difference
from ybus_b200 import FP32, FP64, CudaError, GpuFactor, configs, grids, host

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
