"""The memory a solve takes: a work array for the right-hand sides asked for, and runs of at most the GPU's
work limit, down to the solves that need none; every route to the oracle's solutions."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import right_hand_sides, worst_relative_difference
from test_gpu_complex_passes import batch, columns, networks
from ybus_b200 import FP32, FP64, CudaError, Gpu, GpuFactor, configs, grids, host
from ybus_b200.dc import DcNetwork

pytestmark = pytest.mark.gpu

GROUP = 32 * 1499 * 8  # bytes of a group of 32 FP64 columns of the grid below


@pytest.fixture(scope="module")
def grid():
    a = configs.bprime(grids.make_grid(1500, 520, 11))
    return a, host.cholesky(a)


def test_one_column_takes_the_memory_of_one_group(gpu):
    import torch
    chol = host.cholesky(configs.bprime(configs.grid_10k()))
    factor = GpuFactor.from_cholesky(gpu, chol)
    b = torch.from_numpy(right_hand_sides(chol.n, 1, 5)).cuda()
    x = torch.zeros_like(b)
    factor.spread_info(FP64, 1)  # the layout
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 1, FP64)
    gpu.synchronize()
    # a group's work array is 2.6 MB and its partial sums are of the top's 700 rows and a few a domain
    assert before - torch.cuda.mem_get_info()[0] <= 16 << 20
    assert worst_relative_difference(x.cpu().numpy(), orc.solve_many(chol, b.cpu().numpy())) < 1e-12


@pytest.mark.parametrize("groups", [0, 1, 2, 7])
def test_plain_solves_in_runs(grid, groups):
    """Several runs, one of them ragged; without room for a group, the other solves."""
    import torch
    own = Gpu.new()
    own.set_work_bytes(groups * GROUP)
    chol = grid[1]
    factor = GpuFactor.from_cholesky(own, chol)
    for count in (1, 32, 33, 300, 2113):
        b = torch.from_numpy(right_hand_sides(chol.n, count, count)).cuda()
        cpu = orc.solve_many(chol, b.cpu().numpy()[::7], threads=8)
        for prec, bar in ((FP64, 1e-12), (FP32, 1e-4)):
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            factor.solve_many_device(b.data_ptr(), x.data_ptr(), count, prec)
            own.synchronize()
            assert worst_relative_difference(x.cpu().numpy()[::7], cpu) < bar
        torch.cuda.synchronize()
        factor.solve_many_device(b.data_ptr(), b.data_ptr(), count, FP64)  # in place
        own.synchronize()
        assert worst_relative_difference(b.cpu().numpy()[::7], cpu) < 1e-12


@pytest.mark.parametrize("groups", [0, 3])
def test_refined_solves_and_screening_in_runs(grid, groups):
    import torch
    a, chol = grid
    own = Gpu.new()
    own.set_work_bytes(groups * GROUP)
    factor = GpuFactor.from_cholesky(own, chol)
    factor.attach_matrix(a)
    b = torch.from_numpy(right_hand_sides(chol.n, 500, 5)).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), 500, 4, 1e-10)
    own.synchronize()
    assert worst_relative_difference(x.cpu().numpy(), orc.solve_many(chol, b.cpu().numpy(), threads=8)) < 1e-8
    g = grids.make_grid(1500, 520, 11)
    results = []
    for some in (own, Gpu.new()):
        net = DcNetwork.from_grid(some, g)
        outaged = np.flatnonzero(~net.bridges())[:30]
        sp = np.arange(31) * 10
        inj = np.random.default_rng(3).normal(0.0, 0.1, (300, g.n_bus))
        results.append(net.outage_loadings_batch(outaged, sp, inj))
    assert np.allclose(results[0][1], results[1][1], rtol=1e-10, atol=0.0) and np.array_equal(results[0][3], results[1][3])


@pytest.mark.parametrize("limit", [0, 1 << 20, 3 << 20, 9 << 20])
def test_complex_batches_in_runs(limit):
    """Runs that end inside a network and between two, some networks above the limit (by tiles, beside the
    others), corrections added once each."""
    import torch
    own = Gpu.new()
    nets = networks(own, (1500, 300, 4000, 700), 5)
    lus, factors = zip(*nets)
    rhs = [columns(lu.n, c, 6) for lu, c in zip(lus, (129, 64, 70, 1))]
    cpu = [orc.solve_many_lu(lu, b) for lu, b in zip(lus, rhs)]
    ratios = [torch.zeros(len(b), dtype=torch.float64, device="cuda") for b in rhs]
    for prec, bar in ((FP64, 1e-12), (FP32, 1e-8)):
        for _ in range(5):
            batch(own, list(factors), rhs, prec, max_steps=3, ratios=ratios)
        own.set_work_bytes(limit)
        xs, _ = batch(own, list(factors), rhs, prec, max_steps=3, ratios=ratios)
        own.set_work_bytes(2 << 30)
        for x, c in zip(xs, cpu):
            assert worst_relative_difference(x, c) < bar
        assert prec == FP64 or max(float(r.max()) for r in ratios) <= 1e-10


def test_the_limit_is_checked(gpu):
    with pytest.raises(CudaError):
        gpu.set_work_bytes(-1)
