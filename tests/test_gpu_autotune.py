"""The autotuner leaves a factor on the fastest solve there is: on the spread solve where that is faster than
every shape of the others, which stay for the solves that do not take it."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import right_hand_sides, worst_relative_difference
from ybus_b200 import FP32, FP64, CudaError, GpuFactor, configs, grids, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,bar", [(FP64, 1e-12), (FP32, 1e-4)])
def test_the_spread_solve_stays_where_it_is_faster(gpu, prec, bar):
    import torch
    chol = host.cholesky(configs.bprime(grids.make_grid(2000, 700, grids.SEED_BASE + 1)))
    factor = GpuFactor.from_cholesky(gpu, chol)
    b = torch.from_numpy(right_hand_sides(chol.n, 999, 5)).cuda()
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), 999, prec)  # more than twice as fast as the others
    for _ in range(2):  # again from what it left
        best = factor.autotune(prec, 999)
        assert best["kind"] in (2, 4, 5) and best["ms"] > 0
        assert factor.spread_info(prec, 999)["tasks"] > 1
    factor.solve_many_device(b.data_ptr(), y.data_ptr(), 999, prec)
    gpu.synchronize()
    assert torch.equal(x, y)
    assert worst_relative_difference(y.cpu().numpy()[::7], orc.solve_many(chol, b.cpu().numpy()[::7], threads=8)) < bar
    factor.set_tile_kind(prec, best["kind"])
    with pytest.raises(CudaError):
        factor.spread_info(prec, 999)


def test_a_set_shape_keeps_the_spread_solve_out(gpu):
    chol = host.cholesky(configs.bprime(grids.make_grid(600, 200, 3)))
    factor = GpuFactor.from_cholesky(gpu, chol)
    factor.set_lane_min_count(FP64, 100)
    factor.autotune(FP64, 64)
    with pytest.raises(CudaError):
        factor.spread_info(FP64, 64)
    rhs = np.random.default_rng(3).standard_normal((64, chol.n))
    assert worst_relative_difference(factor.solve_many(rhs), orc.solve_many(chol, rhs)) < 1e-12
