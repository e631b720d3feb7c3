"""Factors that admit no spread layout, by their live values or by their top's condition: each solve takes the
ways it had before, alone and in a complex batch beside networks that have a layout."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import right_hand_sides, worst_relative_difference
from test_gpu_complex_passes import PASSES, batch, columns, networks
from test_gpu_spread_top import branch_columns, solve, wide_grid, worst_residual
from ybus_b200 import FP32, FP64, CudaError, GpuFactor, Pair, configs, host

pytestmark = pytest.mark.gpu


def hubs(leaves, some, cplx=False):
    """Leaves that each touch every hub: more rows than a top holds, and more live values than a lane's slots."""
    r, c = (a.ravel() for a in np.meshgrid(np.arange(leaves), leaves + np.arange(some), indexing="ij"))
    d = np.arange(leaves + some)
    v = np.r_[np.where(d < leaves, 2.0 * some, 2.0 * leaves), np.full(2 * r.size, -1.0)]
    return host.Matrix.from_triplets(d.size, d.size, np.r_[d, r, c], np.r_[d, c, r], v * (1 + 0.5j) if cplx else v,
                                     by_rows=not cplx)


def refused(factor, precision=FP64, count=1):
    with pytest.raises(CudaError):
        factor.spread_info(precision, count)


@pytest.mark.parametrize("count", [1, 33, 1600])
def test_a_factor_of_too_many_live_values(gpu, count):
    import torch
    a = hubs(1600, 80)
    chol = host.cholesky(a)
    factor = GpuFactor.from_cholesky(gpu, chol)
    factor.attach_matrix(a)
    for precision in (FP64, FP32):
        refused(factor, precision, count)
    rhs = right_hand_sides(chol.n, count, 5)
    cpu = orc.solve_many(chol, rhs[::7], threads=8)
    assert worst_relative_difference(solve(gpu, factor, rhs)[::7], cpu) < 1e-12
    b = torch.from_numpy(rhs).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_refined_device(b.data_ptr(), x.data_ptr(), count, 4, 1e-10)
    gpu.synchronize()
    assert worst_relative_difference(x.cpu().numpy()[::7], cpu) < 1e-8
    e = np.zeros((1, chol.n))
    e[0, 3], e[0, 900] = 1.0, -1.0
    assert worst_relative_difference(factor.pair_solves([Pair(3, 900)]).solutions(), orc.solve_many(chol, e)) < 1e-12


@pytest.mark.parametrize("count", [1, 300])
def test_a_factor_of_a_large_condition(gpu, count):
    """Four times the substitution's residual, as where the top is taken densely."""
    g = wide_grid(2000, 700, 11, 9)
    a = configs.bprime(g)
    chol = host.cholesky(a)
    factor = GpuFactor.from_cholesky(gpu, chol)
    refused(factor, FP64, count)
    rhs, _ = branch_columns(g, count, 5)
    some = np.arange(0, count, 9)
    sub = worst_residual(a, orc.solve_many(chol, rhs[some], threads=8), rhs[some])
    assert worst_residual(a, solve(gpu, factor, rhs)[some], rhs[some]) <= 4 * sub


def test_a_complex_batch_with_one_refused(gpu):
    a = hubs(1600, 120, cplx=True)
    lu = host.lu(a, host.COLAMD)
    own = GpuFactor.from_lu_complex(gpu, lu)
    own.attach_matrix_complex(a)
    (lu2, f2), (lu3, f3) = networks(gpu, (700, 300), 41)
    lus, factors = (lu2, lu, lu3), [f2, own, f3]
    rhs = [columns(l.n, c, 3) for l, c in zip(lus, (40, 33, 64))]
    cpu = [orc.solve_many_lu(l, b) for l, b in zip(lus, rhs)]
    for prec, bar in ((FP64, 1e-12), (FP32, 1e-8)):
        runs = [batch(gpu, factors, rhs, prec, max_steps=3)[0] for _ in range(PASSES)]
        for xs in runs:
            for x, c in zip(xs, cpu):
                assert worst_relative_difference(x, c) < bar
        if prec == FP64:  # by tiles in every pass, the others by the spread solve in the last
            assert np.array_equal(runs[0][1], runs[-1][1]) and not np.array_equal(runs[0][0], runs[-1][0])
