"""The spread solve's top: its dense map with one correction leaves the residuals that a substitution leaves,
also where the map's condition is large, in every solve that takes it; and a right-hand side that is infinite
gives what the substitution gives."""
import dataclasses

import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import random_spd, random_square, right_hand_sides, star_spd, worst_relative_difference
from ybus_b200 import FP64, GpuFactor, Pair, configs, grids, host

pytestmark = pytest.mark.gpu


def wide_grid(n_bus, extra, seed, decades):
    g = grids.make_grid(n_bus, extra, seed)
    spread = np.random.default_rng(seed).random(g.x.size) - 0.5
    return dataclasses.replace(g, x=g.x * 10.0 ** (decades * spread))


def branch_columns(g, count, seed):
    rng = np.random.default_rng(seed)
    e = rng.integers(0, g.n_branch, count)
    rhs = np.zeros((count, g.n_bus))
    rhs[np.arange(count), g.frm[e]] += 1.0
    rhs[np.arange(count), g.to[e]] -= 1.0
    return rhs[:, 1:], [Pair(int(f) - 1 if f > 0 else None, int(t) - 1 if t > 0 else None) for f, t in zip(g.frm[e], g.to[e])]


def solve(gpu, factor, rhs):
    import torch
    b = torch.from_numpy(np.ascontiguousarray(rhs)).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    factor.solve_many_device(b.data_ptr(), x.data_ptr(), b.shape[0], FP64)
    gpu.synchronize()
    return x.cpu().numpy()


def worst_residual(a, xs, rhs):
    p, i, v = a.to_csr().arrays()
    return max(orc.relative_residual(p, i, v, x, b) for x, b in zip(xs, rhs))


@pytest.mark.parametrize("count", [1, 64, 999, 2100])
@pytest.mark.parametrize("decades", [0, 3])
def test_residuals_on_grids_of_wide_reactances(gpu, decades, count):
    """Four times the substitution's worst over the same columns (its scatter over orders of summation), and the
    project's bar of 1e-12; plain solves and pair solves."""
    g = wide_grid(2000, 700, 11, decades)
    a = configs.bprime(g)
    chol = host.cholesky(a)
    factor = GpuFactor.from_cholesky(gpu, chol)
    assert factor.spread_info(FP64, count)["top"] > 0
    rhs, pairs = branch_columns(g, count, 5)
    some = np.unique(np.r_[np.arange(min(count, 64)), count - 1])
    sub = worst_residual(a, orc.solve_many(chol, rhs[some], threads=8), rhs[some])
    assert worst_residual(a, solve(gpu, factor, rhs)[some], rhs[some]) <= min(1e-12, max(4 * sub, 1e-14))
    factor.set_block_width(count)
    ys = factor.pair_solves(pairs).solutions()
    assert worst_residual(a, ys[some], rhs[some]) <= min(1e-12, max(4 * sub, 1e-14))


@pytest.mark.parametrize("count", [64, 999])
@pytest.mark.parametrize("n_bus,extra,seed,decades", [(2000, 700, 11, 0), (2000, 700, 12, 3), (1500, 520, 13, 3)])
def test_errors_are_a_substitutions(gpu, n_bus, extra, seed, decades, count):
    """The mean over 64 columns of the error against L L' x = b solved in extended precision, at most twice the
    oracle's substitution's: rounding of the same bound, in other orders."""
    g = wide_grid(n_bus, extra, seed, decades)
    chol = host.cholesky(configs.bprime(g))
    rhs, _ = branch_columns(g, count, 5)
    x = solve(gpu, GpuFactor.from_cholesky(gpu, chol), rhs)[:64]
    b = rhs[:64].T[chol.perm].astype(np.longdouble)
    l, lt = chol.l, chol.lt  # the diagonal last, and first
    for k in range(chol.n):
        some = slice(l.ptr[k], l.ptr[k + 1] - 1)
        b[k] = (b[k] - l.val[some].astype(np.longdouble) @ b[l.idx[some]]) / np.longdouble(l.val[l.ptr[k + 1] - 1])
    for k in range(chol.n - 1, -1, -1):
        some = slice(lt.ptr[k] + 1, lt.ptr[k + 1])
        b[k] = (b[k] - lt.val[some].astype(np.longdouble) @ b[lt.idx[some]]) / np.longdouble(lt.val[lt.ptr[k]])
    exact = np.empty_like(b)
    exact[chol.perm] = b
    error = lambda y: float((np.abs(y - exact.T).max(axis=1) / np.abs(exact.T).max(axis=1)).mean())  # noqa: E731
    assert error(x) <= 2 * error(orc.solve_many(chol, rhs[:64], threads=8))


@pytest.mark.parametrize("count", [1, 40, 300])
@pytest.mark.parametrize("name", ["jacobian", "random"])
def test_residuals_of_real_lu_factors(gpu, name, count):
    if name == "jacobian":
        s = configs.jacobian_system(2000, 1, 5)
        a, lu = s.jacobian, s.lu
    else:
        a = random_square(800, 3, 3)
        lu = host.lu(a)
    factor = GpuFactor.from_lu(gpu, lu)
    rhs = np.random.default_rng(count).standard_normal((count, lu.n))
    some = np.arange(0, count, 5)
    sub = worst_residual(a, orc.solve_many(lu, rhs[some], threads=8), rhs[some])
    assert worst_residual(a, solve(gpu, factor, rhs)[some], rhs[some]) <= 2 * sub


@pytest.mark.parametrize("count", [3, 1000])
def test_an_infinite_right_hand_side_gives_what_substitution_gives(gpu, count):
    g = grids.make_grid(1500, 520, 11)
    chol = host.cholesky(configs.bprime(g))
    factor = GpuFactor.from_cholesky(gpu, chol)
    assert factor.spread_info(FP64, count)["top"] > 0
    rhs = np.random.default_rng(2).standard_normal((count, chol.n))
    rhs[1, 700] = np.inf
    rhs[2, 3] = -np.inf
    x = solve(gpu, factor, rhs)
    cpu = orc.solve_many(chol, rhs[:3])
    assert np.isinf(cpu[1:]).all() and np.array_equal(x[1:3], cpu[1:])
    assert np.isfinite(x[0]).all() and np.isfinite(x[3:]).all()


def hub_grid(n_bus, extra, seed, branches):
    """A grid with a hub: a top row of as many partial sums and entries as fill several warps."""
    g = grids.make_grid(n_bus, extra, seed)
    far = np.random.default_rng(seed).choice(np.arange(2, n_bus), branches, replace=False)
    return dataclasses.replace(g, frm=np.r_[g.frm, np.full(branches, 1)], to=np.r_[g.to, far],
                               x=np.r_[g.x, np.full(branches, 0.1)])


@pytest.mark.parametrize("count", [1, 33, 1100])
@pytest.mark.parametrize("name", ["hub", "dense", "dense lu", "half dense", "half dense lu"])
def test_long_rows_and_dense_tops(gpu, name, count):
    """Against the oracle at the bar of the other solves: the sums and the correction of a hub's rows, shared by a
    block's warps, and corrections by dense triangles, orders around a tile's 16 rows and a block's 64."""
    matrices = {"hub": lambda: [configs.bprime(hub_grid(1200, 400, 7, b)) for b in (70, 300)],
                "dense": lambda: [random_spd(n, n, 7) for n in (31, 48, 65, 130)],
                "dense lu": lambda: [random_square(n, n, 3) for n in (31, 48, 65, 130)],
                "half dense": lambda: [random_spd(200, 3, 7)], "half dense lu": lambda: [random_square(120, 3, 3)]}[name]()
    for a in matrices:
        f = host.lu(a) if name.endswith("lu") else host.cholesky(a)
        factor = GpuFactor.from_lu(gpu, f) if name.endswith("lu") else GpuFactor.from_cholesky(gpu, f)
        assert factor.spread_info(FP64, count)["top"] > 0
        rhs = right_hand_sides(f.n, count, 11)
        assert worst_relative_difference(solve(gpu, factor, rhs)[::7], orc.solve_many(f, rhs[::7], threads=8)) < 1e-12


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_value_not_finite_stays_in_its_island_of_a_dense_top(gpu, bad):
    a = random_spd(40, 40, 7)
    p, i, v = a.to_csr().arrays()
    r = np.repeat(np.arange(40), np.diff(p))
    two = host.Matrix.from_triplets(80, 80, np.r_[2 * r, 2 * r + 1], np.r_[2 * i, 2 * i + 1], np.r_[v, v])
    factor = GpuFactor.from_cholesky(gpu, host.cholesky(two))
    assert factor.spread_info(FP64, 40)["top"] > 0
    b = np.random.default_rng(3).standard_normal((40, 80))
    spoiled = b.copy()
    spoiled[20, 10] = bad
    clean, x = solve(gpu, factor, b), solve(gpu, factor, spoiled)
    others = np.arange(40) != 20
    assert np.array_equal(x[others], clean[others]) and not np.isfinite(x[20, 10])
    assert worst_relative_difference(x[[20], 1::2], clean[[20], 1::2]) < 1e-12


@pytest.mark.parametrize("count", [1, 64, 300])
def test_shallow_factors_keep_the_domain_solve(gpu, count):
    """Its bits: a star, and the smallest factor."""
    for a in (star_spd(200), random_spd(2, 1, 7)):
        chol = host.cholesky(a)
        rhs = right_hand_sides(chol.n, count, 5)
        factor, domain = GpuFactor.from_cholesky(gpu, chol), GpuFactor.from_cholesky(gpu, chol)
        domain.set_tile_kind(FP64, 4)
        x = solve(gpu, factor, rhs)
        assert np.array_equal(x, solve(gpu, domain, rhs))
        assert worst_relative_difference(x, orc.solve_many(chol, rhs)) < 1e-12
