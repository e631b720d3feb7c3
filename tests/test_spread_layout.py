"""The spread solve's layout, checked on the CPU: the packets the layout builder makes, executed by a host
interpreter of the kernel's semantics, solve chains, stars, dense and sparse matrices, the synthetic grids
and pivoted LU factors, real and complex, to the oracle's solutions, with and without a top (no GPU)."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import random_spd, random_square, right_hand_sides, star_spd, worst_relative_difference
from spread_interp import run
from ybus_b200 import YbError, _lib, configs, grids, host


def path(n):
    k = np.arange(n - 1)
    r = np.concatenate([np.arange(n), k, k + 1])
    c = np.concatenate([np.arange(n), k + 1, k])
    v = np.concatenate([np.full(n, 2.5), np.full(2 * n - 2, -1.0)])
    return host.Matrix.from_triplets(n, n, r, c, v)


def islands(n):
    """Even rows and odd rows without a coupling."""
    k = np.arange(n - 2)
    r = np.concatenate([np.arange(n), k, k + 2])
    c = np.concatenate([np.arange(n), k + 2, k])
    v = np.concatenate([np.full(n, 3.0), np.full(2 * n - 4, -1.0)])
    return host.Matrix.from_triplets(n, n, r, c, v)


def complex_ybus(n):
    r, c, v = grids.ybus_triplets(grids.make_complex_grid(n, grids.SEED_BASE + 61))
    return host.lu(host.Matrix.from_triplets(n, n, r, c, v, by_rows=False), host.COLAMD)


def complex_star(n):
    k = list(range(1, n))
    return host.lu(host.Matrix.from_triplets(n, n, [0] + k + k + [0] * (n - 1), [0] + k + [0] * (n - 1) + k,
                                             [3.0 * n] + [2 + 1j] * (n - 1) + [-1j] * (n - 1) + [1 + 0j] * (n - 1),
                                             by_rows=False), host.COLAMD)


FACTORS = {
    "one": lambda: host.cholesky(host.Matrix.from_triplets(1, 1, [0], [0], [4.0])),
    "two": lambda: host.cholesky(random_spd(2, 1, 7)),
    "path": lambda: host.cholesky(path(997)),
    "islands": lambda: host.cholesky(islands(500)),
    "sparse": lambda: host.cholesky(random_spd(200, 3, 7)),
    "dense": lambda: host.cholesky(random_spd(60, 60, 7)),
    "star": lambda: host.cholesky(star_spd(200)),
    "grid": lambda: host.cholesky(configs.bprime(grids.make_grid(1500, 520, 11))),
    "large grid": lambda: host.cholesky(configs.bprime(grids.make_grid(9000, 3100, 12))),  # packets by two threads
    "lu": lambda: host.lu(random_square(120, 3, 3)),
    "jacobian": lambda: configs.jacobian_system(400, 1, 5).lu,
    "complex": lambda: complex_ybus(900),
    "complex star": lambda: complex_star(300),
}


@pytest.mark.parametrize("groups", [1, 32, 512])
@pytest.mark.parametrize("name", sorted(FACTORS))
def test_spread_packets_solve(name, groups):
    f = FACTORS[name]()
    cplx = isinstance(f, host.HostLu) and f.is_complex
    rhs = right_hand_sides(f.n, 3, 11)
    if cplx:
        rhs = rhs + 1j * right_hand_sides(f.n, 3, 12)
    cpu = orc.solve_many_lu(f, rhs) if cplx else orc.solve_many(f, rhs)
    for half in (False, True):
        full = 16 if cplx else 8
        lay = host.spread_layout(f, full // 2 if half else full, groups)
        d = worst_relative_difference(run(lay, rhs), cpu)
        assert d < (1e-4 if half else 1e-12), f"{name} groups {groups} half {half}: {d:e}"


def test_the_cut_depends_on_the_load_and_the_values_on_nothing():
    chol = FACTORS["grid"]()
    few, many = host.spread_layout(chol, 8, 1), host.spread_layout(chol, 8, 512)
    assert few["tasks"] > 1 and few["top"] > 0
    assert (few["tasks"], few["top"]) != (many["tasks"], many["top"])
    assert np.array_equal(few["blob"], host.spread_layout(chol, 8, 1)["blob"])


def test_too_many_live_values_are_refused():
    """Leaves that each touch 300 hubs: more rows than a top holds, more updates than a domain has slots."""
    leaves, hubs = 1600, 300
    r, c = (a.ravel() for a in np.meshgrid(np.arange(leaves), leaves + np.arange(hubs), indexing="ij"))
    d = np.arange(leaves + hubs)
    chol = host.cholesky(host.Matrix.from_triplets(d.size, d.size, np.r_[d, r, c], np.r_[d, c, r],
                                                   np.r_[np.where(d < leaves, 400.0, 4000.0), np.full(2 * r.size, -1.0)]))
    with pytest.raises(YbError) as e:
        host.spread_layout(chol)
    assert e.value.status == _lib.YB_ERROR_TOO_LARGE
