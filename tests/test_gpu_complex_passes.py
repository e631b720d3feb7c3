"""Complex batches over a factor's life: the first solves go by tiles and lay nothing out, the later ones by
the spread solve; every pass is held to the bars of the first, with counts around a group's 32 and a block's
four groups, arrays on 8-byte boundaries, values that are not finite, and FP32 with refinement."""
import numpy as np
import pytest

import oracle.oracle as orc
from fixtures import worst_relative_difference
from test_gpu_spread import BARS, complex_dense, complex_path, complex_star, complex_two
from ybus_b200 import FP32, FP64, GpuFactor, grids, host, solve_batch_complex

pytestmark = pytest.mark.gpu

PASSES = 7  # of which the first four by tiles


def device(b, shift):
    """b on the device from an 8-byte boundary that is (shift 0) or is not a 16-byte one."""
    import torch
    t = torch.zeros(2 * b.size + 2, dtype=torch.float64)
    t[shift:shift + 2 * b.size] = torch.from_numpy(np.ascontiguousarray(b).view(np.float64).ravel())
    return t.cuda()


def batch(gpu, factors, rhs, prec, shifts=None, max_steps=0, ratios=None):
    import torch
    shifts = shifts or [0] * len(rhs)
    bs = [device(b, s) for b, s in zip(rhs, shifts)]
    xs = [torch.full_like(b, 7.0) for b in bs]
    torch.cuda.synchronize()
    steps = solve_batch_complex(factors, [b.data_ptr() + 8 * s for b, s in zip(bs, shifts)],
                                [x.data_ptr() + 8 * s for x, s in zip(xs, shifts)], [len(b) for b in rhs], prec,
                                max_steps=max_steps, d_ratio=None if ratios is None else [r.data_ptr() for r in ratios])
    gpu.synchronize()
    out = []
    for x, b, s in zip(xs, rhs, shifts):
        x = x.cpu().numpy()
        assert np.all(x[:s] == 7.0) and np.all(x[s + 2 * b.size:] == 7.0), "only the solutions are written"
        out.append(x[s:s + 2 * b.size].view(np.complex128).reshape(b.shape))
    return out, steps


def networks(gpu, sizes, seed):
    out = []
    for k, n in enumerate(sizes):
        r, c, v = grids.ybus_triplets(grids.make_complex_grid(n, grids.SEED_BASE + 70 + seed + k))
        a = host.Matrix.from_triplets(n, n, r, c, v, by_rows=False)
        lu = host.lu(a, host.COLAMD)
        f = GpuFactor.from_lu_complex(gpu, lu)
        f.attach_matrix_complex(a)
        out.append((lu, f))
    return out


def columns(n, count, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((count, n)) + 1j * rng.standard_normal((count, n))


def test_a_factors_first_solves_lay_nothing_out(gpu):
    """By the tiles' bits, which arrays on 8-byte boundaries always get; later passes by the spread solve's."""
    (lu, f), (lu2, f2) = networks(gpu, (1500, 400), 3)
    rhs = [columns(lu.n, 70, 1), columns(lu2.n, 33, 2)]
    passes = [batch(gpu, [f, f2], rhs, FP64)[0] for _ in range(PASSES)]
    tiles = batch(gpu, [f, f2], rhs, FP64, shifts=[1, 1])[0]
    for k in range(4):
        assert all(np.array_equal(x, t) for x, t in zip(passes[k], tiles))
    for k in range(4, PASSES):
        assert not np.array_equal(passes[k][0], tiles[0])
        assert all(np.array_equal(x, t) for x, t in zip(passes[k], passes[4]))
    # another class of counts takes the layout that is there, one with a new factor both ways at once
    (lu3, f3), = networks(gpu, (600,), 9)
    rhs = [columns(lu.n, 700, 4), columns(lu3.n, 5, 5)]
    for x, b, l in zip(batch(gpu, [f, f3], rhs, FP64)[0], rhs, (lu, lu3)):
        assert worst_relative_difference(x[::31], orc.solve_many_lu(l, b[::31])) < 1e-12


@pytest.mark.parametrize("prec,bar", BARS)
@pytest.mark.parametrize("counts", [(1, 32, 33, 129), (0, 31, 300, 2), (64, 0, 1, 0)])
def test_every_pass_matches_the_cpu(gpu, counts, prec, bar):
    lus = [lu for _, lu in (complex_two(), complex_path(997), complex_dense(60), complex_star(300))]
    factors = [GpuFactor.from_lu_complex(gpu, lu) for lu in lus]
    if prec == FP32:
        for f, (a, _) in zip(factors, (complex_two(), complex_path(997), complex_dense(60), complex_star(300))):
            f.attach_matrix_complex(a)
    rhs = [columns(lu.n, c, 5) for lu, c in zip(lus, counts)]
    cpu = [orc.solve_many_lu(lu, b) if len(b) else None for lu, b in zip(lus, rhs)]
    for k in range(PASSES):
        for shifts in ([0, 0, 0, 0], [0, 1, 0, 1]):
            for x, c in zip(batch(gpu, factors, rhs, prec, shifts)[0], cpu):
                assert c is None or worst_relative_difference(x, c) < bar


def test_later_passes_of_uneven_networks_and_refinement(gpu):
    """Complex128 to four times the residual of the oracle's own substitution (1.2e-12 on the 600-bus network)."""
    import torch
    nets = networks(gpu, (200, 1500, 600, 3000), 21)
    lus, factors = zip(*nets)
    rhs = [columns(lu.n, c, 6) for lu, c in zip(lus, (3, 7, 16, 40))]
    ratios = [torch.zeros(len(b), dtype=torch.float64, device="cuda") for b in rhs]
    cpu = [orc.solve_many_lu(lu, b) for lu, b in zip(lus, rhs)]

    def residual(n, seed, x, b):
        a = np.zeros((n, n), complex)
        r, c, v = grids.ybus_triplets(grids.make_complex_grid(n, seed))
        np.add.at(a, (r, c), v)
        return (np.abs(b - x @ a.T).max(axis=1) / np.abs(b).max(axis=1)).max()

    oracle = [residual(lu.n, grids.SEED_BASE + 91 + k, x, b) for k, (lu, x, b) in enumerate(zip(lus, cpu, rhs))]
    for k in range(PASSES):
        for prec, bar in ((FP64, 1e-12), (FP32, 1e-8)):
            xs, steps = batch(gpu, list(factors), rhs, prec, max_steps=3, ratios=ratios)
            assert prec == FP64 or 1 <= steps[0] <= 3
            for x, c, r, own in zip(xs, cpu, ratios, oracle):
                assert float(r.max()) <= (4 * own if prec == FP64 else 1e-10)
                assert worst_relative_difference(x, c) < bar


@pytest.mark.parametrize("count", [1, 40])
def test_a_value_not_finite_stays_in_its_island_in_every_pass(gpu, count):
    n = 700
    k = np.arange(n)
    j = (k // 2 * 2 + 37 * (1 + k % 5)) % n  # neighbours of a parity: even rows and odd rows are islands
    j = np.where((j + k) % 2 == 0, j, (j + 1) % n)
    r, c, w = np.r_[k, k, j], np.r_[k, j, k], 1.0 + (k % 7) / 7.0
    keep = r != c
    keep[:n] = True
    v = np.r_[np.full(n, 30.0), -w, -w][keep] * (1 + 0.25j)
    factor = GpuFactor.from_lu_complex(gpu, host.lu(host.Matrix.from_triplets(n, n, r[keep], c[keep], v, by_rows=False),
                                                    host.COLAMD))
    b = columns(n, count, 7)
    spoiled = b.copy()
    spoiled[count // 2, 10] = np.nan
    others = np.arange(count) != count // 2
    for _ in range(3):
        (clean,), _ = batch(gpu, [factor], [b], FP64)
        (x,), _ = batch(gpu, [factor], [spoiled], FP64)
        (clean2,), _ = batch(gpu, [factor], [b], FP64)
        assert np.isnan(x[count // 2, 10]) and np.isfinite(x[others]).all()
        assert worst_relative_difference(x[others], clean[others]) < 1e-12 if count > 1 else True
        assert worst_relative_difference(x[[count // 2], 1::2], clean2[[count // 2], 1::2]) < 1e-12


@pytest.mark.parametrize("count", [1, 16, 129, 700])
def test_residuals_of_a_network_with_a_hub(gpu, count):
    """One column a piece; the ratios told are those of the solutions."""
    import torch
    n = 400
    k = np.arange(1, n)
    r, c = np.r_[np.arange(n), np.zeros(n - 1, int), k], np.r_[np.arange(n), k, np.zeros(n - 1, int)]
    v = np.r_[np.full(n, n + 1.0), np.full(2 * n - 2, -1.0)] * (1 + 0.3j)
    a = host.Matrix.from_triplets(n, n, r, c, v, by_rows=False)
    lu = host.lu(a, host.COLAMD)
    f = GpuFactor.from_lu_complex(gpu, lu)
    f.attach_matrix_complex(a)
    dense = np.zeros((n, n), complex)
    dense[r, c] = v
    b = columns(n, count, 8)
    ratio = [torch.zeros(count, dtype=torch.float64, device="cuda")]
    for prec in (FP64, FP32):
        (x,), _ = batch(gpu, [f], [b], prec, max_steps=3, ratios=ratio)
        own = np.abs(b - x @ dense.T).max(axis=1) / np.abs(b).max(axis=1)
        # both sums of 400 products: a bound on their rounding
        assert np.abs(ratio[0].cpu().numpy() - own).max() <= 400 * 2.0 ** -52
        assert worst_relative_difference(x, orc.solve_many_lu(lu, b)) < (1e-12 if prec == FP64 else 1e-8)
