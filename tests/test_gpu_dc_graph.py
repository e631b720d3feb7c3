"""The N-1 screening's kept graph, which the domain solve takes (the automatic choice takes the spread solve
and keeps none): it replays with new inputs of its sizes, and is dropped by a call of other sizes whichever
way that call goes, since such a call may move the buffers that the graph holds."""
import numpy as np
import pytest

from ybus_b200 import FP32, FP64, grids
from ybus_b200._lib import lib
from ybus_b200.dc import DcNetwork

pytestmark = pytest.mark.gpu

AUTO, DOMAIN = 0, 4


def network(gpu):
    g = grids.make_grid(2000, 700, grids.SEED_BASE + 4)
    net = DcNetwork.from_grid(gpu, g)
    return g, net, np.flatnonzero(~net.bridges())


def kind(net, which):
    assert lib().yb_factor_set_tile_kind(lib().yb_dc_network_factor(net._h), FP64, which) == 0


def batch(g, branches, cases, per_case, seed):
    rng = np.random.default_rng(seed)
    sp = np.arange(cases + 1) * per_case
    return rng.choice(branches, cases, replace=False), sp, rng.normal(0.0, 0.1, (sp[-1], g.n_bus)), rng.uniform(0.5, 2.0, g.n_branch)


def close(a, b):
    return np.allclose(a[1], b[1], rtol=1e-10, atol=0.0) and np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])


def test_the_domain_solves_graph_replays_new_inputs(gpu):
    g, net, branches = network(gpu)
    outaged, sp, inj, weights = batch(g, branches, 25, 3, 5)
    spread = net.outage_loadings_batch(outaged, sp, inj, weights)
    kind(net, DOMAIN)
    first = net.outage_loadings_batch(outaged, sp, inj, weights)
    again = net.outage_loadings_batch(outaged, sp, inj, weights)
    assert close(first, spread) and all(np.array_equal(a, b) for a, b in zip(first, again))
    scaled = net.outage_loadings_batch(outaged, sp, 2.0 * inj, weights)
    assert np.array_equal(scaled[0], first[0]) and np.allclose(scaled[1], 2.0 * first[1], rtol=1e-12)


@pytest.mark.parametrize("between", ["spread", "domain", "fp32"])
def test_a_call_of_other_sizes_drops_the_graph(gpu, between):
    g, net, branches = network(gpu)
    small, large = batch(g, branches, 20, 2, 5), batch(g, branches, 300, 9, 6)
    expected = net.outage_loadings_batch(*small)
    kind(net, DOMAIN)
    net.outage_loadings_batch(*small)
    if between == "spread":
        kind(net, AUTO)
    net.outage_loadings_batch(*large, precision=FP32 if between == "fp32" else FP64)
    kind(net, DOMAIN)
    other = (small[0], small[1], small[2][::-1].copy(), small[3])  # other inputs in buffers that have moved
    kind(net, AUTO)
    flipped = net.outage_loadings_batch(*other)
    kind(net, DOMAIN)
    assert close(net.outage_loadings_batch(*other), flipped)
    assert close(net.outage_loadings_batch(*small), expected)
