"""BFS by topology-driven pull: progress inside an iteration, and its use beside other styles."""
import numpy as np
import pytest

import indigo2suite_b200 as i2
import oracle

pytestmark = pytest.mark.gpu


def _chain(n, vertices):
    """A path through `vertices` in a graph of n, both directions."""
    a, b = np.array(vertices[:-1]), np.array(vertices[1:])
    u, v = np.concatenate([a, b]), np.concatenate([b, a])
    o = np.lexsort((v, u))
    ni = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(u, minlength=n), out=ni[1:])
    return i2.ECLGraph(n, len(u), ni, v[o].astype(np.int32), np.ones(len(u), np.int32))


@pytest.mark.parametrize("loop", [i2.I2_LOOP_GRAPH, i2.I2_LOOP_RELAUNCH, i2.I2_LOOP_HOST])
def test_fixed_pull_topo_uses_levels_of_the_same_iteration(gpu, loop):
    # one block per SM: vertices a whole grid of threads apart belong to one
    # thread, which visits them in ascending order in every sweep
    import torch

    step = torch.cuda.get_device_properties(0).multi_processor_count * 256
    hops = 12
    g = _chain((hops + 1) * step, [k * step + 5 for k in range(hops + 1)])
    dg = i2.DeviceGraph.upload(g)
    dg.tune(blocks_per_sm=1)
    d, rep = dg.bfs(5, variant="pull_topo", loop=loop)
    np.testing.assert_array_equal(d, oracle.bfs(g, 5))
    assert rep.iterations == 2  # all levels in the first sweep; the second finds nothing to lower
    # beside another style it keeps to levels, which the edge-balanced push relies on
    for at in (1, 3, hops):
        d, rep = dg.bfs(5, variant="pull_topo", then_variant="vp_cta", then_at=at, loop=loop)
        np.testing.assert_array_equal(d, oracle.bfs(g, 5))
        assert rep.iterations >= hops
    dg.free()


@pytest.mark.parametrize("n", [33, 1025, 40000])
def test_pull_topo_levels_on_random_graphs(gpu, n):
    g = i2.gen_er(n, 3 * n, seed=n)
    dg = i2.DeviceGraph.upload(g)
    s = dg.hub()
    ref = oracle.bfs(g, s)
    for kw in ({}, {"then_variant": "vp_cta", "then_at": 2}):
        d, rep = dg.bfs(s, variant="pull_topo", **kw)
        np.testing.assert_array_equal(d, ref)
        assert rep.reached_vertices == int((ref != i2.INF).sum())
    dg.free()
