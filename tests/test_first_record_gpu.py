"""Record of the first iteration where no frontier list is built (union-find CC, MIS)."""
import numpy as np
import pytest

import indigo2suite_b200 as i2
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,first,star", [(5, 2, 2), (70, 33, 20), (4000, 1, 300), (4000, 3999, 0)])
def test_first_record_counts_the_vertices_with_edges(gpu, n, first, star):
    # vertices before `first` and after the star are isolated
    leaves = np.arange(first + 1, first + 1 + star)
    u = np.concatenate([np.full(star, first), leaves])
    v = np.concatenate([leaves, np.full(star, first)])
    o = np.lexsort((v, u))
    ni = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(u[o], minlength=n), out=ni[1:])
    g = i2.ECLGraph(n, len(u), ni, v[o].astype(np.int32), np.ones(len(u), np.int32))
    dg = i2.DeviceGraph.upload(g)
    dg.tune(heavy_threshold=32)
    linked = star + 1 if star else 0
    for loop in (i2.I2_LOOP_GRAPH, i2.I2_LOOP_RELAUNCH, i2.I2_LOOP_HOST):
        for run, ref in ((lambda: dg.cc(variant="union_find", loop=loop), oracle.cc(g)),
                         (lambda: dg.cc(variant="vp_cta", loop=loop), oracle.cc(g)),
                         (lambda: dg.mis(loop=loop), oracle.mis(g))):
            np.testing.assert_array_equal(run()[0], ref)
            r = dg.records()[0]
            assert (r["size"], r["edges"], r["hsize"]) == (linked, 2 * star, int(star >= 32))
            assert (r["maxdeg"], r["mindist"]) == (star, first if star else i2.INF)
    dg.free()
