"""Per-iteration sweep: every style is timed, however the graph came to the device."""
import numpy as np
import pytest

import indigo2suite_b200 as i2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [i2.I2_BFS, i2.I2_SSSP, i2.I2_CC])
def test_sweep_times_the_same_styles_on_uploaded_and_generated_graphs(gpu, algo):
    host = i2.gen_rmat(10, 8, seed=3)
    edge_topo = i2.VARIANTS.index("edge_topo")
    made = {
        "uploaded": lambda: i2.DeviceGraph.upload(host),
        "generated": lambda: i2.DeviceGraph.generate_rmat(10, 8, seed=3),
    }
    styles = {}
    for name, make in made.items():
        for follow in (-1, edge_topo):  # a fresh handle each: nothing an earlier call has built
            g = make()
            recs, times = g.sweep(algo, g.hub(), follow=follow)
            assert len(recs) > 0
            styles[name, follow] = np.flatnonzero((times > 0).any(axis=0)).tolist()
            if follow >= 0:
                assert all(r["variant"] == edge_topo for r in recs)
            g.free()
    assert len({tuple(s) for s in styles.values()}) == 1, styles
    assert edge_topo in styles["generated", -1]
