"""The shared-memory carveout is an attribute of kernels that all graphs share."""
import pytest

import indigo2suite_b200 as i2
import oracle

pytestmark = pytest.mark.gpu


def test_a_graph_stays_resident_after_another_changed_the_carveout(gpu, monkeypatch):
    host = i2.gen_er(3000, 12000, seed=4)
    a, b = i2.DeviceGraph.upload(host), i2.DeviceGraph.upload(host)
    ref = oracle.bfs(host, 0)
    try:
        assert (a.bfs(0)[0] == ref).all()
        b.tune(smem_carveout=0)  # fewer blocks of the kernel fit an SM than a's grid takes
        assert (b.bfs(0)[0] == ref).all()
        assert (a.bfs(0)[0] == ref).all()
        # only a resident traversal has a release to withhold
        monkeypatch.setenv("I2_TEST_HOLD_BARRIER", "1")
        monkeypatch.setenv("I2_STALL_MS", "50")
        with pytest.raises(i2.I2Error) as e:
            a.bfs(0)
        assert e.value.status == i2._capi.I2_ERR_STALL
        monkeypatch.delenv("I2_TEST_HOLD_BARRIER")
        assert (a.bfs(0)[0] == ref).all()
    finally:
        a.tune(smem_carveout=-1)
        a.free()
        b.free()
