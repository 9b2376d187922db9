"""DGV_OPT_TCSETMB is megabytes of block records, whatever the nodes per cell:
a block of 8 nodes has one record of 4 KB, so a set of 1 MB closes after 256
blocks; the default there is what suits those records."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def test_sets_of_eight_node_records_are_counted_in_their_bytes():
    import dgv0d3v_direct_collision_b200 as m
    from dgv0d3v_direct_collision_b200 import _lib
    s = m.DGVSolver(2, 7, 6.0)
    s.generate_synthetic_A(seed=5, support=1)
    try:
        assert s.get_option(_lib.DGV_OPT_TCSETMB) == 6
        f = np.exp(-(s.nodes_u ** 2 + s.nodes_v ** 2 + s.nodes_w ** 2)) * np.linspace(0.5, 1.5, 5)[:, None]
        q0 = s.EvalCollisionPeriodicAPlus_DGV(f, precision="tc")
        nblocks = s.A_info()["blocks"]
        for mb in (1, 2, 7):
            s.set_tc_set_mb(mb)
            s.set_tc_persistent(False)
            assert s.tc_plan(5)["launches"] == -(-nblocks // (256 * mb)), mb
            # the sets change the order of the FP64 sums alone
            assert rel_err(s.EvalCollisionPeriodicAPlus_DGV(f, precision="tc"), q0) < 1e-10
    finally:
        s.close()
    s = m.DGVSolver(3, 2, 6.0)
    assert s.get_option(_lib.DGV_OPT_TCSETMB) == 48
    s.close()
