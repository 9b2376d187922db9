"""The FP64, mixed-terms and FP32-compensated kernels at the grid sizes where
what lies in shared memory changes: tiles added at once at a unit's end, stages
per warp, the partial Q in shared or global memory, f (and g) in shared or
global memory.  Checked against dgv_collide_f64_noalloc with the tolerances of
test_gpu_mma_f64; the mixed terms as (Q(f+d) - Q(f-d)) / 2 of that kernel."""
import numpy as np
import pytest

from conftest import max_rel_err, rel_err
from test_gpu_mma_f64 import TOL, _lanewise, _vdfs

pytestmark = pytest.mark.gpu

# cells: where Q / the mixed terms (227 KB of shared memory) / FP32 change
SIZES = [
    (3, (5, 6, 8)),    # 240: 4 tiles / 1 tile at once
    (3, (5, 7, 7)),    # 245: - / partial Q in global memory beside f and g
    (3, (7, 7, 7)),    # 343: 1 tile / partial Q in global memory, 2 stages
    (3, (8, 8, 6)),    # 384: partial Q in global memory / f and g in global memory
    (3, (8, 9, 8)),    # 576: - / 2 tiles / FP32: partial Q in global memory
    (3, (9, 9, 10)),   # 810: f and the partial Q in global memory for both
    (2, (11, 10, 10)),  # 1,100: - / partial Q in global memory beside f and g
    (2, (12, 12, 11)),  # 1,584: 2 tiles / 2 stages
    (2, (12, 12, 12)),  # 1,728: partial Q in global memory / f and g in global memory
    (2, (13, 13, 14)),  # 2,366: - / - / FP32: partial Q in global memory
]


@pytest.mark.parametrize("s_,cells", SIZES, ids=lambda x: str(x))
def test_every_placement_gives_the_same_sums(s_, cells):
    import dgv0d3v_direct_collision_b200 as m
    s = m.DGVSolver(su=s_, sv=s_, sw=s_, Mu=cells[0], Mv=cells[1], Mw=cells[2],
                    bounds=(-4.0, 4.0, -4.5, 4.5, -5.0, 5.0))
    s.generate_synthetic_A(seed=3, Trad=2.0, support=1)
    try:
        assert s.A_info()["pairs"] > 1000
        f, d = _vdfs(s, 2)
        ref = _lanewise(s, np.stack([f, f + d, f - d]))
        q = s.EvalCollisionPeriodicAPlus_DGV(f, precision="f64")
        assert rel_err(q, ref[0]) < TOL and max_rel_err(q, ref[0]) < TOL
        scale = np.abs(ref[1]).max()
        assert np.abs(s.jvp(f, d) - (ref[1] - ref[2]) / 2.0).max() < TOL * scale
        assert rel_err(s.EvalCollisionPeriodicAPlus_DGV(f, precision="f32c"), ref[0]) < 1e-6
    finally:
        s.close()
