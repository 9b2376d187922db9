"""The bounded waits of the FP64 and FP32-compensated kernels, of the FP64
adjoint and of the block form with eight nodes per cell: with a copy or an
arrival withheld (DGV_OPT_TEST_WITHHOLD) the wait for it runs out, the call
returns DGV_ETIMEOUT, and the same context then gives its earlier results."""
import time

import numpy as np
import pytest

from conftest import rel_err
from helpers import mixture_vdf

pytestmark = pytest.mark.gpu

CALLS = {
    "f64": lambda s, f, v: s.EvalCollisionPeriodicAPlus_DGV(f, precision="f64"),
    "f32c": lambda s, f, v: s.EvalCollisionPeriodicAPlus_DGV(f, precision="f32c"),
    "jvp": lambda s, f, v: s.jvp(f[0].copy(), v[0].copy()),
    "vjp": lambda s, f, v: s.vjp(f, v),
    "tc": lambda s, f, v: s.EvalCollisionPeriodicAPlus_DGV(f, precision="tc"),
}


@pytest.mark.parametrize("s_,M", [(3, 5), (2, 7)])
@pytest.mark.parametrize("f_global", [False, True])
def test_wait_runs_out_and_context_stays_usable(s_, M, f_global):
    import dgv0d3v_direct_collision_b200 as m
    from dgv0d3v_direct_collision_b200 import _lib
    L = _lib.load()
    s = m.DGVSolver(s_, M, 6.0)
    s.generate_synthetic_A(seed=11, support=1)
    s.set_f_global(f_global)
    rng = np.random.default_rng(4)
    f = np.stack([mixture_vdf(s.nodes_u, s.nodes_v, s.nodes_w, rng, normalise_w=s.nodes_gwts) for _ in range(3)])
    v = rng.standard_normal(f.shape)
    try:
        for name, call in CALLS.items():
            ref = call(s, f, v)
            assert L.dgv_set_option(s._h, _lib.DGV_OPT_WAIT_LIMIT_US, 20000) == 0  # 20 ms
            assert L.dgv_set_option(s._h, _lib.DGV_OPT_TEST_WITHHOLD, 1) == 0
            t = time.perf_counter()
            with pytest.raises(_lib.DGVError) as ei:
                call(s, f, v)
            elapsed = time.perf_counter() - t
            assert ei.value.code == _lib.DGV_ETIMEOUT, name
            assert elapsed < 10.0, (name, elapsed)
            assert L.dgv_set_option(s._h, _lib.DGV_OPT_WAIT_LIMIT_US, 0) == 0
            assert rel_err(call(s, f, v), ref) < 1e-12, name
    finally:
        s.close()
