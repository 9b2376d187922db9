"""Slices of the output cells by the thousand: what the context keeps per slice
is bounded, a slice met again gives the same numbers, and a slice that a
caller's CUDA graph has recorded replays after others have come and gone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32c"])
def test_plans_of_many_slices_are_given_up(precision):
    import torch
    import dgv0d3v_direct_collision_b200 as m
    from dgv0d3v_direct_collision_b200 import _lib
    s = m.DGVSolver(2, 7, 6.0)
    s.generate_synthetic_A(seed=5, support=1)
    rng = np.random.default_rng(0)
    f = torch.tensor(np.exp(-(s.nodes_u ** 2 + s.nodes_v ** 2 + s.nodes_w ** 2)) * (1 + 0.2 * rng.standard_normal(s.N)),
                     device="cuda")
    prec = {"f64": _lib.DGV_PREC_F64, "f32c": _lib.DGV_PREC_F32C}[precision]
    stream = torch.cuda.Stream()
    out = torch.empty(s.N, dtype=torch.float64, device="cuda")

    def cells(a, b, q):
        assert s._lib.dgv_collide_cells(s._h, 1, f.data_ptr(), q.data_ptr(), a, b, prec) == 0

    try:
        # the work buffers at their largest first: they do not move afterwards
        s.EvalCollisionPeriodicAPlus_DGV(f.repeat(4, 1), precision=precision)
        slices = [(a, b) for a in range(0, s.Nc, 3) for b in range(a + 1, s.Nc + 1, 3)][:4000]
        cells(*slices[0], out)
        first = out[:(slices[0][1] - slices[0][0]) * s.P].clone()
        # a slice in the caller's own graph
        a, b = s.Nc // 3, s.Nc // 2
        rec = torch.empty((b - a) * s.P, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        s._check(s._lib.dgv_set_stream(s._h, stream.cuda_stream))
        s._check(s._lib.dgv_set_async(s._h, 1))
        cells(a, b, rec)
        stream.synchronize()
        want = rec.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            cells(a, b, rec)
        s._check(s._lib.dgv_set_async(s._h, 0))
        s._check(s._lib.dgv_set_stream(s._h, None))
        for c0, c1 in slices[:100]:
            cells(c0, c1, out)
        before = torch.cuda.mem_get_info()[0]
        for c0, c1 in slices[100:]:
            cells(c0, c1, out)
        after = torch.cuda.mem_get_info()[0]
        assert before - after < 8 << 20, (before - after) / 2 ** 20  # 3,900 slices; a plan takes 16 KB and more
        cells(*slices[0], out)
        assert torch.equal(out[:first.numel()], first)
        rec.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(rec, want)
    finally:
        s.close()
