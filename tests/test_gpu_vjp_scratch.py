"""The FP64 adjoint's work space does not grow with the batch: a batch whose
sums and cotangents would take 0.6 GB runs in pieces, each VDF as by itself."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def test_large_batch_in_bounded_scratch():
    import torch
    import dgv0d3v_direct_collision_b200 as m
    s = m.DGVSolver(2, 2, 4.0)
    s.generate_synthetic_A(seed=3, support=1)
    try:
        nb = 600_000
        gen = torch.Generator(device="cuda").manual_seed(1)
        base = torch.tensor(np.exp(-(s.nodes_u ** 2 + s.nodes_v ** 2 + s.nodes_w ** 2) / 2), device="cuda")
        f = base * (1 + 0.2 * torch.rand(nb, s.N, generator=gen, device="cuda", dtype=torch.float64))
        v = torch.randn(nb, s.N, generator=gen, device="cuda", dtype=torch.float64)
        g = torch.empty_like(f)
        s.vjp(f[:2], v[:2], out=g[:2])
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s.vjp(f, v, out=g)
        # beside the room that the call reserves for two host arrays (reserve_in)
        assert before - torch.cuda.mem_get_info()[0] - 2 * f.numel() * 8 < 200 << 20
        # 128 MB hold 131,072 VDFs of 64 nodes: both sides of the seams, and the ends
        for b in (0, 131071, 131072, 262143, 262144, nb - 1):
            one = s.vjp(f[b].contiguous(), v[b].contiguous())
            assert rel_err(g[b].cpu().numpy(), one.cpu().numpy()) < 1e-13, b
    finally:
        s.close()
