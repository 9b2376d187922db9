"""The FP64 adjoint on the double-precision tensor instructions at the edges of
its tiles: <g, d> = <v, J d> with the mixed-terms operator (a separate kernel)
for several d, and results written over their own inputs.  Tolerance: both
sides are FP64 sums of the same products, 1e-12 of the sum of magnitudes."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

GRIDS = [
    dict(su=3, sv=3, sw=3, Mu=1, Mv=1, Mw=1),   # one cell, c1 = c2
    dict(su=3, sv=3, sw=3, Mu=2, Mv=3, Mw=5),
    dict(su=2, sv=2, sw=2, Mu=5, Mv=5, Mw=7),   # several items per block
    dict(su=1, sv=2, sw=4, Mu=3, Mv=3, Mw=2),
    dict(su=3, sv=3, sw=3, Mu=4, Mv=4, Mw=4),
]


def _solver(g):
    import dgv0d3v_direct_collision_b200 as m
    s = m.DGVSolver(**g, bounds=(-4.0, 4.0, -4.5, 4.5, -5.0, 5.0))
    s.generate_synthetic_A(seed=3, support=1)
    return s


@pytest.mark.parametrize("g", GRIDS, ids=lambda g: "x".join(str(v) for v in g.values()))
def test_transpose_of_the_mixed_terms(g):
    s = _solver(g)
    try:
        rng = np.random.default_rng(4)
        r2 = s.nodes_u ** 2 + s.nodes_v ** 2 + s.nodes_w ** 2
        f = np.exp(-r2 / 2.0) * (1.0 + 0.3 * rng.standard_normal((3, s.N)))
        v = rng.standard_normal((3, s.N))
        gs = s.vjp(f, v)
        for b in range(3):
            assert rel_err(s.vjp(f[b], v[b]), gs[b]) < 1e-13  # one VDF or a batch
            for _ in range(3):
                d = rng.standard_normal(s.N)
                Jd = s.jvp(f[b], d)
                assert abs(gs[b] @ d - v[b] @ Jd) < 1e-12 * (np.abs(gs[b]) @ np.abs(d) + np.abs(v[b]) @ np.abs(Jd))
        # a sparse cotangent reaches what its node's pairs reach, and nothing else
        e = np.zeros(s.N)
        e[s.N // 2] = 1.0
        full = s.vjp(f[0], e)
        d = rng.standard_normal(s.N)
        assert abs(full @ d - s.jvp(f[0], d)[s.N // 2]) < 1e-12 * (np.abs(full) @ np.abs(d))
    finally:
        s.close()


def test_result_over_an_input():
    import torch
    s = _solver(GRIDS[1])
    try:
        rng = np.random.default_rng(5)
        f = torch.tensor(rng.random((2, s.N)), device="cuda")
        v = torch.tensor(rng.standard_normal((2, s.N)), device="cuda")
        torch.cuda.synchronize()
        want = s.vjp(f, v).cpu().numpy()
        got = v.clone()
        torch.cuda.synchronize()
        s.vjp(f, got, got)
        assert rel_err(got.cpu().numpy(), want) < 1e-13
        got = f.clone()
        torch.cuda.synchronize()
        s.vjp(got, v, got)
        assert rel_err(got.cpu().numpy(), want) < 1e-13
    finally:
        s.close()
