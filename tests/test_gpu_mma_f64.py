"""The FP64 operator on the double-precision tensor instructions (8 or 27 nodes
per cell) at the edges of its tiles: boxes of one to many cells, grids whose
axes differ, one and several ranges, ranges of output cells cut inside a box.

Checked against dgv_collide_f64_noalloc, a separate kernel with one output
cell per lane.  Tolerance: both add K <= 1e5 products of at most N unit
roundings each way, so they differ by at most a few sqrt(K) eps of the sum of
magnitudes, which synthetic records (random signs) hold within ~1e2 of |Q|:
1e-12 of max |Q|, the FP64 tolerance of the parity tests."""
import numpy as np
import pytest

from conftest import max_rel_err, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12
GRIDS = [
    dict(su=3, sv=3, sw=3, Mu=1, Mv=1, Mw=1),   # one cell: one box of one cell
    dict(su=3, sv=3, sw=3, Mu=2, Mv=3, Mw=5),   # 30 cells, axes differ, tiles of 1 to 4
    dict(su=2, sv=2, sw=2, Mu=5, Mv=5, Mw=7),   # boxes of up to 175 cells: several units
    dict(su=1, sv=2, sw=4, Mu=3, Mv=3, Mw=2),   # 8 nodes per cell, unequal per axis
    dict(su=3, sv=3, sw=3, Mu=4, Mv=4, Mw=4),
]


def _solver(g):
    import dgv0d3v_direct_collision_b200 as m
    s = m.DGVSolver(**g, bounds=(-4.0, 4.0, -4.5, 4.5, -5.0, 5.0))
    s.generate_synthetic_A(seed=3, support=1)
    return s


def _vdfs(s, nb, seed=1):
    rng = np.random.default_rng(seed)
    r2 = s.nodes_u ** 2 + s.nodes_v ** 2 + s.nodes_w ** 2
    return np.exp(-r2 / 2.0) * (1.0 + 0.3 * rng.standard_normal((nb, s.N)))


def _lanewise(s, f):
    import torch
    fd = torch.tensor(f, device="cuda")
    q = torch.empty_like(fd)
    torch.cuda.synchronize()
    rc = s._lib.dgv_collide_f64_noalloc(s._h, fd.data_ptr(), q.data_ptr(), f.shape[0], None)
    assert rc == 0, s._lib.dgv_last_error(s._h)
    torch.cuda.synchronize()
    return q.cpu().numpy()


@pytest.mark.parametrize("g", GRIDS, ids=lambda g: "x".join(str(v) for v in g.values()))
def test_equals_the_lanewise_kernel(g):
    s = _solver(g)
    try:
        for nb in (1, 3):
            f = _vdfs(s, nb)
            ref = _lanewise(s, f)
            for chunks in (0, 1, 7, 300):
                s.set_nchunks(chunks)
                q = s.EvalCollisionPeriodicAPlus_DGV(f, precision="f64")
                assert rel_err(q, ref) < TOL and max_rel_err(q, ref) < TOL, (nb, chunks)
            s.set_nchunks(0)
            # output cells in uneven slices, cut inside boxes
            cuts = sorted({0, 1 % s.Nc, s.Nc // 3, (2 * s.Nc) // 3 + 1 if s.Nc > 2 else 0, s.Nc})
            parts = [s.collide_cells(f, a, b, precision="f64") for a, b in zip(cuts, cuts[1:]) if b > a]
            q = np.concatenate(parts, axis=-1)
            assert rel_err(q, ref) < TOL and max_rel_err(q, ref) < TOL
    finally:
        s.close()


@pytest.mark.parametrize("g", GRIDS[1:3], ids=["s3", "s2"])
def test_mixed_terms_are_the_polarisation_of_q(g):
    """Q(f+d) - Q(f-d) = 2 (mixed terms of f and d), exactly in the bilinear form."""
    s = _solver(g)
    try:
        f, d = _vdfs(s, 2)
        scale = np.abs(s.EvalCollisionPeriodicAPlus_DGV(f + d, precision="f64")).max()
        want = (s.EvalCollisionPeriodicAPlus_DGV(f + d, precision="f64") -
                s.EvalCollisionPeriodicAPlus_DGV(f - d, precision="f64")) / 2.0
        for on in (False, True):
            s.set_f_global(on)
            assert np.abs(s.jvp(f, d) - want).max() < TOL * scale
    finally:
        s.close()


def test_non_finite_values_stay_where_they_belong():
    """An infinite f value reaches the output nodes it reaches lane by lane, and no others."""
    s = _solver(GRIDS[1])
    try:
        f = _vdfs(s, 1)
        f[0, 5] = np.inf
        ref = _lanewise(s, f)
        q = s.EvalCollisionPeriodicAPlus_DGV(f, precision="f64")
        assert np.array_equal(np.isfinite(q), np.isfinite(ref))
        ok = np.isfinite(ref)
        assert np.abs(q[ok] - ref[ok]).max() < TOL * np.abs(ref[ok]).max() if ok.any() else True
    finally:
        s.close()


@pytest.mark.parametrize("g", GRIDS, ids=lambda g: "x".join(str(v) for v in g.values()))
def test_fp32_compensated_on_the_same_units(g):
    """FP32 products in groups of 16 pairs, compensated: within the 1e-6 of the
    arithmetic from FP64, and the same up to the order of the compensated group
    sums (a few 2^-48) whatever the ranges, slices or the place of f."""
    s = _solver(g)
    try:
        f = _vdfs(s, 3)
        ref = _lanewise(s, f)
        q = s.EvalCollisionPeriodicAPlus_DGV(f, precision="f32c")
        assert rel_err(q, ref) < 1e-6
        for chunks in (1, 7, 300):
            s.set_nchunks(chunks)
            assert rel_err(s.EvalCollisionPeriodicAPlus_DGV(f, precision="f32c"), q) < 1e-11
        s.set_nchunks(0)
        s.set_f_global(True)
        assert np.array_equal(s.EvalCollisionPeriodicAPlus_DGV(f, precision="f32c"), q)
        s.set_f_global(False)
        cuts = sorted({0, s.Nc // 3, s.Nc})
        parts = [s.collide_cells(f, a, b, precision="f32c") for a, b in zip(cuts, cuts[1:])]
        assert rel_err(np.concatenate(parts, axis=-1), q) < 1e-11
    finally:
        s.close()
