"""The block form with eight nodes per cell (one group of 64 columns, K = 16,
four item slots, eight accumulators): batches that fill and do not fill the
tiles of 32, 64 and 128 VDFs, one and several VDF tiles, both launch forms, the
operator and its adjoint, against the FP64 kernels.  Tolerance: 1e-6
norm-wise, that of the arithmetic (as in the parity tests of 27 nodes)."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import mixture_vdf

pytestmark = pytest.mark.gpu

TOLTC = 1e-6


def _solver(**g):
    import dgv0d3v_direct_collision_b200 as m
    s = m.DGVSolver(**g, bounds=(-5.0, 5.0, -4.5, 4.5, -5.0, 5.0))
    s.generate_synthetic_A(seed=3, support=1)
    return s


@pytest.fixture(scope="module", params=[
    dict(su=2, sv=2, sw=2, Mu=5, Mv=4, Mw=5),
    dict(su=1, sv=2, sw=4, Mu=5, Mv=3, Mw=2),  # unequal nodes per axis, 30 cells: a ragged last row tile
], ids=lambda g: "x".join(str(v) for v in g.values()))
def sol(request):
    s = _solver(**request.param)
    yield s
    s.close()


@pytest.mark.parametrize("nb", [1, 32, 33, 65, 150, 300])
def test_eight_nodes_against_fp64(sol, nb):
    s = sol
    rng = np.random.default_rng(nb)
    f = np.stack([mixture_vdf(s.nodes_u, s.nodes_v, s.nodes_w, rng, normalise_w=s.nodes_gwts) * 10.0 ** rng.uniform(-2, 2)
                  for _ in range(nb)])
    v = rng.standard_normal(f.shape)
    q64 = s.EvalCollisionPeriodicAPlus_DGV(f)
    g64 = s.vjp(f, v)
    for tiles in (2, 1):
        s.set_tc_tiles_per_cta(tiles)
        res = []
        for pers in (False, True):
            s.set_tc_persistent(pers)
            res.append((s.EvalCollisionPeriodicAPlus_DGV(f, precision="tc"), s.vjp(f, v, precision="tc")))
        assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])
        for k in range(nb):
            assert rel_err(res[0][0][k], q64[k]) < TOLTC and rel_err(res[0][1][k], g64[k]) < TOLTC, (tiles, k)
