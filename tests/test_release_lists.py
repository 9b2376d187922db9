"""dgv_release_layouts(F32) gives back what only the FP32 rows need: the rows
and the work lists of their 16-pair groups; the FP64 lists stay.  Host code, on
the stand-in runtime of test_host_copies."""
import subprocess

from test_host_copies import HARNESS, build_harness

MAIN = r"""
static void *dev(size_t n) { void *p = nullptr; cudaMalloc(&p, n); return p; }
static void fill(MmaList &m)
{
    m.segs = dev(64);
    m.sfirst = dev(64);
    m.box.resize(2);
    MmaPlan &pl = m.plans[{0, 5}];
    pl.units = dev(64);
    pl.bounds[3] = dev(64);
}
int main()
{
    dgv_ctx h;
    Ctx *c = &h.c;
    c->stream = (cudaStream_t)0x40;
    c->lay.rows64 = dev(64);
    c->lay.rows32 = dev(64);
    fill(c->lay.mma);
    fill(c->lay.groups);
    CHECK(blocks.size() == 10);
    CHECK(release_layouts(c, DGV_LAYOUT_F32) == DGV_OK);
    CHECK(blocks.size() == 5);
    CHECK(!c->lay.rows32 && !c->lay.groups.segs && !c->lay.groups.sfirst && c->lay.groups.plans.empty());
    CHECK(c->lay.rows64 && c->lay.mma.segs && c->lay.mma.plans.size() == 1);
    CHECK(release_layouts(c, DGV_LAYOUT_F32) == DGV_OK);
    free_layout(c->lay);
    CHECK(blocks.empty());
    return 0;
}
"""


def test_f32_release_frees_the_group_lists(tmp_path):
    exe = build_harness(tmp_path, HARNESS[:HARNESS.index("int main")] + MAIN)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
