"""Host-to-device copies are complete, and in order with the context's stream,
when the library goes on.  cudaMemcpy from pageable memory may return once the
data is staged, and a stream made with cudaStreamNonBlocking does not wait for
the legacy stream it runs on, so a kernel launched next could read the array
before the data is there.  The host sources run here against a stand-in for
the CUDA runtime that lands such copies as late as the runtime's rules allow."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dgv0d3v_direct_collision_b200", "csrc")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <vector>
#include "dgv_internal.h"

// the stand-in runtime: work on a stream takes effect when the stream is
// synchronised; pageable host data is staged when a copy is issued
static std::map<cudaStream_t, std::vector<std::function<void()>>> work;
static std::map<char *, size_t> blocks;
static bool on_device(const void *p)
{
    for (auto &b : blocks)
        if ((const char *)p >= b.first && (const char *)p < b.first + b.second) return true;
    return false;
}
static cudaStream_t canon(cudaStream_t s) { return s == cudaStreamLegacy ? nullptr : s; }
static void run(cudaStream_t s)
{
    auto w = std::move(work[canon(s)]);
    work[canon(s)].clear();
    for (auto &f : w) f();
}
static size_t pending()
{
    size_t n = 0;
    for (auto &w : work) n += w.second.size();
    return n;
}
static cudaError_t copy(void *d, const void *s, size_t n, cudaStream_t st, bool sync)
{
    if (!on_device(d) || on_device(s)) {  // to the host (or within the device)
        work[canon(st)].push_back([=] { std::memcpy(d, s, n); });
        if (sync) run(st);
        return cudaSuccess;
    }
    std::vector<char> staged((const char *)s, (const char *)s + n);
    if (sync) run(st);
    work[canon(st)].push_back([=] { std::memcpy(d, staged.data(), n); });
    return cudaSuccess;
}
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = std::calloc(1, n);
    blocks[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { blocks.erase((char *)p); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { return copy(d, s, n, nullptr, true); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) { return copy(d, s, n, st, false); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
}

namespace dgv {
int set_err(Ctx *c, int code, const std::string &m) { c->err = m; return code; }
void release_graphs(const Ctx *) {}
// as stepping.cu's: both end with the context's stream synchronised
int ab_history_get(Ctx *c, int *order, std::vector<double> &frhs) { *order = 0; frhs.clear(); cudaStreamSynchronize(c->stream); return DGV_OK; }
int ab_history_set(Ctx *c, int, const double *) { cudaStreamSynchronize(c->stream); return DGV_OK; }
}
using namespace dgv;

extern "C" int dgv_write_solution(dgv_ctx *, const char *, const double *, double, double);
extern "C" int dgv_read_solution(dgv_ctx *, const char *, double *, double *, double *);
extern "C" int dgv_load_A(dgv_ctx *, int64_t, const int32_t *, const double *, const int32_t *, const int32_t *, int) { return DGV_EUNSUP; }
extern "C" int dgv_export_A(const dgv_ctx *, int64_t *, int32_t *, double *, int32_t *, int32_t *) { return DGV_EUNSUP; }

#define CHECK(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); return 1; } } while (0)

int main(int, char **argv)
{
    dgv_ctx h;
    Ctx *c = &h.c;
    c->own_stream = c->stream = (cudaStream_t)0x40;  // a non-blocking stream
    dgv_grid_desc d{};
    d.su = d.sv = d.sw = 1;
    d.Mu = d.Mv = d.Mw = 3;
    d.u_L = d.v_L = d.w_L = -3;
    d.u_R = d.v_R = d.w_R = 3;
    d.kappa = 1;
    CHECK(build_grid(d, c->grid, c->err) == DGV_OK);
    const int N = (int)c->grid.N;
    // the records of the canonical node: pairs (i, i + 1)
    std::vector<int32_t> phi(N, 0), xi, xi1;
    std::vector<double> A;
    phi[c->grid.ccell] = N - 1;
    for (int i = 0; i + 1 < N; i++) { xi.push_back(i); xi1.push_back(i + 1); A.push_back(1.0 + i); }
    std::string what = argv[1];
    if (what == "layout") {
        CHECK(layout_from_reference(c, N - 1, phi.data(), A.data(), xi.data(), xi1.data(), 0) == DGV_OK);
        CHECK(pending() == 0);
        CHECK(((double *)c->lay.rows64)[1] == 1.0);
    } else if (what == "chunks") {
        CHECK(layout_from_reference(c, N - 1, phi.data(), A.data(), xi.data(), xi1.data(), 0) == DGV_OK);
        run(nullptr);
        int *b = nullptr;
        CHECK(get_chunks(c, 3, &b) == DGV_OK);
        CHECK(pending() == 0);
        CHECK(b[3] == (int)c->lay.nblocks);
    } else {  // solution files, with a step of the context's stream still to run
        double *f = nullptr;
        cudaMalloc((void **)&f, N * sizeof(double));
        work[c->stream].push_back([=] { for (int i = 0; i < N; i++) f[i] = 7.0 + i; });
        CHECK(dgv_write_solution(&h, argv[2], f, 1.0, 0.1) == DGV_OK);
        work[c->stream].push_back([=] { for (int i = 0; i < N; i++) f[i] = -1.0; });
        CHECK(dgv_read_solution(&h, argv[2], f, nullptr, nullptr) == DGV_OK);
        CHECK(pending() == 0);
        for (int i = 0; i < N; i++) CHECK(f[i] == 7.0 + i);
    }
    return 0;
}
"""


def build_harness(d, text):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src = d / "harness.cpp"
    src.write_text(text)
    exe = d / "harness"
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"), "-I", os.path.join(ROOT, "include"),
                           "-I", CSRC, str(src)] + [os.path.join(CSRC, f) for f in ("layout.cpp", "afile.cpp", "grid.cpp")] +
                          ["-o", str(exe)])
    return str(exe)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    return build_harness(tmp_path_factory.mktemp("host_copies"), HARNESS)


@pytest.mark.parametrize("what", ["layout", "chunks"])
def test_uploads_are_complete_on_return(harness, what):
    r = subprocess.run([harness, what], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_device_sources_upload_the_same_way():
    """The work lists of the kernels' own files: no blocking copy from the host."""
    for path in glob.glob(os.path.join(CSRC, "*")):
        if not path.endswith((".cu", ".cpp", ".cuh", ".h")):
            continue
        src = re.sub(r"//[^\n]*", "", open(path).read())
        calls = re.findall(r"cudaMemcpy(?:2D|ToSymbol)?\([^;]*;", src)
        assert all("cudaMemcpyHostToDevice" not in c for c in calls), (os.path.basename(path), calls)


def test_solution_files_are_in_stream_order(harness, tmp_path):
    r = subprocess.run([harness, "solution", str(tmp_path / "f.sol")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
