// adjoint_mma.cu -- FP64 vector-Jacobian product of the collision operator on
// the double-precision tensor instructions (grids of 8 or 27 nodes per cell).
//
// g_k = sum_i c_i sum_j A_j (delta_{k,a_j} f(b_j) + delta_{k,b_j} f(a_j)),
// c = 2 v / w (the adjoint of collision_mod.f90:213-216).  For a block (cells
// c1, c2) and output cell D, with pair k = (l1, l2):
//   vA[D, k]     = sum_p c(D, p) V[k, p]              (a matrix product)
//   g(c1+D, l1) += sum_l2 vA[D, k] f(c2+D, l2)
//   g(c2+D, l2) += sum_l1 vA[D, k] f(c1+D, l1).
// One cell per lane and two atomics per pair and cell (adjoint.cu) is bound by
// the atomics.  Here a warp takes a block and up to 16 of its cells (rows) at a
// time, keeps their c as A fragments in registers, and multiplies them with
// tiles of up to 8 pairs of one l1 (mma.m8n8k4, K = P padded to a multiple of
// 4).  Both scatters stay inside the warp: the sums over l2 in registers until
// the l1 ends, those over l1 in shared memory until the block ends, so that at
// most 2 P atomics per cell go to g, 54 instead of ~745 at 27^3.  As before the
// order of the atomics, and so the last bits of g, vary from run to run.
//
// Warps are independent (no CTA barrier): each takes the next item, heaviest
// blocks first, from a counter, and streams the block's rows through a ring of
// bulk copies of its own.
//
// Measured (B200, 1965 MHz), one VDF at 21^3: 44.9 ms with one cell per lane,
// 5.5 ms here (27^3: 260 -> 40.5).  The products take 2.4 ms of that (76 % of a tile's pairs are
// real: a block has ~16 pairs per l1); shared memory delivers 63 % of its words
// and the warps' own dependent steps per tile fill the rest, so four warps per
// scheduler with two row tiles are faster than two with three (6.8 ms, also
// with the scatter of a tile behind the products of the next).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "dgv_internal.h"
#include "pipeline.cuh"

namespace dgv {

constexpr int VJ_WARPS = 16;
constexpr int VJ_NT = 2;              // row tiles of 8 per item
constexpr int VJ_S = 8 * VJ_NT + 4;   // row stride of the per-node arrays: lanes (4 pairs x 4 rows) hit 16 banks of 8 B
constexpr int VJ_NST = 3;             // ring stages per warp, a tile each
constexpr int VJ_MAXT = 108;          // tiles per block, at most: 27 nodes l1 x 4

struct __align__(16) VjpItem {
    int block, row0, nrow, pad;
};

struct VjpMmaArgs {
    const double *f, *c;  // [nvdf][N]
    double *g;            // [nvdf][N], zeroed
    const BlockInfo *blk;
    const char *rows;
    const int *tfirst;        // [nblocks + 1]: first tile of each block
    const unsigned *tiles;    // first pair of the tile within its block | pairs << 10 | l1 << 14 | last of its l1 << 19
    const VjpItem *items;
    unsigned long long *next;
    int *err;
    long long N, nitems, total;
    int Nc, Mv, Mw, ccell, rowb;
    int withhold;    // test: 1 = the tiles' barriers wait for an arrival that does not come
    unsigned magic;  // x = l * Nc -> l = high word of x * magic (Nc > 1)
    unsigned long long wait_ns;
};

__device__ __forceinline__ void vjp_dmma(double &c0, double &c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

#define VJP_ALIGN(x) (((x) + 15) / 16 * 16)
// bytes of one warp's shared memory: ring, F2, G2, tile list, barriers
__host__ __device__ constexpr int vjp_warp_bytes(int P, int rowb)
{
    return VJP_ALIGN(VJ_NST * 8 * rowb) + 2 * VJP_ALIGN(P * VJ_S * 8) + VJ_MAXT * 4 + VJP_ALIGN(VJ_NST * 8);
}

template <int P>
__global__ void __launch_bounds__(32 * VJ_WARPS, 1) k_vjp_mma(const __grid_constant__ VjpMmaArgs a)
{
    constexpr int KT = (P + 3) / 4;  // K steps
    constexpr unsigned ALL = 0xffffffffu;
    extern __shared__ __align__(128) unsigned char smem_all[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = lane & 3, r8 = lane >> 2;
    unsigned char *smem = smem_all + warp * vjp_warp_bytes(P, a.rowb);
    unsigned char *ring = smem;
    double *F2 = reinterpret_cast<double *>(smem + VJP_ALIGN(VJ_NST * 8 * a.rowb));  // f(c2+D, l2) per row
    double *G2 = F2 + VJP_ALIGN(P * VJ_S * 8) / 8;                                     // sums for it
    unsigned *tl = reinterpret_cast<unsigned *>(G2 + VJP_ALIGN(P * VJ_S * 8) / 8);
    uint64_t *full = reinterpret_cast<uint64_t *>(tl + VJ_MAXT);
    if (lane == 0) {
        for (int s = 0; s < VJ_NST; s++) mbar_init(&full[s], 1 + a.withhold);
        fence_mbar_init();
    }
    __syncwarp();
    auto node = [&](int x) { return a.Nc > 1 ? (int)__umulhi((unsigned)x, a.magic) : x; };
    int slot = 0, phase = 0;
    bool ok = true;
    unsigned long long id = 0;
    if (lane == 0) id = atomicAdd(a.next, 1ULL);
    id = __shfl_sync(ALL, id, 0);
    while (id < (unsigned long long)a.total && ok) {
        const long long v = (long long)(id / (unsigned long long)a.nitems);
        const VjpItem im = a.items[id - (unsigned long long)v * a.nitems];
        const BlockInfo bi = a.blk[im.block];
        const int t0 = a.tfirst[im.block], nt = a.tfirst[im.block + 1] - t0;
        const int o1c = bi.c1 - a.ccell, o2c = bi.c2 - a.ccell;
        for (int t = lane; t < nt; t += 32) tl[t] = __ldg(a.tiles + t0 + t);
        __syncwarp();
        int sent = 0, sslot = slot;
        auto send = [&]() {  // the next tile's rows into the ring
            if (sent >= nt) return;
            if (lane == 0) {
                const unsigned x = tl[sent];
                const int n = (int)(x >> 10 & 15u);
                mbar_arrive_expect_tx(&full[sslot], (uint32_t)(n * a.rowb));
                bulk_g2s(ring + sslot * 8 * a.rowb, a.rows + (size_t)(bi.start + (x & 1023u)) * a.rowb,
                         (uint32_t)(n * a.rowb), &full[sslot]);
            }
            sent++;
            sslot = sslot + 1 == VJ_NST ? 0 : sslot + 1;
        };
        for (int s = 0; s < VJ_NST; s++) send();
        // rows: lane l has the cell of row l
        int D = 0;
        {
            const int r = im.row0 + min(lane, im.nrow - 1), lw = bi.hi[2] - bi.lo[2] + 1, lv = bi.hi[1] - bi.lo[1] + 1;
            const int w = r % lw, y = r / lw;
            D = ((bi.lo[0] + y / lv) * a.Mv + bi.lo[1] + y % lv) * a.Mw + bi.lo[2] + w;
        }
        const double *f = a.f + v * a.N, *cv = a.c + v * a.N;
        // f of cell c2 + D of every row, node-major; rows past the last are zero
#pragma unroll 4
        for (int r = 0; r < 8 * VJ_NT; r++) {
            const int Dr = __shfl_sync(ALL, D, r);
            if (lane < P) {
                F2[lane * VJ_S + r] = r < im.nrow ? __ldg(f + (size_t)(Dr + o2c) * P + lane) : 0.0;
                G2[lane * VJ_S + r] = 0.0;
            }
        }
        // A fragments: c of row 8 i + r8, node q + 4 t
        double cf[VJ_NT][KT];
        long long n1[VJ_NT];  // first node of cell c1 + D of this lane's rows; -1: no row
#pragma unroll
        for (int i = 0; i < VJ_NT; i++) {
            const int Dr = __shfl_sync(ALL, D, 8 * i + r8);
            n1[i] = 8 * i + r8 < im.nrow ? (long long)(Dr + o1c) * P : -1;
#pragma unroll
            for (int t = 0; t < KT; t++)
                cf[i][t] = 8 * i + r8 < im.nrow && q + 4 * t < P ? __ldg(cv + (size_t)Dr * P + q + 4 * t) : 0.0;
        }
        __syncwarp();
        double *g = a.g + v * a.N;
        double y1[VJ_NT], f1[VJ_NT];
        bool fresh = true;  // the next tile begins an l1
        int t = 0;
        for (; t < nt; t++) {
            const bool got = mbar_wait(&full[slot], (uint32_t)phase, a.err, a.wait_ns);
            if (!__all_sync(ALL, got)) { ok = false; break; }
            const unsigned x = tl[t];
            const int n = (int)(x >> 10 & 15u), l1 = (int)(x >> 14 & 31u);
            const unsigned char *rows = ring + slot * 8 * a.rowb;
            if (fresh) {
#pragma unroll
                for (int i = 0; i < VJ_NT; i++) {
                    f1[i] = n1[i] >= 0 ? __ldg(f + n1[i] + l1) : 0.0;
                    y1[i] = 0.0;
                }
            }
            // V fragments: pair r8, node q + 4 k (past P the row's last: times a zero of cf)
            const double *vr = reinterpret_cast<const double *>(rows + min(r8, n - 1) * a.rowb) + 1;
            double b[KT];
#pragma unroll
            for (int k = 0; k < KT; k++) b[k] = vr[4 * k + 4 > P ? min(q + 4 * k, P - 1) : q + 4 * k];
            // nodes l2 of the pairs 2 q, 2 q + 1 (this lane's columns)
            const bool p0 = 2 * q < n, p1 = 2 * q + 1 < n;
            const int l20 = node(reinterpret_cast<const int *>(rows + min(2 * q, n - 1) * a.rowb)[1] - o2c) * VJ_S + r8;
            const int l21 = node(reinterpret_cast<const int *>(rows + min(2 * q + 1, n - 1) * a.rowb)[1] - o2c) * VJ_S + r8;
            double acc[VJ_NT][2];
#pragma unroll
            for (int i = 0; i < VJ_NT; i++) acc[i][0] = acc[i][1] = 0.0;
#pragma unroll
            for (int k = 0; k < KT; k++)
#pragma unroll
                for (int i = 0; i < VJ_NT; i++) vjp_dmma(acc[i][0], acc[i][1], cf[i][k], b[k]);
            if (p0) {
#pragma unroll
                for (int i = 0; i < VJ_NT; i++) {
                    y1[i] = fma(acc[i][0], F2[l20 + 8 * i], y1[i]);
                    G2[l20 + 8 * i] = fma(acc[i][0], f1[i], G2[l20 + 8 * i]);
                }
            }
            if (p1) {
#pragma unroll
                for (int i = 0; i < VJ_NT; i++) {
                    y1[i] = fma(acc[i][1], F2[l21 + 8 * i], y1[i]);
                    G2[l21 + 8 * i] = fma(acc[i][1], f1[i], G2[l21 + 8 * i]);
                }
            }
            fresh = (x >> 19 & 1u) != 0;
            if (fresh) {  // the l1 ends
#pragma unroll
                for (int i = 0; i < VJ_NT; i++) {
                    y1[i] += __shfl_xor_sync(ALL, y1[i], 1);
                    y1[i] += __shfl_xor_sync(ALL, y1[i], 2);
                    if (q == 0 && n1[i] >= 0) atomicAdd(g + n1[i] + l1, y1[i]);
                }
            }
            if (++slot == VJ_NST) {
                slot = 0;
                phase ^= 1;
            }
            __syncwarp();  // G2 of this tile before the next one's; the rows are read
            send();
        }
        if (!ok) {  // let the copies still in flight land: those of the tiles t .. sent - 1
            for (; t < sent; t++) {
                mbar_wait(&full[slot], (uint32_t)phase, a.err, a.wait_ns);
                if (++slot == VJ_NST) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            break;
        }
        if (lane == 0) id = atomicAdd(a.next, 1ULL);
        for (int r = 0; r < im.nrow; r++) {
            const int Dr = __shfl_sync(ALL, D, r);
            if (lane < P) {
                const double y = G2[lane * VJ_S + r];
                if (y != 0.0) atomicAdd(g + (size_t)(Dr + o2c) * P + lane, y);
            }
        }
        __syncwarp();
        id = __shfl_sync(ALL, id, 0);
    }
}

// c = 2 v / w
__global__ void k_vjp_c(const double *v, const double *w, double *c, long long N, long long n)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        c[i] = 2.0 * v[i] / w[i % N];
}

// tiles of a block: its pairs (sorted by l1) cut at every change of l1 and into
// eights; tiles == nullptr counts them
__global__ void k_vjp_tiles(const BlockInfo *blk, const double *rows64, int RD64, int Nc, int ccell, int P, int *count,
                            const int *first, unsigned *tiles)
{
    __shared__ int n[32];
    const BlockInfo b = blk[blockIdx.x];
    if (threadIdx.x < 32) n[threadIdx.x] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < b.count; k += blockDim.x) {
        const long long o = __double_as_longlong(rows64[(size_t)(b.start + k) * RD64]);
        atomicAdd(&n[((int)(unsigned)(o & 0xffffffffLL) - (b.c1 - ccell)) / Nc], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0, t = tiles ? first[blockIdx.x] : 0;
        for (int l = 0; l < P; l++) {
            for (int k = 0; k < n[l]; k += 8, t++)
                if (tiles)
                    tiles[t] = (unsigned)(s + k) | (unsigned)min(8, n[l] - k) << 10 | (unsigned)l << 14 |
                               (k + 8 >= n[l] ? 1u : 0u) << 19;
            s += n[l];
        }
        if (!tiles) count[blockIdx.x] = t;
    }
}

// tiles and items of the layout: built on the first adjoint call
static int vjp_prepare(Ctx *c)
{
    Layout &L = c->lay;
    if (L.vjp_items) return DGV_OK;
    const Grid &g = c->grid;
    const int nb = (int)L.nblocks;
    std::vector<int> cnt(nb), first(nb + 1, 0);
    int *d_cnt = nullptr, *d_first = nullptr;
    unsigned *d_tiles = nullptr;
    void *d_items = nullptr;
    std::vector<VjpItem> items;
    cudaError_t e = cudaMalloc(&d_cnt, sizeof(int) * std::max(1, nb));
    if (e == cudaSuccess && nb) {
        k_vjp_tiles<<<(unsigned)nb, 128, 0, c->stream>>>(L.blk, (const double *)L.rows64, L.RD64, g.Nc, g.ccell, g.P, d_cnt,
                                                         nullptr, nullptr);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(cnt.data(), d_cnt, sizeof(int) * nb, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    }
    if (e == cudaSuccess) {
        for (int b = 0; b < nb; b++) first[b + 1] = first[b] + cnt[b];
        std::vector<int> order(nb);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cnt[x] > cnt[y]; });
        for (int b : order) {
            const BlockInfo &bi = L.h_blk[b];
            int n = 1;
            for (int d = 0; d < 3; d++) n *= std::max(0, bi.hi[d] - bi.lo[d] + 1);
            const int tiles = (n + 7) / 8, ni = (tiles + VJ_NT - 1) / VJ_NT;
            for (int k = 0, t0 = 0; k < ni; k++) {
                const int t1 = (int)((long long)tiles * (k + 1) / ni);
                items.push_back(VjpItem{b, 8 * t0, std::min(8 * (t1 - t0), n - 8 * t0), 0});
                t0 = t1;
            }
        }
        e = cudaMalloc(&d_first, sizeof(int) * (nb + 1));
    }
    if (e == cudaSuccess) e = cudaMalloc(&d_tiles, sizeof(unsigned) * std::max(1, first[nb]));
    if (e == cudaSuccess) e = cudaMalloc(&d_items, sizeof(VjpItem) * std::max<size_t>(1, items.size()));
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_first, first.data(), sizeof(int) * (nb + 1), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess && nb) {
        k_vjp_tiles<<<(unsigned)nb, 128, 0, c->stream>>>(L.blk, (const double *)L.rows64, L.RD64, g.Nc, g.ccell, g.P, nullptr,
                                                         d_first, d_tiles);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_items, items.data(), sizeof(VjpItem) * items.size(), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    cudaFree(d_cnt);
    if (e != cudaSuccess) {
        cudaGetLastError();
        cudaFree(d_first);
        cudaFree(d_tiles);
        cudaFree(d_items);
        return set_err(c, e == cudaErrorMemoryAllocation ? DGV_ENOMEM : DGV_ECUDA,
                       std::string("vjp: work list: ") + cudaGetErrorString(e));
    }
    L.vjp_first = d_first;
    L.vjp_tiles = d_tiles;
    L.vjp_items = d_items;
    L.vjp_nitems = (long long)items.size();
    return DGV_OK;
}

// Scratch of one launch at most: 2 N doubles per VDF are 426 VDFs at 27^3,
// seconds of work, beside which another launch's start is nothing
constexpr long long VJ_SCRATCH = 128LL << 20;

static int vjp_mma_launch(Ctx *c, const double *d_f, const double *d_v, double *d_g, int nvdf);

int vjp_mma_device(Ctx *c, const double *d_f, const double *d_v, double *d_g, int nvdf)
{
    if (!c->lay.blk) return set_err(c, DGV_ESTATE, "vjp: no A-arrays loaded");
    const Grid &g = c->grid;
    if (g.N > INT32_MAX / 2) return set_err(c, DGV_EUNSUP, "vjp: grid too large");
    int rc = vjp_prepare(c);
    if (rc) return rc;
    if ((rc = ensure_errflag(c))) return rc;
    const long long most = std::max<long long>(1, VJ_SCRATCH / (16 * g.N));
    for (long long v = 0; v < nvdf; v += most) {
        const long long at = v * g.N;
        if ((rc = vjp_mma_launch(c, d_f + at, d_v + at, d_g + at, (int)std::min(most, nvdf - v)))) return rc;
    }
    return DGV_OK;
}

static int vjp_mma_launch(Ctx *c, const double *d_f, const double *d_v, double *d_g, int nvdf)
{
    const Grid &g = c->grid;
    const Layout &L = c->lay;
    int rc;
    const long long n = (long long)nvdf * g.N;
    // the sums (f, v and g of the caller may be one array), the item counter, c
    if ((rc = ensure_buffer(c, &c->d_glm, &c->glm_bytes, sizeof(double) * (size_t)(2 * n + 1)))) return rc;
    double *acc = c->d_glm, *cv = c->d_glm + n + 1;
    int nsm = 148;
    DGV_CUDA(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    DGV_CUDA(c, cudaMemsetAsync(acc, 0, sizeof(double) * (size_t)(n + 1), c->stream));
    k_vjp_c<<<(unsigned)std::min<long long>((n + 255) / 256, 148LL * 16), 256, 0, c->stream>>>(d_v, c->d_nwt, cv, g.N, n);
    DGV_CUDA(c, cudaGetLastError());
    VjpMmaArgs a;
    std::memset(&a, 0, sizeof(a));
    a.f = d_f; a.c = cv; a.g = acc; a.blk = L.blk; a.rows = (const char *)L.rows64;
    a.tfirst = (const int *)L.vjp_first; a.tiles = (const unsigned *)L.vjp_tiles; a.items = (const VjpItem *)L.vjp_items;
    a.next = reinterpret_cast<unsigned long long *>(acc + n);
    a.err = c->d_err; a.N = g.N; a.nitems = L.vjp_nitems; a.total = L.vjp_nitems * nvdf;
    a.Nc = g.Nc; a.Mv = g.d.Mv; a.Mw = g.d.Mw; a.ccell = g.ccell; a.rowb = L.RD64 * 8;
    a.magic = g.Nc > 1 ? (unsigned)((1ULL << 32) / (unsigned)g.Nc + 1) : 0u;
    a.wait_ns = wait_limit_ns(c);
    a.withhold = c->test_withhold ? 1 : 0;
    c->test_withhold = false;
    const size_t smem = (size_t)VJ_WARPS * vjp_warp_bytes(g.P, a.rowb);
    auto fn = g.P == 27 ? k_vjp_mma<27> : k_vjp_mma<8>;
    DGV_CUDA(c, cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long ctas = std::min<long long>(nsm, (a.total + VJ_WARPS - 1) / VJ_WARPS);
    if (ctas > 0) {
        fn<<<(unsigned)ctas, 32 * VJ_WARPS, smem, c->stream>>>(a);
        DGV_CUDA(c, cudaGetLastError());
    }
    DGV_CUDA(c, cudaMemcpyAsync(d_g, acc, sizeof(double) * (size_t)n, cudaMemcpyDeviceToDevice, c->stream));
    count_launches(c, 2);
    return DGV_OK;
}

}  // namespace dgv
