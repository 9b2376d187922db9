// collide_mma.cu -- Q(f,f) and its mixed terms in FP64 on the double-precision
// tensor instructions (grids of 8 or 27 nodes per cell).
//
// For the blocks (cell pairs) that share one box of output cells, the operator
// is one matrix product with the pairs of all those blocks as its inner index:
//   Q[D, p] += sum_k X[D, k] V[k, p],
//   X[D, k] = f(o1_k + D) f(o2_k + D),   V[k, p] = A value of basis function p.
// At 27^3 the 151,854 blocks have 8,775 distinct boxes; a box holds 11,000
// pairs and 205 cells (averages weighted by work).  A unit of work is a box
// and up to 64 of its cells (rows); rows are the box's cells counted off in
// node order, so almost no lane works for a cell outside the box: 98 % of the
// rows of the 8-row tiles are live at 27^3, 90 % at 15^3 (one cell per lane,
// as in collide.cu: 41 % of the lanes).
//
// mma.m8n8k4 (FP64): one lane forms X of one (row, pair) -- two shared-memory
// gathers and a product -- and the warp multiplies it with ceil(P/8) column
// tiles of V; a V fragment is read once for up to 8 row tiles.  The
// instruction does the work of 8 multiply-adds per lane without operand
// traffic in between: 36.8 TFLOP/s measured alone, DFMA 28; the lane-wise
// kernel reached 3.9, each of its multiply-adds needing a broadcast
// shared-memory read.
//
// A CTA (8 warps) works through a range of (unit, stage); a stage is 16 pairs
// of the box, fetched by one bulk copy per block it draws on.  Stages go round
// robin to the warps, each warp streaming its own through a ring; at the end
// of a unit the warps' sums are added in a fixed order and once into the CTA's
// partial Q.  Ranges hold equal work and may be cut anywhere, so one wave of
// CTAs is balanced (the longest within 2.6 % of the mean at 27^3, 5 to 6 % at
// 15^3 and 21^3 and at 20^3 with eight nodes, whose costs are those of 27);
// k_reduce_partials adds the ranges in a fixed order: results are the same
// from run to run.
//
// What bounds it (B200, 1965 MHz): the FP64 tensor pipe, 80 % busy at 27^3,
// 76 % at 21^3, 67 % at 15^3 (148 ranges of three boxes each, and 680 cycles a
// tile at a unit's end).  A stage of 8 tiles takes 605 SM cycles, 512 of them
// products; the rest is the gathers' latency, which two warps per scheduler
// hide but for those 93.  Tried: explicit double buffering of the gathers
// across steps and stages (620-730, more registers and spills), 12 warps of 6
// or 5 tiles and 16 of 4 (the same share), 32 pairs a stage (2 % faster, no
// room at 27^3).  Per VDF, one lane per cell -> this kernel: 27^3 129.7 -> 20.1
// ms, 21^3 mixed terms 32.1 -> 3.2 ms, 15^3 with projection 1.95 -> 0.285 ms.
// Eight nodes per cell leave one column tile per product: shared-memory
// gathers bound it (20^3: 31 % of the tensor pipe, 60 % of shared memory's
// words; 13.5 -> 2.7 ms per VDF).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "dgv_internal.h"
#include "pipeline.cuh"

namespace dgv {

constexpr int MM_WARPS = 8;
constexpr int MM_THREADS = 32 * MM_WARPS;
constexpr int MM_SP = 16;    // pairs per stage
constexpr int MM_MT = 8;     // row tiles of 8 per unit
constexpr int MM_MAXST = 4;  // ring stages per warp, at most
// One box of output cells and up to 8 * MM_MT of its cells: rows row0 ..
// row0 + nrow - 1 of the box's cells in node order (u outer, w inner); the
// stages [stage0, stage1) hold the pairs of all blocks with this box.
struct __align__(16) MmaUnit {
    int stage0, stage1;
    int row0, nrow;
    signed char lo[3], len[3];
    short pad;
    int pad2[2];
};

struct MmaArgs {
    const double *f, *g;    // [nvdf][N]; g: second argument of the mixed terms
    const double *fg, *gg;  // local-major copies in global memory (GF)
    double *partial;        // [nvdf][nchunks][(cell1 - cell0) * P]
    const char *rows;
    const unsigned long long *segs;  // first pair << 16 | place in its stage << 8 | pairs
    const int *sfirst;               // per stage: its first segment
    const MmaUnit *units;
    const int2 *bounds;     // [nchunks + 1]: unit, stage
    int *err;
    long long N;
    int Nc, Mv, Mw, nchunks, cell0, ncell, rowb, nst;
    int part_smem, red_tiles;
    int off_f, off_g, off_part, off_red, off_bar;  // shared-memory layout (bytes)
    unsigned long long wait_ns;
};

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// the cell of row r of a box
__device__ __forceinline__ int mma_cell(const MmaUnit &u, int r, int Mv, int Mw)
{
    const int w = r % u.len[2], t = r / u.len[2], v = t % u.len[1], x = t / u.len[1];
    return ((u.lo[0] + x) * Mv + u.lo[1] + v) * Mw + u.lo[2] + w;
}

// Walks the stages of one warp: every W-th stage of every unit of the
// CTA's range.
template <int W>
struct MmaWalk {
    int u, s, end;
    __device__ __forceinline__ void enter(const MmaArgs &a, int2 b0, int2 b1, int warp)
    {
        for (; u <= b1.x; u++) {
            const int lo = u == b0.x ? b0.y : a.units[u].stage0;
            end = u == b1.x ? b1.y : a.units[u].stage1;
            s = lo + warp;
            if (s < end) return;
        }
    }
    __device__ __forceinline__ void next(const MmaArgs &a, int2 b0, int2 b1, int warp)
    {
        s += W;
        if (s < end) return;
        u++;
        enter(a, b0, b1, warp);
    }
};

__device__ __forceinline__ double lds_f64(uint32_t addr)
{
    double x;
    asm("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(addr));
    return x;
}

// Where f (and g) of the VDF are gathered from, by the offsets of a row plus
// the place of an output cell: local-major copies in shared memory (offsets in
// bytes) or in global memory (GF; offsets in elements).
template <bool GF>
struct MmaF {
    uint32_t f_s, g_s;
    const double *f, *g;
    __device__ __forceinline__ int scaled(int o) const { return GF ? o : 8 * o; }
    __device__ __forceinline__ double fat(int q) const
    {
        if constexpr (GF) return __ldg(f + q);
        else return lds_f64(f_s + q);
    }
    __device__ __forceinline__ double gat(int q) const
    {
        if constexpr (GF) return __ldg(g + q);
        else return lds_f64(g_s + q);
    }
};

// One warp's stages: walks its range, keeps the ring of bulk copies full (one
// copy per segment of a stage, lane k the k-th), and hands the stages out.  A
// stage's segments are loaded one stage before their use, their range two
// before: no load is waited for where it is issued.
template <int W>
struct MmaFetch {
    unsigned char *ring;
    uint64_t *full;
    volatile int *cnt;
    int2 b0, b1;
    MmaWalk<W> pw;
    unsigned long long ent = 0;    // this lane's segment of the next stage to issue
    int nseg = 0, s0 = 0, s1 = 0;  // its segments; segment range of the stage after it
    bool have = false, have2 = false, ok = true;
    int warp, lane, islot = 0, cslot = 0, cphase = 0, inflight = 0;

    __device__ __forceinline__ MmaFetch(const MmaArgs &a, unsigned char *smem, int w, int2 from, int2 to)
        : b0(from), b1(to), warp(w), lane(threadIdx.x & 31)
    {
        ring = smem + warp * a.nst * MM_SP * a.rowb;
        full = reinterpret_cast<uint64_t *>(smem + a.off_bar) + warp * MM_MAXST;
        cnt = reinterpret_cast<volatile int *>(smem + a.off_bar + W * MM_MAXST * 8) + warp * MM_MAXST;
        if (lane == 0) {
            for (int s = 0; s < a.nst; s++) mbar_init(&full[s], 1);
            fence_mbar_init();
        }
        __syncwarp();
        pw.u = b0.x;
        pw.enter(a, b0, b1, warp);
        advance(a);
        advance(a);
        for (int s = 0; s < a.nst; s++) issue(a);
    }
    __device__ __forceinline__ void advance(const MmaArgs &a)
    {
        have = have2;
        nseg = s1 - s0;
        if (have && lane < nseg) ent = __ldg(a.segs + s0 + lane);
        have2 = pw.u <= b1.x;
        if (have2) {
            s0 = __ldg(a.sfirst + pw.s);
            s1 = __ldg(a.sfirst + pw.s + 1);
            pw.next(a, b0, b1, warp);
        }
    }
    __device__ __forceinline__ void issue(const MmaArgs &a)
    {
        if (!have) return;
        const int off = (int)(ent >> 8 & 255ULL), len = (int)(ent & 255ULL);
        const int n = __shfl_sync(0xffffffffu, off + len, nseg - 1);
        if (lane == 0) {
            cnt[islot] = n;
            mbar_arrive_expect_tx(&full[islot], (uint32_t)(n * a.rowb));
        }
        if (lane < nseg)
            bulk_g2s(ring + (islot * MM_SP + off) * a.rowb, a.rows + (size_t)(ent >> 16) * a.rowb,
                     (uint32_t)(len * a.rowb), &full[islot]);
        inflight++;
        islot = islot + 1 == a.nst ? 0 : islot + 1;
        advance(a);
    }
    // waits for the next stage: n = its pairs; false once a wait has given up
    __device__ __forceinline__ bool wait(const MmaArgs &a, int &n)
    {
        if (ok) {
            const bool got = mbar_wait(&full[cslot], cphase, a.err, a.wait_ns);
            ok = __all_sync(0xffffffffu, got);
        }
        if (ok) n = cnt[cslot];
        return ok;
    }
    __device__ __forceinline__ const unsigned char *stage(const MmaArgs &a) const { return ring + cslot * MM_SP * a.rowb; }
    // done with it: its slot takes the next copy
    __device__ __forceinline__ void done(const MmaArgs &a)
    {
        inflight--;
        if (++cslot == a.nst) {
            cslot = 0;
            cphase ^= 1;
        }
        __syncwarp();  // every lane has read the slot
        issue(a);
    }
    // after a wait that gave up: let the copies already issued land
    __device__ __forceinline__ void drain(const MmaArgs &a)
    {
        if (ok) return;
        for (; inflight > 0; inflight--) {
            mbar_wait(&full[cslot], cphase, a.err, a.wait_ns);
            if (++cslot == a.nst) {
                cslot = 0;
                cphase ^= 1;
            }
        }
    }
};

// Adds the n pairs of one stage for NT row tiles.  Lane l: row l/4 of every
// tile, pair l%4 of every step of four pairs; V fragments: that pair, column
// l/4 of every column tile.  FULL: n = MM_SP, all steps unrolled; else pairs
// past n multiply zero with zero.
template <int P, int NT, bool FULL, bool BIL, bool GF>
__device__ __forceinline__ void mma_stage(const unsigned char *st, int n, int rowb, const int *doff,
                                          double (*acc)[(P + 7) / 8][2], const MmaF<GF> &F)
{
    constexpr int NTN = (P + 7) / 8;
    const int lane = threadIdx.x & 31, kq = lane & 3, cq = lane >> 2;
    const int cl = 8 * (NTN - 1) + cq < P ? 8 * (NTN - 1) + cq : P - 1;  // columns past P repeat the last (not stored)
#pragma unroll(FULL ? 4 : 1)
    for (int k0 = 0; k0 < (FULL ? MM_SP : n); k0 += 4) {
        const bool live = FULL || k0 + kq < n;
        const unsigned char *row = st + (live ? k0 + kq : 0) * rowb;
        const int2 o = *reinterpret_cast<const int2 *>(row);
        const int a1 = F.scaled(o.x), a2 = F.scaled(o.y);
        double b[NTN], x[NT];
#pragma unroll
        for (int i = 0; i < NT; i++) {
            const int q1 = a1 + doff[i], q2 = a2 + doff[i];
            if constexpr (BIL) x[i] = fma(F.gat(q1), F.fat(q2), F.fat(q1) * F.gat(q2));
            else x[i] = F.fat(q1) * F.fat(q2);
        }
        const double *r = reinterpret_cast<const double *>(row) + 1;
#pragma unroll
        for (int t = 0; t < NTN; t++) b[t] = r[t == NTN - 1 ? cl : 8 * t + cq];
        if (!FULL && !live) {
#pragma unroll
            for (int i = 0; i < NT; i++) x[i] = 0.0;
#pragma unroll
            for (int t = 0; t < NTN; t++) b[t] = 0.0;
        }
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int t = 0; t < NTN; t++) dmma(acc[i][t][0], acc[i][t][1], x[i], b[t]);
    }
}

// BIL: the mixed terms 2/w sum A (f g + g f).  GF: f (and g) gathered from
// local-major copies in global memory instead of shared memory, for grids
// where they do not fit; the sums are the same bit for bit.
template <int P, bool BIL, bool GF>
__global__ void __launch_bounds__(MM_THREADS, 1) k_collide_mma(const __grid_constant__ MmaArgs a)
{
    constexpr int NTN = (P + 7) / 8, CW = 8 * NTN;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int vdf = blockIdx.x, chunk = blockIdx.y;
    double *f_s = reinterpret_cast<double *>(smem + a.off_f), *g_s = reinterpret_cast<double *>(smem + a.off_g);
    double *red = reinterpret_cast<double *>(smem + a.off_red);  // [red_tiles][MM_WARPS][8][CW]
    __shared__ int rowcell[8 * MM_MT];
    // the CTA's partial Q: in shared memory where that has room
    double *part = a.part_smem ? reinterpret_cast<double *>(smem + a.off_part)
                               : a.partial + ((size_t)vdf * a.nchunks + chunk) * ((size_t)a.ncell * P);
    MmaFetch<MM_WARPS> fetch(a, smem, warp, a.bounds[chunk], a.bounds[chunk + 1]);

    if constexpr (!GF) {
        const double *f = a.f + (size_t)vdf * a.N;
        for (int i = threadIdx.x; i < (int)a.N; i += MM_THREADS) {
            const int cell = i / P, l = i - cell * P;
            f_s[l * a.Nc + cell] = __ldg(f + i);
        }
        if constexpr (BIL) {
            const double *g = a.g + (size_t)vdf * a.N;
            for (int i = threadIdx.x; i < (int)a.N; i += MM_THREADS) {
                const int cell = i / P, l = i - cell * P;
                g_s[l * a.Nc + cell] = __ldg(g + i);
            }
        }
    }
    for (int i = threadIdx.x; i < a.ncell * P; i += MM_THREADS) part[i] = 0.0;
    __syncthreads();
    MmaF<GF> F;
    F.f_s = smem_u32(f_s);
    F.g_s = smem_u32(g_s);
    F.f = GF ? a.fg + (size_t)vdf * a.N : nullptr;
    F.g = (GF && BIL) ? a.gg + (size_t)vdf * a.N : nullptr;

    for (int u = fetch.b0.x; u <= fetch.b1.x; u++) {
        const MmaUnit un = a.units[u];
        const int sa = u == fetch.b0.x ? fetch.b0.y : un.stage0, sb = u == fetch.b1.x ? fetch.b1.y : un.stage1;
        if (sa >= sb) continue;  // the same in every warp
        const int nt = (un.nrow + 7) / 8;
        // the rows' cells: lane l has rows l and l + 32; rows past the last
        // repeat it (they are not stored)
        const int ca = mma_cell(un, un.row0 + min(lane, un.nrow - 1), a.Mv, a.Mw);
        const int cb = mma_cell(un, un.row0 + min(lane + 32, un.nrow - 1), a.Mv, a.Mw);
        int doff[MM_MT];
#pragma unroll
        for (int i = 0; i < MM_MT; i++)
            doff[i] = F.scaled(__shfl_sync(0xffffffffu, i < 4 ? ca : cb, 8 * (i & 3) + (lane >> 2)));
        if (warp == 0) {  // read at the unit's end, after a barrier
            rowcell[lane] = ca - a.cell0;
            rowcell[lane + 32] = cb - a.cell0;
        }
        double acc[MM_MT][NTN][2];
#pragma unroll
        for (int i = 0; i < MM_MT; i++)
#pragma unroll
            for (int t = 0; t < NTN; t++) acc[i][t][0] = acc[i][t][1] = 0.0;
        // the stages of this warp: sa + warp, sa + warp + MM_WARPS, ...
        const int nmine = (sb - sa - warp + MM_WARPS - 1) / MM_WARPS;
#define DGV_MMA_CASE(NT)                                                                              \
    case NT:                                                                                          \
        for (int s = 0; s < nmine; s++) {                                                             \
            int n = 0;                                                                                \
            if (!fetch.wait(a, n)) break;                                                             \
            if (n == MM_SP) mma_stage<P, NT, true, BIL, GF>(fetch.stage(a), n, a.rowb, doff, acc, F); \
            else mma_stage<P, NT, false, BIL, GF>(fetch.stage(a), n, a.rowb, doff, acc, F);           \
            fetch.done(a);                                                                            \
        }                                                                                             \
        break;
        switch (nt) {
            DGV_MMA_CASE(1)
            DGV_MMA_CASE(2)
            DGV_MMA_CASE(3)
            DGV_MMA_CASE(4)
            DGV_MMA_CASE(5)
            DGV_MMA_CASE(6)
            DGV_MMA_CASE(7)
            DGV_MMA_CASE(8)
        }
#undef DGV_MMA_CASE
        // the warps' sums in warp order into the CTA's partial Q: a.red_tiles
        // tiles at a time; where the partial Q is in global memory one, with its
        // old values on their way before the first
        const int prow = threadIdx.x / P, pp = threadIdx.x - prow * P;
        double old[MM_MT];
        if (!a.part_smem) {
            __syncthreads();  // rowcell
#pragma unroll
            for (int i = 0; i < MM_MT; i++)
                old[i] = prow < 8 && 8 * i + prow < un.nrow ? part[(size_t)rowcell[8 * i + prow] * P + pp] : 0.0;
        }
        auto put = [&](int i, int at) {  // tile i's sums of this warp
            double *r = red + (size_t)((at * MM_WARPS + warp) * 8 + (lane >> 2)) * CW + 2 * (lane & 3);
#pragma unroll
            for (int t = 0; t < NTN; t++)
                *reinterpret_cast<double2 *>(r + 8 * t) = make_double2(acc[i][t][0], acc[i][t][1]);
        };
        auto sum = [&](int row, int p) {  // over the warps
            const double *r = red + (size_t)((row >> 3) * MM_WARPS * 8 + (row & 7)) * CW + p;
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < MM_WARPS; w++) s += r[(size_t)w * 8 * CW];
            return s;
        };
        if (a.part_smem) {
            for (int i0 = 0; i0 < nt; i0 += a.red_tiles) {
                const int i1 = min(nt, i0 + a.red_tiles), nrow = min(un.nrow - 8 * i0, 8 * (i1 - i0));
#pragma unroll
                for (int i = 0; i < MM_MT; i++)
                    if (i >= i0 && i < i1) put(i, i - i0);
                __syncthreads();
                for (int e = threadIdx.x; e < nrow * P; e += MM_THREADS) {
                    const int row = e / P, p = e - row * P;
                    part[rowcell[8 * i0 + row] * P + p] += sum(row, p);
                }
                __syncthreads();
            }
        } else {
#pragma unroll
            for (int i = 0; i < MM_MT; i++) {
                if (i >= nt) break;
                put(i, 0);
                __syncthreads();
                if (prow < 8 && 8 * i + prow < un.nrow)
                    part[(size_t)rowcell[8 * i + prow] * P + pp] = old[i] + sum(prow, pp);
                __syncthreads();
            }
        }
    }
    if (a.part_smem) {
        double *out = a.partial + ((size_t)vdf * a.nchunks + chunk) * ((size_t)a.ncell * P);
        for (int i = threadIdx.x; i < a.ncell * P; i += MM_THREADS) out[i] = part[i];
    }
    fetch.drain(a);
}

// ----------------------------------------------------------------------------
// FP32-compensated Q on the same units.  The arithmetic is that of the
// lane-wise kernel, sum for sum: FP32 products f(a) f(b), the 16-pair groups of
// a block summed by FP32 multiply-adds in pair order, group sums added with
// two-sum into (sum, correction); only the order of the group sums differs.
// A stage is one group.  The warp's 32 lanes are 4 column groups x 8 row
// groups: lane (pg, rg) keeps the sums of rows rg + 8j (j < A) and columns
// PB pg .. PB pg + PB - 1 (PB = ceil(P/4)), so that a pair costs it PB values
// and A products from shared memory or other lanes for A * PB multiply-adds:
// shared memory delivers one word per lane and cycle to one warp of the SM,
// which bounds a kernel with one row and all P columns per lane (32 words for
// 27 multiply-adds).  A product is formed by one of the four lanes that need
// it and handed on by shuffles.
// Rows are taken in pairs by packed FP32x2 operations (multiply-adds and the
// two-sum), half the instructions of scalar ones for the same roundings.
// Measured (B200): a stage of 64 rows takes 630 SM cycles (724 with scalar
// operations), 216 of them multiply-adds at the scalar rate; shared memory's
// and the shuffles' ~21 words per pair and their latency bound it (scalar: two
// rows and all columns per lane 655, but rows in steps of 32; 12 or 16 warps of
// 32 rows 405 per 32 rows).  Per Q at 21^3 with projection, one cell per lane ->
// this kernel: 18.3 -> 3.3 ms.  The FP64 kernel above has become the faster one
// all the same (one VDF, FP64 / FP32: 15^3 0.27 / 0.38 ms, 21^3 2.98 / 3.34,
// 27^3 20.4 / 23.0; eight nodes 14^3 0.24 / 0.29, 20^3 2.7 / 3.6).
constexpr int FC_WARPS = 8, FC_THREADS = 32 * FC_WARPS;
constexpr int FC_TILE = 16, FC_MT = 4;  // rows per tile (A = 2 per tile); tiles per unit

template <bool GF>
struct F32F {
    uint32_t f_s;
    const float *f;
    __device__ __forceinline__ int scaled(int o) const { return GF ? o : 4 * o; }
    __device__ __forceinline__ float fat(int q) const
    {
        if constexpr (GF) {
            return __ldg(f + q);
        } else {
            float x;
            asm("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(f_s + q));
            return x;
        }
    }
};

// the n pairs of one group added into (sum, correction); d1, d2: places of the
// cells whose products this lane forms (rows rg + 8 pg and rg + 8 pg + 32).
// Rows rg + 16 j and rg + 16 j + 8 share packed operations: each half rounds
// like the scalar one.
template <int P, int A, bool GF>
__device__ __forceinline__ void f32_stage(const unsigned char *st, int n, int d1, int d2, float2 (*sm)[(P + 3) / 4],
                                          float2 (*cr)[(P + 3) / 4], const F32F<GF> &F)
{
    constexpr int RB = ((2 + P) + 3) / 4 * 16;  // bytes of a row: offsets, values, zeros
    constexpr int PB = (P + 3) / 4;
    const int pg = threadIdx.x & 3;
    float2 part[A / 2][PB];
#pragma unroll
    for (int j = 0; j < A / 2; j++)
#pragma unroll
        for (int i = 0; i < PB; i++) part[j][i] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < n; k++) {
        const int2 o = *reinterpret_cast<const int2 *>(st + k * RB);
        const float *row = reinterpret_cast<const float *>(st + k * RB) + 2 + PB * pg;
        const int a1 = F.scaled(o.x), a2 = F.scaled(o.y);
        const float x1 = F.fat(a1 + d1) * F.fat(a2 + d1);
        const float x2 = A > 4 ? F.fat(a1 + d2) * F.fat(a2 + d2) : 0.f;
        float v[PB];
#pragma unroll
        for (int i = 0; i < PB; i++) v[i] = row[i];
#pragma unroll
        for (int j = 0; j < A; j += 2) {
            const float xl = j < 4 ? x1 : x2;
            const float2 x = make_float2(__shfl_sync(0xffffffffu, xl, j & 3, 4), __shfl_sync(0xffffffffu, xl, j + 1 & 3, 4));
#pragma unroll
            for (int i = 0; i < PB; i++) part[j / 2][i] = __ffma2_rn(make_float2(v[i], v[i]), x, part[j / 2][i]);
        }
    }
    const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll
    for (int j = 0; j < A / 2; j++)
#pragma unroll
        for (int i = 0; i < PB; i++) {  // two-sum: sum + correction carries the group sum exactly
            const float2 x = part[j][i], s = sm[j][i], t = __fadd2_rn(s, x), bp = __ffma2_rn(s, m1, t);
            const float2 e = __fadd2_rn(__ffma2_rn(__ffma2_rn(bp, m1, t), m1, s), __ffma2_rn(bp, m1, x));
            cr[j][i] = __fadd2_rn(cr[j][i], e);
            sm[j][i] = t;
        }
}

template <int P, bool GF>
__global__ void __launch_bounds__(FC_THREADS, 1) k_collide_f32(const __grid_constant__ MmaArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int rowcell[FC_TILE * FC_MT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int vdf = blockIdx.x, chunk = blockIdx.y, pg = lane & 3, rg = lane >> 2;
    constexpr int PB = (P + 3) / 4, CW = 4 * PB;
    float *f_s = reinterpret_cast<float *>(smem + a.off_f);
    double *red = reinterpret_cast<double *>(smem + a.off_red);  // [FC_WARPS][8][CW]
    double *part = a.part_smem ? reinterpret_cast<double *>(smem + a.off_part)
                               : a.partial + ((size_t)vdf * a.nchunks + chunk) * ((size_t)a.ncell * P);
    MmaFetch<FC_WARPS> fetch(a, smem, warp, a.bounds[chunk], a.bounds[chunk + 1]);
    if constexpr (!GF) {
        const double *f = a.f + (size_t)vdf * a.N;
        for (int i = threadIdx.x; i < (int)a.N; i += FC_THREADS) {
            const int cell = i / P, l = i - cell * P;
            f_s[l * a.Nc + cell] = (float)__ldg(f + i);
        }
    }
    for (int i = threadIdx.x; i < a.ncell * P; i += FC_THREADS) part[i] = 0.0;
    __syncthreads();
    F32F<GF> F;
    F.f_s = smem_u32(f_s);
    F.f = GF ? reinterpret_cast<const float *>(a.fg) + (size_t)vdf * a.N : nullptr;

    for (int u = fetch.b0.x; u <= fetch.b1.x; u++) {
        const MmaUnit un = a.units[u];
        const int sa = u == fetch.b0.x ? fetch.b0.y : un.stage0, sb = u == fetch.b1.x ? fetch.b1.y : un.stage1;
        if (sa >= sb) continue;  // the same in every warp
        const int nt = (un.nrow + FC_TILE - 1) / FC_TILE;
        // rows past the last repeat it (they are not stored)
        const int d1 = F.scaled(mma_cell(un, un.row0 + min(rg + 8 * pg, un.nrow - 1), a.Mv, a.Mw));
        const int d2 = F.scaled(mma_cell(un, un.row0 + min(rg + 8 * pg + 32, un.nrow - 1), a.Mv, a.Mw));
        if (warp < 2) {
            const int r = 32 * warp + lane;
            rowcell[r] = mma_cell(un, un.row0 + min(r, un.nrow - 1), a.Mv, a.Mw) - a.cell0;
        }
        float2 sm[FC_MT][PB], cr[FC_MT][PB];  // rows rg + 16 j, rg + 16 j + 8
#pragma unroll
        for (int j = 0; j < FC_MT; j++)
#pragma unroll
            for (int i = 0; i < PB; i++) sm[j][i] = cr[j][i] = make_float2(0.f, 0.f);
        const int nmine = (sb - sa - warp + FC_WARPS - 1) / FC_WARPS;
#define DGV_F32_CASE(NT)                                                    \
    case NT:                                                                \
        for (int s = 0; s < nmine; s++) {                                   \
            int n = 0;                                                      \
            if (!fetch.wait(a, n)) break;                                   \
            f32_stage<P, 2 * NT, GF>(fetch.stage(a), n, d1, d2, sm, cr, F); \
            fetch.done(a);                                                  \
        }                                                                   \
        break;
        switch (nt) {
            DGV_F32_CASE(1)
            DGV_F32_CASE(2)
            DGV_F32_CASE(3)
            DGV_F32_CASE(4)
        }
#undef DGV_F32_CASE
        // the warps' sums in FP64, eight rows at a time, in warp order, into
        // the CTA's partial Q
#pragma unroll
        for (int j = 0; j < 2 * FC_MT; j++) {
            if (8 * j >= un.nrow) break;
            const int row = threadIdx.x / P, p = threadIdx.x - row * P;
            const bool mine = row < 8 && 8 * j + row < un.nrow;
#pragma unroll
            for (int i = 0; i < PB; i++)
                red[(size_t)(warp * 8 + rg) * CW + PB * pg + i] =
                    j & 1 ? (double)sm[j / 2][i].y + (double)cr[j / 2][i].y : (double)sm[j / 2][i].x + (double)cr[j / 2][i].x;
            __syncthreads();
            if (mine) {
                double *dst = part + (size_t)rowcell[8 * j + row] * P + p;
                const double old = *dst;
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < FC_WARPS; w++) s += red[(size_t)(w * 8 + row) * CW + p];
                *dst = old + s;
            }
            __syncthreads();
        }
    }
    if (a.part_smem) {
        double *out = a.partial + ((size_t)vdf * a.nchunks + chunk) * ((size_t)a.ncell * P);
        for (int i = threadIdx.x; i < a.ncell * P; i += FC_THREADS) out[i] = part[i];
    }
    fetch.drain(a);
}

// q[v][i] = scale * (2 * sum_chunks partial[v][chunk][i]) / w[cell0*P + i]:
// eight threads share an output, each adding every eighth chunk; their sums
// are added in a fixed order
__global__ void __launch_bounds__(256) k_reduce_partials(const double *partial, const double *w, double *q, int nchunks,
                                                         long long len, int nvdf, double scale)
{
    __shared__ double sh[8][33];
    const long long per = (len + 31) / 32;
    const int v = (int)(blockIdx.x / per), x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const long long i = (blockIdx.x - (long long)v * per) * 32 + x;
    double s = 0.0;
    if (i < len) {
        const double *src = partial + (size_t)v * nchunks * len + i;
#pragma unroll 4
        for (int c = y; c < nchunks; c += 8) s += __ldg(src + (size_t)c * len);
    }
    sh[y][x] = s;
    __syncthreads();
    if (y == 0 && i < len) {
        for (int k = 1; k < 8; k++) s += sh[k][x];
        double val = 2.0 * s / w[i];
        if (scale != 1.0) val = val * scale;
        q[(size_t)v * len + i] = val;
    }
}

// ----------------------------------------------------------------------------
// The stage list of the layout (blocks sorted by box) and, per range of output
// cells, the units: built on first use and kept with the A-arrays.
static int mma_boxes(Ctx *c, MmaList &M, bool across)
{
    const Layout &L = c->lay;
    if (M.segs) return DGV_OK;
    std::vector<int> order(L.nblocks);
    std::iota(order.begin(), order.end(), 0);
    auto key = [&](int b) {
        const BlockInfo &bi = L.h_blk[b];
        unsigned long long k = 0;
        for (int d = 0; d < 3; d++) k = k << 16 | (unsigned long long)(unsigned char)bi.lo[d] << 8 | (unsigned char)bi.hi[d];
        return k;
    };
    std::vector<unsigned long long> keys(L.nblocks);
    for (long long b = 0; b < L.nblocks; b++) keys[b] = key((int)b);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return keys[x] < keys[y]; });
    // a box's pairs in block order, cut into stages of MM_SP: across blocks (a
    // segment for each block a stage draws on), or anew from each block's start
    std::vector<unsigned long long> seg;
    std::vector<int> sfirst;
    seg.reserve((size_t)(L.npairs / MM_SP + 2 * L.nblocks + 1));
    sfirst.reserve((size_t)(L.npairs / MM_SP + L.nblocks + 2));
    M.box.clear();
    int room = 0;  // pairs the open stage still takes
    for (long long i = 0; i < L.nblocks; i++) {
        const BlockInfo &bi = L.h_blk[order[i]];
        if (i == 0 || keys[order[i]] != keys[order[i - 1]]) {
            MmaBox bx;
            for (int d = 0; d < 3; d++) { bx.lo[d] = bi.lo[d]; bx.hi[d] = bi.hi[d]; }
            bx.stage0 = (long long)sfirst.size();
            M.box.push_back(bx);
            room = 0;
        }
        if (!across) room = 0;
        for (int o = 0; o < bi.count;) {
            if (room == 0) {
                sfirst.push_back((int)seg.size());
                room = MM_SP;
            }
            const int n = std::min(room, bi.count - o);
            seg.push_back((unsigned long long)(bi.start + o) << 16 | (unsigned long long)(MM_SP - room) << 8 |
                          (unsigned long long)n);
            room -= n;
            o += n;
        }
        M.box.back().stage1 = (long long)sfirst.size();
    }
    if (seg.size() > (size_t)INT32_MAX) return set_err(c, DGV_EUNSUP, "collide: too many pairs for the stage list");
    sfirst.push_back((int)seg.size());
    void *d = nullptr, *e = nullptr;
    cudaError_t rc = cudaMalloc(&d, std::max<size_t>(1, seg.size()) * sizeof(unsigned long long));
    if (rc == cudaSuccess) rc = cudaMalloc(&e, sfirst.size() * sizeof(int));
    if (rc == cudaSuccess) rc = upload(d, seg.data(), seg.size() * sizeof(unsigned long long));
    if (rc == cudaSuccess) rc = upload(e, sfirst.data(), sfirst.size() * sizeof(int));
    if (rc != cudaSuccess) {
        cudaGetLastError();
        cudaFree(d);
        cudaFree(e);
        return set_err(c, rc == cudaErrorMemoryAllocation ? DGV_ENOMEM : DGV_ECUDA,
                       std::string("collide: stage list: ") + cudaGetErrorString(rc));
    }
    M.segs = d;
    M.sfirst = e;
    return DGV_OK;
}

// Units of the boxes' cells in [cell0, cell1) (contiguous in a box's node
// order), tiles of `rows` cells spread evenly over a box's units.
struct MmaShape {
    int rows, tiles;                       // rows per tile, tiles per unit at most
    int c_tile, c_stage, c_unit, c_flush;  // costs (SM cycles, fitted): stage per tile, stage, unit, its end per tile
};

// Plans of slices of the output cells kept per list, the least recently used
// given up: a rank has one slice, a caller may walk through all Nc^2 / 2.  (A
// plan is 32 bytes per box on the device, 0.3 MB at 27^3, and a pass over the
// boxes to build.)  The whole grid's plan stays, which captured steps hold, and
// so do the plans that a caller's capture has recorded.
constexpr int MMA_SLICES = 64;

static int mma_make_room(Ctx *c, MmaList &M)
{
    for (;;) {
        auto old = M.plans.end();
        int n = 0;
        for (auto it = M.plans.begin(); it != M.plans.end(); ++it) {
            if (it->second.captured || it->first == std::make_pair(0, c->grid.Nc)) continue;
            n++;
            if (old == M.plans.end() || it->second.used < old->second.used) old = it;
        }
        if (n < MMA_SLICES) return DGV_OK;
        DGV_CUDA(c, cudaStreamSynchronize(c->stream));  // launches that read it
        free_plan(old->second);
        M.plans.erase(old);
    }
}

static int mma_plan(Ctx *c, MmaList &M, const MmaShape &S, int cell0, int cell1, MmaPlan **out)
{
    const Grid &g = c->grid;
    const std::pair<int, int> key(cell0, cell1);
    bool captured = false;
    if (key != std::make_pair(0, g.Nc)) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess) cudaGetLastError();
        captured = st != cudaStreamCaptureStatusNone;
    }
    M.clock++;
    auto it = M.plans.find(key);
    if (it != M.plans.end()) {
        it->second.used = M.clock;
        it->second.captured |= captured;
        *out = &it->second;
        return DGV_OK;
    }
    if (!captured) {
        const int rc = mma_make_room(c, M);
        if (rc) return rc;
    }
    std::vector<MmaUnit> units;
    MmaPlan pl;
    pl.cost.push_back(0);
    for (const MmaBox &bx : M.box) {
        const int len[3] = {bx.hi[0] - bx.lo[0] + 1, bx.hi[1] - bx.lo[1] + 1, bx.hi[2] - bx.lo[2] + 1};
        if (len[0] <= 0 || len[1] <= 0 || len[2] <= 0) continue;
        // rows of the box whose cell lies before `cell`
        auto before = [&](int cell) {
            int n = 0;
            for (int u = 0; u < len[0]; u++)
                for (int v = 0; v < len[1]; v++) {
                    const int first = ((bx.lo[0] + u) * g.d.Mv + bx.lo[1] + v) * g.d.Mw + bx.lo[2];
                    n += std::max(0, std::min(len[2], cell - first));
                }
            return n;
        };
        const int whole = len[0] * len[1] * len[2];
        const int r0 = cell0 > 0 ? before(cell0) : 0, r1 = cell1 < g.Nc ? before(cell1) : whole;
        const int tiles = (r1 - r0 + S.rows - 1) / S.rows, nu = (tiles + S.tiles - 1) / S.tiles;
        int t0 = 0;
        for (int k = 0; k < nu; k++) {
            const int t1 = (int)((long long)tiles * (k + 1) / nu);
            MmaUnit un;
            std::memset(&un, 0, sizeof(un));
            un.stage0 = (int)bx.stage0;
            un.stage1 = (int)bx.stage1;
            un.row0 = r0 + S.rows * t0;
            un.nrow = std::min(S.rows * (t1 - t0), r1 - un.row0);
            for (int d = 0; d < 3; d++) { un.lo[d] = (signed char)bx.lo[d]; un.len[d] = (signed char)len[d]; }
            units.push_back(un);
            pl.per_stage.push_back(S.c_tile * (t1 - t0) + S.c_stage);
            pl.cost.push_back(pl.cost.back() + (long long)pl.per_stage.back() * (un.stage1 - un.stage0) + S.c_unit +
                              S.c_flush * (t1 - t0));
            pl.first.push_back(un.stage0);
            pl.last.push_back(un.stage1);
            t0 = t1;
        }
    }
    pl.nunits = (int)units.size();
    pl.used = M.clock;
    pl.captured = captured;
    DGV_CUDA(c, cudaMalloc(&pl.units, std::max<size_t>(1, units.size()) * sizeof(MmaUnit)));
    const cudaError_t e = upload(pl.units, units.data(), units.size() * sizeof(MmaUnit));
    if (e != cudaSuccess) {
        cudaFree(pl.units);
        return set_err(c, DGV_ECUDA, std::string("collide plan: ") + cudaGetErrorString(e));
    }
    *out = &(M.plans[key] = std::move(pl));
    return DGV_OK;
}

// (unit, stage) bounds of nchunks ranges of equal cost
static int mma_bounds(Ctx *c, MmaPlan *pl, int nchunks, const int2 **out)
{
    auto it = pl->bounds.find(nchunks);
    if (it != pl->bounds.end()) { *out = reinterpret_cast<const int2 *>(it->second); return DGV_OK; }
    std::vector<int2> b(nchunks + 1);
    const long long tot = pl->cost.back();
    const int last = std::max(0, pl->nunits - 1);
    int u = 0;
    for (int k = 0; k <= nchunks; k++) {
        const long long at = (long long)((double)tot * k / nchunks);
        while (u < last && pl->cost[u + 1] <= at) u++;
        if (pl->nunits == 0) b[k] = make_int2(0, 0);
        else if (k == nchunks) b[k] = make_int2(last, pl->last[last]);
        else b[k] = make_int2(u, (int)std::min<long long>(pl->last[u], pl->first[u] + (at - pl->cost[u]) / pl->per_stage[u]));
    }
    void *d = nullptr;
    DGV_CUDA(c, cudaMalloc(&d, sizeof(int2) * b.size()));
    const cudaError_t e = upload(d, b.data(), sizeof(int2) * b.size());
    if (e != cudaSuccess) {
        cudaFree(d);
        return set_err(c, DGV_ECUDA, std::string("collide plan: ") + cudaGetErrorString(e));
    }
    pl->bounds[nchunks] = d;
    *out = reinterpret_cast<const int2 *>(d);
    return DGV_OK;
}

// Ranges per VDF: the smallest count whose CTAs fill the last wave to 99.5 % (one
// CTA per SM, all of equal cost), else the one that fills it best, with at
// least four stages per warp and at most four waves.
static int mma_chunks(int nsm, int nvdf, int warps, long long stages)
{
    int best = 1;
    double eff = 0.0;
    const int most = (int)std::max<long long>(1, std::min<long long>((4LL * nsm + nvdf - 1) / nvdf, stages / (4 * warps)));
    for (int k = 1; k <= most; k++) {
        const long long ctas = (long long)nvdf * k, waves = (ctas + nsm - 1) / nsm;
        const double e = (double)ctas / (double)(waves * nsm);
        if (e > eff + 1e-9) { eff = e; best = k; }
        if (eff >= 0.995) break;
    }
    return best;
}

// DGV_OPT_TEST_WITHHOLD: for one launch a segment of two pairs or more begins
// one pair later, so that its stage's barrier, which expects the bytes up to
// the last segment's end, waits for a pair that is not copied.  In the list and
// not in the kernel: one more operand of the barriers' set-up there cost 0.5 %
// at 27^3 (80.0 -> 80.4 ms for 4 VDFs).
struct MmaWithhold {
    unsigned long long *at = nullptr, was = 0;
    int take(Ctx *c, const MmaList &M)
    {
        c->test_withhold = false;
        int head[2] = {0, 0};
        DGV_CUDA(c, cudaMemcpyAsync(head, M.sfirst, sizeof(head), cudaMemcpyDeviceToHost, c->stream));
        DGV_CUDA(c, cudaStreamSynchronize(c->stream));
        std::vector<unsigned long long> seg(head[1] - head[0]);  // the first stage's
        unsigned long long *d = static_cast<unsigned long long *>(M.segs) + head[0];
        DGV_CUDA(c, cudaMemcpyAsync(seg.data(), d, seg.size() * sizeof(was), cudaMemcpyDeviceToHost, c->stream));
        DGV_CUDA(c, cudaStreamSynchronize(c->stream));
        for (size_t k = 0; k < seg.size() && !at; k++)
            if ((seg[k] & 255ULL) >= 2) {
                was = seg[k];
                at = d + k;
                const unsigned long long later = was + (1ULL << 16) + (1ULL << 8) - 1ULL;
                DGV_CUDA(c, cudaMemcpyAsync(at, &later, sizeof(later), cudaMemcpyHostToDevice, c->stream));
                DGV_CUDA(c, cudaStreamSynchronize(c->stream));
            }
        return DGV_OK;
    }
    int give_back(Ctx *c)
    {
        DGV_CUDA(c, cudaMemcpyAsync(at, &was, sizeof(was), cudaMemcpyHostToDevice, c->stream));
        DGV_CUDA(c, cudaStreamSynchronize(c->stream));
        return DGV_OK;
    }
};

typedef void (*MmaFn)(const MmaArgs);

template <int P>
static MmaFn mma_pick(bool f32, bool bil, bool gf)
{
    if (f32) return gf ? k_collide_f32<P, true> : k_collide_f32<P, false>;
    if (bil) return gf ? k_collide_mma<P, true, true> : k_collide_mma<P, true, false>;
    return gf ? k_collide_mma<P, false, true> : k_collide_mma<P, false, false>;
}

bool mma_serves(const Ctx *c) { return c->grid.P == 27 || c->grid.P == 8; }

// Q(f,f) in FP64 or FP32-compensated arithmetic, or with d_g the mixed terms
// of f and g in FP64, on the output cells [cell0, cell1)
int collide_mma_device(Ctx *c, const double *d_f, const double *d_g, double *d_q, int nvdf, int precision, double scale,
                       int cell0, int cell1)
{
    const Grid &g = c->grid;
    Layout &L = c->lay;
    const bool bil = d_g != nullptr, f32 = precision == DGV_PREC_F32C;
    int maxsm = 0, nsm = 148;
    DGV_CUDA(c, cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
    DGV_CUDA(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    if (g.N > INT32_MAX / 2) return set_err(c, DGV_EUNSUP, "collide: grid too large");  // gather indices are ints
    int rc;
    if (f32 && (rc = ensure_rows32(c))) return rc;  // rebuilt if released
    // costs fitted to the measured cycles of the ranges at 15^3, 21^3 and 27^3
    // (27 nodes); at eight nodes, 20^3, they leave the longest range 5 % above
    // the mean, as at 21^3
    const MmaShape S = f32 ? MmaShape{FC_TILE, FC_MT, 125, 235, 3000, 1500} : MmaShape{8, MM_MT, 66, 80, 3000, 600};
    MmaList &M = f32 ? L.groups : L.mma;
    MmaPlan *pl = nullptr;
    if ((rc = mma_boxes(c, M, !f32))) return rc;
    if ((rc = mma_plan(c, M, S, cell0, cell1, &pl))) return rc;
    MmaArgs a;
    std::memset(&a, 0, sizeof(a));
    a.rowb = f32 ? L.RW32 * 4 : L.RD64 * 8;
    const int warps = f32 ? FC_WARPS : MM_WARPS;
    const int stage = warps * MM_SP * a.rowb;  // one ring stage of every warp
    const int nf = bil ? 2 : 1, fb = (int)std::min<long long>((g.N * (f32 ? 4 : 8) + 15) / 16 * 16, 1 << 28);
    // a tile's sums of every warp at a unit's end
    const int red = warps * 8 * (f32 ? (g.P + 3) / 4 * 4 : (g.P + 7) / 8 * 8) * 8;
    const int tail = red + warps * MM_MAXST * 12 + 16 + 8 * MM_MT * 4;
    // at least two stages beside the shared copies, else f from global memory;
    // what room is left goes to the partial Q, then (FP64) to up to four tiles
    // at a time at a unit's end, then to more stages
    const bool gf = c->f_global == 1 || (long long)nf * fb + tail + 2 * stage > maxsm;
    int room = maxsm - tail - (gf ? 0 : nf * fb) - 2 * stage;
    if (room < 0) return set_err(c, DGV_EUNSUP, "collide: the row ring does not fit in shared memory");
    const size_t len = (size_t)(cell1 - cell0) * g.P;
    const int pb = len * 8 < (size_t)room ? (int)((len * 8 + 15) / 16 * 16) : 0;
    a.part_smem = pb > 0 && pb <= room;
    if (a.part_smem) room -= pb;
    a.red_tiles = 1;
    while (!f32 && a.part_smem && a.red_tiles < 4 && room >= a.red_tiles * red) {
        room -= a.red_tiles * red;
        a.red_tiles *= 2;
    }
    a.nst = std::min(MM_MAXST, 2 + room / stage);
    a.off_f = a.nst * stage;
    a.off_g = a.off_f + (gf ? 0 : fb);
    a.off_part = a.off_f + (gf ? 0 : nf * fb);
    a.off_red = a.off_part + (a.part_smem ? pb : 0);
    a.off_bar = a.off_red + a.red_tiles * red;
    const size_t smem = (size_t)a.off_bar + warps * MM_MAXST * 12;
    const int nchunks = c->nchunks_opt > 0 ? (int)std::min<long long>(c->nchunks_opt, std::max<long long>(1, L.nblocks))
                                           : mma_chunks(nsm, nvdf, warps, pl->cost.back() / (S.c_tile * S.tiles + S.c_stage));
    const int2 *bounds = nullptr;
    if ((rc = mma_bounds(c, pl, nchunks, &bounds))) return rc;
    if ((rc = ensure_buffer(c, &c->d_partial, &c->partial_bytes, (size_t)nvdf * nchunks * len * sizeof(double)))) return rc;
    if ((rc = ensure_errflag(c))) return rc;
    if (gf) {
        const void *p = nullptr;
        if ((rc = f_local_major(c, d_f, d_g, nvdf, f32, &p))) return rc;
        a.fg = static_cast<const double *>(p);
        a.gg = bil ? a.fg + (size_t)nvdf * g.N : nullptr;
    }
    a.f = d_f; a.g = d_g; a.partial = c->d_partial; a.rows = (const char *)(f32 ? L.rows32 : L.rows64);
    a.segs = (const unsigned long long *)M.segs; a.sfirst = (const int *)M.sfirst;
    a.units = (const MmaUnit *)pl->units; a.bounds = bounds;
    a.err = c->d_err; a.N = g.N; a.Nc = g.Nc; a.Mv = g.d.Mv; a.Mw = g.d.Mw; a.nchunks = nchunks;
    a.cell0 = cell0; a.ncell = cell1 - cell0; a.wait_ns = wait_limit_ns(c);
    MmaWithhold wh;
    if (c->test_withhold && (rc = wh.take(c, M))) return rc;
    MmaFn fn = g.P == 27 ? mma_pick<27>(f32, bil, gf) : mma_pick<8>(f32, bil, gf);
    DGV_CUDA(c, cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KTimer kt(c);
    if (pl->nunits > 0) {
        // VDF fastest: the CTAs resident at one time read the same rows
        fn<<<dim3(nvdf, nchunks), 32 * warps, smem, c->stream>>>(a);
        DGV_CUDA(c, cudaGetLastError());
    } else {
        DGV_CUDA(c, cudaMemsetAsync(c->d_partial, 0, (size_t)nvdf * nchunks * len * sizeof(double), c->stream));
    }
    kt.stop(1);
    if (wh.at && (rc = wh.give_back(c))) return rc;
    const long long nred = (long long)nvdf * ((long long)(len + 31) / 32);
    k_reduce_partials<<<(unsigned)nred, 256, 0, c->stream>>>(c->d_partial, c->d_nwt + (size_t)cell0 * g.P, d_q, nchunks,
                                                             (long long)len, nvdf, scale);
    DGV_CUDA(c, cudaGetLastError());
    count_launches(c, 2);
    return DGV_OK;
}

}  // namespace dgv
