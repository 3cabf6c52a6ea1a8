// Row gathers: SpMV (y = A x over the out-edge CSR) and PageRank pull sweeps (over the in-edge CSR).
//
// Reference: csr_spmv_kernel (apps/SpMV/src/SpMV_kernel.cu:81-96) and pagerank_thread_pull_kernel
// (apps/pagerank/src/pagerank_kernel.cu:95-120) map one thread to one row, so a power-law hub row
// serialises a thread; the consolidation variants hand rows of degree >= 64 to CDP children that
// block-reduce them (SpMV_kernel.cu:196-216, pagerank_kernel.cu:357-382).
//
// Here the rows are cut (on the device, once per graph) into warp tiles of at most 256 merge items
// (rows + nonzeros):
//   - a normal tile holds whole rows of degree <= 255; each lane walks 8 consecutive merge items
//     (merge-path over row ends and nonzeros), and a warp segmented scan joins rows that cross lanes.
//     SpMV stages the gathered products in shared memory and walks them with a start row and a row-end
//     mask that the plan keeps per lane; the sweeps of PageRank read a stream of the merge items
//     themselves (renamed column or row-end mark), laid out so that a lane's 8 come with two 16-byte
//     loads, and walk in registers;
//   - a row of degree > 255 (a hub) is split into 256-nonzero segments whose partial sums are
//     combined afterwards, in segment order, by the hub fix-up kernel.
// Every sum has a fixed order, so results are bit-reproducible run to run; no float atomics.
// With renamed columns (dpg_layout.cu) `col` holds the new ids, `x` is indexed by them, and the
// PageRank epilogue writes row v's contribution at perm[v].
// PageRank folds rank/outdeg into the sweep's epilogue (contrib[v] = rank[v]/outdeg[v]), so the
// gather reads one 4-byte value per in-edge instead of the reference's rank and outdegree pair and
// divide per edge (pagerank_kernel.cu:114), and sums the dangling mass on the device (the reference
// copies every dangling rank to the host each sweep, pagerank_wrapper.cu:212-218).

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "dpg_kernels.h"

namespace dpg {
namespace {

// One CTA per SM: its dynamic shared memory holds the hot-value cache (the first `hot` renamed
// entries of x, i.e. the most gathered columns) and its warps' tile staging. DPG_GATHER_BLOCK is a
// build-time tuning knob (DPG_NVCC_EXTRA); the default is measured.
#ifndef DPG_GATHER_BLOCK
#define DPG_GATHER_BLOCK 1024
#endif
constexpr int kBlock = DPG_GATHER_BLOCK;
constexpr int kWarps = kBlock / 32;
constexpr int kInitBlock = 256;
constexpr int kIpl = kRowTileItems / 32;  // merge items per lane
constexpr int kFixBlock = 256;
constexpr int kFixBatch = 8;  // loads the fix-up issues before it adds them
// What limits the gathers is the L1 left beside the shared memory, where their sectors in flight need
// lines: the shared-memory budget is set with the hot-cache size (see hot_entries). Fewer warps lose at
// any setting (an earlier PageRank sweep of R-MAT 22: 0.20 ms with 1,024 threads, 0.245 with 768, 0.35 with
// 512).
// Shared-memory index with one pad word per 32: lane l walking items 8l.. then hits 32 distinct banks
// instead of 4 (an 8-way conflict without the pad).
constexpr int kPadded = kRowTileItems + kRowTileItems / 32;
__device__ __forceinline__ int pad(int i) { return i + (i >> 5); }

enum { kModeSpmv = 0, kModePagerank = 1, kModeWeighted = 2 };

// Loads of the streams every tile reads once (columns, values, items, out-degrees and the like):
// written before the first kernel of the call's chain starts, so read-only for the launch (nc), and kept
// out of L1 (L1::no_allocate), so the L1 lines are left to the scattered gathers of x, which are what a
// sweep waits on. SpMV also marks them first for
// eviction from L2, which keeps more of x there. Measured per launch (R-MAT 22; R-MAT 24 for
// PageRank): PageRank 0.1623 -> 0.1603 ms and 0.749 -> 0.720 ms with L1::no_allocate, 0.171 and
// 0.764 ms with the L2 hint too; SpMV 0.2146 -> 0.2137 ms, and 0.2063 ms with the L2 hint.
template <int MODE>
__device__ __forceinline__ int ld_stream(const int* p) {
    int v;
    if constexpr (MODE == kModeSpmv) {
        asm("{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
            "ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], pol;\n\t}"
            : "=r"(v) : "l"(p));
    } else {
        asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    }
    return v;
}
template <int MODE>
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    if constexpr (MODE == kModeSpmv) {
        asm("{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
            "ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], pol;\n\t}"
            : "=f"(v) : "l"(p));
    } else {
        asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    }
    return v;
}

// What the kernels before this one in a chain write (the gathered vector, the previous ranks, a batch's
// uniform terms) may still change after this kernel has started, ahead of chain_wait: it is read by
// ordinary loads, which the wait orders, never by the read-only path. ld_live_once stays out of L1. No slower
// than the read-only path was; __ldca (ld.global.ca) was: PageRank R-MAT 22 3.07 against 3.06 ms, gradient
// R-MAT 20 7.68 against 7.60 ms.
__device__ __forceinline__ float ld_live(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_live_once(const float* p) {
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// 16 bytes of a stream; every word -1 unless `in` (kItemNone; a NaN as an arc value, which no tile past
// the last is walked for). Never kept in L1.
__device__ __forceinline__ int4 ld_stream4(const int4* p, bool in) {
    int4 v = make_int4(kItemNone, kItemNone, kItemNone, kItemNone);
    if (in) asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// PageRank epilogue of one row: new rank, next contribution, dangling mass, convergence flag.
// od / pos are the row's out-degree and contribution slot (perm[v] with renamed columns).
// BATCH: packed graphs, `base` being the uniform term of the row's graph.
template <bool BATCH>
__device__ __forceinline__ void pr_epilogue(const RowGatherLaunch& L, int v, float sum, float base, int od, int pos,
                                            double& dang, bool& moved) {
    const float nv = fmaf(L.damping, sum, base);
    if (L.rank_out) L.rank_out[v] = nv;
    if (L.rank_prev && fabsf(nv - ld_live(L.rank_prev + v)) > L.epsilon) moved = true;
    // Only vertices with out-arcs are ever gathered (they are the columns), so the contribution
    // slot of a dangling vertex is free: a batch parks its rank there for the per-graph reduction.
    // The division runs for every row (by 1 for a dangling one) so a warp's rows do not diverge
    // around it; only the stores and the dangling sum depend on the out-degree.
    const float q = nv / static_cast<float>(od > 0 ? od : 1);
    if (BATCH) {
        L.y[pos] = od > 0 ? q : nv;
    } else {
        if (od > 0) L.y[pos] = q;
        if (od <= 0) dang += static_cast<double>(nv);
    }
}

__device__ __forceinline__ float batch_base(const RowGatherLaunch& L, int v) {
    return ld_live(L.gbase + __ldg(L.vgraph + v));
}

// Epilogue of one row of a weighted PageRank sweep (dpg_prgrad.cu): forward (no seed) the new rank and
// its contribution rank / W; adjoint the new lambda, which is also the next gathered vector. x goes to
// rank_out[v], the gathered vector's entry to y[pos]; `dang` collects the dangling ranks, or all lambdas.
__device__ __forceinline__ void weighted_epilogue(const RowGatherLaunch& L, int v, float sum, float base, float W,
                                                  int pos, float seed, float prev, double& dang, bool& moved) {
    float x;
    if (!L.seed) {
        x = fmaf(L.damping, sum, base);
        if (W > 0.0f) L.y[pos] = x / W;
        else dang += static_cast<double>(x);
    } else {
        x = W > 0.0f ? seed + L.damping * (sum / W) : seed + base;
        L.y[pos] = x;
        dang += static_cast<double>(x);
    }
    if (L.rank_prev && fabsf(x - prev) > L.epsilon * fabsf(x)) moved = true;
    L.rank_out[v] = x;
}

__device__ __forceinline__ void weighted_epilogue(const RowGatherLaunch& L, int v, float sum, float base,
                                                  double& dang, bool& moved) {
    weighted_epilogue(L, v, sum, base, __ldg(L.W + v), L.perm ? __ldg(L.perm + v) : v,
                      L.seed ? __ldg(L.seed + v) : 0.0f, L.rank_prev ? ld_live(L.rank_prev + v) : 0.0f, dang, moved);
}

__device__ __forceinline__ float pr_base(const RowGatherLaunch& L) {
    return static_cast<float>(L.base_const + L.dangling_scale * __ldcg(L.dsum_in));
}

// Hub rows: the segment partials summed in segment order, then the row epilogue. Small hubs go one
// per thread, big hubs one per warp. The loads are issued in batches before they are added in the
// same order as a plain loop would, so the sums are unchanged and each batch costs one round trip.
template <int MODE>
__device__ __forceinline__ void fixup_hubs(const RowGatherLaunch& L, int tid, int nthreads, int gwarp, int nwarps,
                                           int lane, float base, double& dang, bool& moved) {
    // The epilogue inputs (out-degree, contribution slot) are loaded with the partials.
    for (int h = tid; h < L.plan.nhub_small; h += nthreads) {
        const int4 H = __ldg(L.plan.hubs_small + h);
        int od = 0, pos = 0;
        if (MODE == kModePagerank) {
            od = __ldg(L.outdeg + H.x);
            pos = L.perm ? __ldg(L.perm + H.x) : H.x;
        }
        float p[kSmallHubSegs];
#pragma unroll
        for (int s = 0; s < kSmallHubSegs; ++s) p[s] = s < H.z ? L.partial[H.y + s] : 0.0f;
        float acc = 0.0f;
#pragma unroll
        for (int s = 0; s < kSmallHubSegs; ++s) acc += p[s];
        if (MODE == kModeSpmv) L.y[H.x] = acc;
        else if (MODE == kModeWeighted) weighted_epilogue(L, H.x, acc, base, dang, moved);
        else if (L.vgraph) pr_epilogue<true>(L, H.x, acc, batch_base(L, H.x), od, pos, dang, moved);
        else pr_epilogue<false>(L, H.x, acc, base, od, pos, dang, moved);
    }
    for (int h = gwarp; h < L.plan.nhub_big; h += nwarps) {
        const int4 H = __ldg(L.plan.hubs_big + h);
        int od = 0, pos = 0;
        if (MODE == kModePagerank && lane == 0) {
            od = __ldg(L.outdeg + H.x);
            pos = L.perm ? __ldg(L.perm + H.x) : H.x;
        }
        float acc = 0.0f;
        for (int s0 = lane; s0 < H.z; s0 += 32 * kFixBatch) {
            float p[kFixBatch];
#pragma unroll
            for (int q = 0; q < kFixBatch; ++q) p[q] = s0 + 32 * q < H.z ? L.partial[H.y + s0 + 32 * q] : 0.0f;
#pragma unroll
            for (int q = 0; q < kFixBatch; ++q) acc += p[q];
        }
        acc = warp_sum_f32(acc);
        if (lane == 0) {
            if (MODE == kModeSpmv) L.y[H.x] = acc;
            else if (MODE == kModeWeighted) weighted_epilogue(L, H.x, acc, base, dang, moved);
            else if (L.vgraph) pr_epilogue<true>(L, H.x, acc, batch_base(L, H.x), od, pos, dang, moved);
            else pr_epilogue<false>(L, H.x, acc, base, od, pos, dang, moved);
        }
    }
}

// Thread t's share of a[0, n) (entries t, t + NT, ...) in index order, loads in batches.
template <int NT>
__device__ __forceinline__ double strided_sum_f64(const double* a, int n, double acc) {
    for (int i0 = threadIdx.x; i0 < n; i0 += NT * kFixBatch) {
        double p[kFixBatch];
#pragma unroll
        for (int q = 0; q < kFixBatch; ++q) p[q] = i0 + NT * q < n ? __ldcg(a + i0 + NT * q) : 0.0;
#pragma unroll
        for (int q = 0; q < kFixBatch; ++q) acc += p[q];
    }
    return acc;
}

// Sum over the block of each thread's v, warps in order; valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum_f64(double v) {
    __shared__ double s_red[NT / 32];
    v = warp_sum_f64(v);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    double total = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < NT / 32; ++w) total += s_red[w];
    return total;
}

// The hot cache: the first `hot` (most gathered) entries of x, loads issued in batches of 8 (one round
// trip each instead of one per entry).
__device__ __forceinline__ void fill_hot(const float* x, int hot, float* s_hot) {
    for (int i0 = threadIdx.x; i0 < hot; i0 += kBlock * 8) {
        float h[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) h[q] = i0 + kBlock * q < hot ? ld_live(x + i0 + kBlock * q) : 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (i0 + kBlock * q < hot) s_hot[i0 + kBlock * q] = h[q];
    }
    __syncthreads();
}

// SpMV. A warp takes one tile at a time through its staging area; the next tile's columns and values are
// loaded while this one's gathers are in flight, and the descriptor of the one after that, so a tile costs
// one round trip. Same box, R-MAT 22: 224 us with two tiles per step and nothing loaded ahead, 206 this way
// (290 with the values not loaded ahead).
__global__ void __launch_bounds__(kBlock) spmv_gather_kernel(RowGatherLaunch L) {
    extern __shared__ __align__(16) unsigned char rg_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * kWarps + warp;
    const int nwarps = gridDim.x * kWarps;
    float* val = reinterpret_cast<float*>(rg_smem) + warp * (2 * kPadded);
    float* out = val + kPadded;
    float* s_hot = reinterpret_cast<float*>(rg_smem) + kWarps * 2 * kPadded;

    const int ntiles = L.plan.ntiles;
    int4 Tn;  // descriptor and lane walk two tiles ahead, columns and values one tile ahead
    int infon, cn[kIpl];
    float an[kIpl];
    auto fetch_tile = [&](int t) {
        Tn = t < ntiles ? __ldg(L.plan.tiles + t) : make_int4(0, 0, 0, 0);
        infon = t < ntiles ? __ldg(L.plan.lane_info + t * 32 + lane) : 0;
    };
    auto fetch_values = [&] {
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            const int j = i * 32 + lane;
            cn[i] = j < Tn.w ? ld_stream<kModeSpmv>(L.col + Tn.z + j) : 0;
            an[i] = j < Tn.w ? ld_stream<kModeSpmv>(L.vals + Tn.z + j) : 0.0f;
        }
    };
    fetch_tile(gwarp);
    fetch_values();
    int4 Tc = Tn;
    int infoc = infon;
    fetch_tile(gwarp + nwarps);
    chain_wait();  // only x may still be on its way (the renaming of x, in the same call)
    fill_hot(L.x, L.hot, s_hot);
    for (int t0 = gwarp; t0 < ntiles; t0 += nwarps) {
        const int4 T = Tc;
        const int info = infoc;
        int cols[kIpl];
        float av[kIpl], pv[kIpl];
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            cols[i] = cn[i];
            av[i] = an[i];
        }
        fetch_values();
        Tc = Tn;
        infoc = infon;
        fetch_tile(t0 + 2 * nwarps);
        // The gathers, with no branch at all: the hot test is a select and the shared-memory read
        // unconditional (entry 0 for cold columns; the launch allocates at least one).
        const int row = T.x, nrows = T.y, nnz = T.w;
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            const int c = cols[i];
            const bool hot = c < L.hot;
            const float hv = s_hot[hot ? c : 0];
            float gv = 0.0f;
            if (!hot) gv = ld_live(L.x + c);
            pv[i] = i * 32 + lane < nnz ? (hot ? hv : gv) * av[i] : 0.0f;
        }
        if (nrows < 0) {
            // Hub segment: fixed-order lane sums, then a butterfly; partial goes to the fix-up.
            // Values past the segment's end are 0, so every lane adds all of its own.
            float acc = 0.0f;
#pragma unroll
            for (int i = 0; i < kIpl; ++i) acc += pv[i];
            acc = warp_sum_f32(acc);
            if (lane == 0) L.partial[-(nrows + 1)] = acc;
            continue;
        }
        // All 8 values are staged (0 past nnz; pad(255) = 262 is inside the 264-entry row), so the
        // stores need no predicate; the walk reads only the first nnz of them as nonzeros.
#pragma unroll
        for (int i = 0; i < kIpl; ++i) val[pad(i * 32 + lane)] = pv[i];
        __syncwarp();
        // Merge-path: lane owns merge items [d0, d1) starting at row r0; the plan's mask says
        // which of them are row ends (emit the open row) and which are nonzeros (take one).
        // r = row ends consumed, kk = nonzeros consumed. The walk is branch-free.
        const int total = nrows + nnz;
        const int d0 = min(lane * kIpl, total);
        const int nlive = min(d0 + kIpl, total) - d0;
        const unsigned ends = static_cast<unsigned>(info) >> 8;
        int r = d0 < total ? (info & 0xFF) : nrows;
        int kk = d0 - r;
        float acc = 0.0f;
        // Rows advance only at row ends, so the first row the lane closes is its start row.
        const int first_emit = ends != 0u ? r : -1;
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            const bool emit = (ends >> i) & 1u;
            const bool take = i < nlive && !emit;
            const float v = val[pad(kk)];  // kk <= nnz <= 255 stays inside the padded row
            if (emit) out[pad(r)] = acc;
            acc = take ? acc + v : (emit ? 0.0f : acc);
            kk += take ? 1 : 0;
            r += emit ? 1 : 0;
        }
        // Segmented inclusive scan of the lanes' open partials (key = row still open at lane end).
        float cv = acc;
        const int key = r;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float tv = __shfl_up_sync(kFullMask, cv, o);
            const int tk = __shfl_up_sync(kFullMask, key, o);
            if (lane >= o && tk == key) cv += tv;
        }
        const float cin = __shfl_up_sync(kFullMask, cv, 1);
        const int kin = __shfl_up_sync(kFullMask, key, 1);
        if (lane > 0 && first_emit >= 0 && kin == first_emit) out[pad(first_emit)] += cin;
        __syncwarp();
        for (int rr = lane; rr < nrows; rr += 32) L.y[row + rr] = out[pad(rr)];
        __syncwarp();
    }
}

// Sweeps of PageRank and of the weighted PageRank. A lane's 8 merge items of a tile arrive as two
// 16-byte loads and stay in registers with their gathered values, so only the row sums pass through
// shared memory; the next tile's items, descriptor and start rows are loaded while this one's gathers
// are in flight, so a tile costs one round trip.
// What bounds it: the load-store pipe (a gathered line, or a shared-memory wavefront, per cycle and SM)
// and the instruction issue. Walking values staged in shared memory took 490 warp instructions per
// tile, both pipes at 65-69 % (R-MAT 20). Same box, 20 sweeps with the staged walk, two tiles per step /
// this one with two tiles per step / one / one with its items a step ahead: R-MAT 22 3.54 / 3.29 /
// 3.19 / 3.15 ms, 608,712 vertices x 16 810 / 723 / 705 / 682 us; gradient of R-MAT 20 10.8 / 9.6 / 9.0 /
// 8.55 ms. Three tiles per step spill (4.6 ms). Shared-memory budgets (hot cache) of 132 / 164 / 196
// KB: R-MAT 22 3.23 / 3.16 / 3.31 ms.
// CONV: sweeps with a convergence test (rank_prev given).
// BATCH: packed graphs. Each graph's most gathered columns open its own range of columns, so a hot cache
// of the first ones would serve the first graph alone. Each CTA takes a consecutive run of tiles, and
// with them the windows of L.win in turn: a window's tiles are those of one graph, or of several small
// ones that fit in the cache together, and the cache is filled from the window's first column on. A tile
// that reaches into the next window only misses it. 48 graphs (107 M arcs), same box, per sweep: 0.35 ms
// with one cache at 0 for all, 0.26 with windows, 0.22 with the epilogue inputs of 64 rows ahead as well.
template <int MODE, bool CONV, bool BATCH>
__global__ void __launch_bounds__(kBlock) rowgather_kernel(RowGatherLaunch L) {
    if (!CONV) L.rank_prev = nullptr;
    extern __shared__ __align__(16) unsigned char rg_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * kWarps + warp;
    const int nwarps = gridDim.x * kWarps;
    float* out = reinterpret_cast<float*>(rg_smem) + warp * kPadded;
    float* s_hot = reinterpret_cast<float*>(rg_smem) + kWarps * kPadded + 1;
    if (threadIdx.x == 0) s_hot[-1] = 0.0f;  // what the marks gather
    float base = 0.0f;
    double dang = 0.0;
    bool moved = false;

    // Tiles [first, ntiles) by `step`; BATCH: of the CTA's window, one after the other.
    int ntiles = L.plan.ntiles, first = gwarp, step = nwarps;
    int hot = L.hot, hot0 = 0;  // the cache holds columns [hot0, hot0 + hot)
    int cta_end = 0, w = 0;
    const bool windows = BATCH && L.nwin > 0;
    if (windows) {
        const int2 c0 = __ldg(L.cta_first + blockIdx.x);  // {first tile, its window}
        first = c0.x;
        w = c0.y;
        cta_end = __ldg(L.cta_first + blockIdx.x + 1).x;
        step = kWarps;
    }
    do {
    if (windows) {
        if (first >= cta_end) break;
        const int2 W = __ldg(L.win + w);  // {first tile, first column}
        ntiles = w + 1 < L.nwin ? min(cta_end, __ldg(L.win + w + 1).x) : cta_end;
        hot0 = W.y;
        hot = min(L.hot, L.V - hot0);
        first += warp;
    }
    int2 Tn;          // the next tile: {row, nrows}, start row of the lane, items
    int infon;
    int4 qn[kIpl / 4];
    int4 wn[kIpl / 4];  // weighted: arc values
    auto fetch = [&](int t) {
        const bool in = t < ntiles;
        Tn = in ? __ldg(reinterpret_cast<const int2*>(L.plan.tiles + t)) : make_int2(0, 0);
        infon = in ? __ldg(L.plan.lane_info + t * 32 + lane) : 0;
        const int4* src = reinterpret_cast<const int4*>(L.items) + static_cast<int64_t>(t) * (kRowTileItems / 4) + lane;
#pragma unroll
        for (int h = 0; h < kIpl / 4; ++h) qn[h] = ld_stream4(src + 32 * h, in);
        if (MODE == kModeWeighted) {
            const int4* sw = reinterpret_cast<const int4*>(L.witems) + static_cast<int64_t>(t) * (kRowTileItems / 4) + lane;
#pragma unroll
            for (int h = 0; h < kIpl / 4; ++h) wn[h] = ld_stream4(sw + 32 * h, in);
        }
    };
    fetch(first);  // the plan's arrays: fixed, so they may be read ahead of the wait
    chain_wait();
    if (!BATCH) base = pr_base(L);
    fill_hot(L.x + hot0, hot, s_hot);
    for (int t = first; t < ntiles; t += step) {
        const int row = Tn.x, nrows = Tn.y, r0 = infon & 0xFF;
        int item[kIpl];
#pragma unroll
        for (int h = 0; h < kIpl / 4; ++h) {
            item[4 * h + 0] = qn[h].x;
            item[4 * h + 1] = qn[h].y;
            item[4 * h + 2] = qn[h].z;
            item[4 * h + 3] = qn[h].w;
        }
        // Epilogue inputs of the first 32 rows (64 in a batch, whose graphs of 8 arcs per vertex have
        // about 28 rows per tile): predicated loads rather than branches.
        constexpr int NE = BATCH ? 2 : 1;
        int eod[NE], epos[NE], egraph[NE];
#pragma unroll
        for (int q = 0; q < NE; ++q) {
            const int v = row + lane + 32 * q;
            const bool in = lane + 32 * q < nrows;
            eod[q] = 0;
            epos[q] = v;
            egraph[q] = 0;
            if (MODE == kModePagerank) {
                eod[q] = in ? ld_stream<MODE>(L.outdeg + v) : 0;
                if (L.perm) epos[q] = in ? ld_stream<MODE>(L.perm + v) : 0;
            }
            if (BATCH) egraph[q] = in ? ld_stream<MODE>(L.vgraph + v) : 0;
        }
        int4 w[kIpl / 4];
        if (MODE == kModeWeighted) {
#pragma unroll
            for (int h = 0; h < kIpl / 4; ++h) w[h] = wn[h];
        }
        fetch(t + step);
        // The gathers. The hot test stays a select between a shared and a global load (written as an
        // if/else it became a divergent branch: 0.192 ms per sweep against 0.176 on R-MAT 22). Marks are
        // negative and read the zero in front of the hot cache.
        float pv[kIpl];
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            const int c = item[i];
            if (BATCH) {
                const int d = c < 0 ? -1 : c - hot0;
                pv[i] = c < 0 || static_cast<unsigned>(d) < static_cast<unsigned>(hot) ? s_hot[d] : ld_live(L.x + c);
            } else {
                pv[i] = c < hot ? s_hot[max(c, -1)] : ld_live(L.x + c);
            }
        }
        if (MODE == kModeWeighted) {
#pragma unroll
            for (int h = 0; h < kIpl / 4; ++h) {
                const int4 q = w[h];
                pv[4 * h + 0] *= __int_as_float(q.x);
                pv[4 * h + 1] *= __int_as_float(q.y);
                pv[4 * h + 2] *= __int_as_float(q.z);
                pv[4 * h + 3] *= __int_as_float(q.w);
            }
        }
        if (nrows < 0) {
            // Hub segment: lane sums in item order, then a butterfly; the partial goes to the fix-up.
            float acc = 0.0f;
#pragma unroll
            for (int i = 0; i < kIpl; ++i) acc += pv[i];
            acc = warp_sum_f32(acc);
            if (lane == 0) L.partial[-(nrows + 1)] = acc;
            continue;
        }
        float ebase[NE];
#pragma unroll
        for (int q = 0; q < NE; ++q) ebase[q] = BATCH ? ld_live(L.gbase + egraph[q]) : base;
        float eW = 0.0f, eseed = 0.0f, eprev = 0.0f;
        if (MODE == kModeWeighted && lane < nrows) {
            eW = ld_stream<MODE>(L.W + row + lane);
            if (L.perm) epos[0] = ld_stream<MODE>(L.perm + row + lane);
            if (L.seed) eseed = ld_stream<MODE>(L.seed + row + lane);
            if (CONV) eprev = ld_live_once(L.rank_prev + row + lane);
        }
        // The lane's items in order: a nonzero is added to the open row, a row end closes it.
        int r = r0;
        float acc = 0.0f;
        bool any_end = false;
#pragma unroll
        for (int i = 0; i < kIpl; ++i) {
            const bool end = item[i] == kItemRowEnd;
            acc += pv[i];  // marks hold 0
            if (end) out[pad(r)] = acc;
            acc = end ? 0.0f : acc;
            r += end ? 1 : 0;
            any_end |= end;
        }
        // Segmented inclusive scan of the lanes' open partials (key = row still open at lane end).
        float cv = acc;
        const int key = r;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float tv = __shfl_up_sync(kFullMask, cv, o);
            const int tk = __shfl_up_sync(kFullMask, key, o);
            if (lane >= o && tk == key) cv += tv;
        }
        const float cin = __shfl_up_sync(kFullMask, cv, 1);
        const int kin = __shfl_up_sync(kFullMask, key, 1);
        // The first row the lane closes is its start row, open in the lanes before it.
        if (lane > 0 && any_end && kin == r0) out[pad(r0)] += cin;
        __syncwarp();
        for (int rr = lane; rr < nrows; rr += 32) {
            const float sum = out[pad(rr)];
            const int v = row + rr;
            if (MODE == kModeWeighted) {
                if (rr < 32) weighted_epilogue(L, v, sum, base, eW, epos[0], eseed, eprev, dang, moved);
                else weighted_epilogue(L, v, sum, base, dang, moved);
            } else if (rr < 32) {
                pr_epilogue<BATCH>(L, v, sum, ebase[0], eod[0], epos[0], dang, moved);
            } else if (NE > 1 && rr < 64) {
                pr_epilogue<BATCH>(L, v, sum, ebase[NE - 1], eod[NE - 1], epos[NE - 1], dang, moved);
            } else {
                pr_epilogue<BATCH>(L, v, sum, BATCH ? batch_base(L, v) : base, __ldg(L.outdeg + v),
                                   L.perm ? __ldg(L.perm + v) : v, dang, moved);
            }
        }
        __syncwarp();
    }
    if (windows) {
        __syncthreads();  // the cache is free again
        first = ntiles;
        ++w;
    }
    } while (windows);
    dang = warp_sum_f64(dang);
    if (lane == 0) L.dpart[gwarp] = dang;
    // One store per CTA at most: a store per moved row queued up on that one word (700,001 vertices, 11 M
    // arcs: 50 us per sweep with it, 37 without; weighted sweep of R-MAT 20: 94 and 64 us).
    if (CONV && __syncthreads_or(moved) && threadIdx.x == 0) *L.nonstop = 1u;
}

// The hub fix-up after each gather launch (and, with no hubs, after the initial vector). For
// PageRank it also reduces the sweep's dangling mass into dsum_out.
template <int MODE>
__global__ void __launch_bounds__(kFixBlock) hub_fixup_kernel(RowGatherLaunch L, int gather_warps, DevStatus* st) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthreads = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const int gwarp = tid >> 5;
    const int nwarps = nthreads >> 5;
    chain_wait();
    chain_next();
    float base = 0.0f;
    if (MODE != kModeSpmv) base = pr_base(L);
    double dang = 0.0;
    bool moved = false;
    fixup_hubs<MODE>(L, tid, nthreads, gwarp, nwarps, lane, base, dang, moved);
    if (MODE == kModeSpmv) return;
    if (L.nonstop && __syncthreads_or(moved) && threadIdx.x == 0) *L.nonstop = 1u;
    // Block b adds its slice of the gather warps' dangling partials to its own rows' (slices in
    // index order), leaves one partial, and the last block to finish adds those in block order.
    const int per = (gather_warps + gridDim.x - 1) / gridDim.x;
    const int lo = min(gather_warps, static_cast<int>(blockIdx.x) * per);
    const int hi = min(gather_warps, lo + per);
    double slice = 0.0;
    for (int i = lo + static_cast<int>(threadIdx.x); i < hi; i += kFixBlock) slice += __ldcg(L.dpart + i);
    const double bsum = block_sum_f64<kFixBlock>(slice + dang);
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        L.dfix[blockIdx.x] = bsum;
        __threadfence();
        s_last = atomicAdd(&st->fix_count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const double total = block_sum_f64<kFixBlock>(strided_sum_f64<kFixBlock>(L.dfix, gridDim.x, 0.0));
    if (threadIdx.x == 0) {
        *L.dsum_out = total;
        st->fix_count = 0u;
        if (L.nonstop) {  // the sweep's verdict, straight to the host; the flag is clear for the next sweep
            *reinterpret_cast<volatile unsigned*>(L.host_flag) = *reinterpret_cast<volatile unsigned*>(L.nonstop);
            *L.nonstop = 0u;
            __threadfence_system();
        }
    }
}

// Initial contribution vector and its dangling mass. Uses the gather grid so dpart lines up.
__global__ void __launch_bounds__(kInitBlock) pr_init_kernel(RowGatherLaunch L, float init_rank, float* rank_prev) {
    const int lane = threadIdx.x & 31;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nthreads = gridDim.x * blockDim.x;
    double dang = 0.0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < L.V; v += nthreads) {
        const int od = __ldg(L.outdeg + v);
        const float r0 = L.vgraph ? __ldg(L.ginit + __ldg(L.vgraph + v)) : init_rank;
        const int pos = L.perm ? __ldg(L.perm + v) : v;
        if (od > 0) L.y[pos] = r0 / static_cast<float>(od);
        else if (L.vgraph) L.y[pos] = r0;
        else dang += static_cast<double>(r0);
        if (rank_prev) rank_prev[v] = r0;
    }
    dang = warp_sum_f64(dang);
    if (lane == 0) L.dpart[gwarp] = dang;
}

// Per lane of each normal tile, once per graph: the merge-path start row, i.e. the largest r with
// (row end r-1) + r <= 8 * lane (the row ends the lane's first merge item comes after), and which
// of the lane's 8 merge items are row ends rather than nonzeros. With both, the gather kernel walks
// its items without reading any row end.
// With d_ntiles the tile count is read on the device (clamped to cap), and a set bad-offsets flag
// makes the kernel do nothing: the plan it would read was built from offsets that failed the check.
__global__ void tile_lane_starts_kernel(const int4* __restrict__ tiles, int ntiles, const int64_t* d_ntiles,
                                        int64_t cap, const int* bad, const int32_t* __restrict__ off,
                                        uint16_t* __restrict__ lane_info) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    if (d_ntiles) {
        if (bad && (*reinterpret_cast<const volatile int*>(bad) & 4)) return;
        const int64_t n = *d_ntiles;
        ntiles = static_cast<int>(n < cap ? n : cap);
    }
    for (int t = w; t < ntiles; t += nw) {
        const int4 T = __ldg(tiles + t);
        int lo = 0;
        unsigned ends = 0;
        if (T.y > 0) {
            const int row = T.x, nrows = T.y, nb = T.z, nnz = T.w;
            const int total = nrows + nnz;
            const int d0 = min(lane * kIpl, total);
            lo = max(0, d0 - nnz);
            int hi = min(d0, nrows);
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (__ldg(off + row + mid) - nb + mid <= d0) lo = mid;
                else hi = mid - 1;
            }
            // The lane's items in merge order: nonzero kk while kk < (end of row r), else the end of r.
            int r = lo, kk = d0 - lo;
            const int d1 = min(d0 + kIpl, total);
            int rend = r < nrows ? __ldg(off + row + r + 1) - nb : 0x7FFFFFFF;
            for (int i = 0; d0 + i < d1; ++i) {
                if (kk < rend) {
                    ++kk;
                } else {
                    ends |= 1u << i;
                    ++r;
                    rend = r < nrows ? __ldg(off + row + r + 1) - nb : 0x7FFFFFFF;
                }
            }
        }
        lane_info[static_cast<int64_t>(t) * 32 + lane] = static_cast<uint16_t>(lo | (ends << 8));
    }
}

}  // namespace

cudaError_t launch_tile_lane_starts(const RowPlanDev& plan, const int32_t* off, cudaStream_t s, int sm_count) {
    if (plan.ntiles > 0)
        tile_lane_starts_kernel<<<sm_count * 8, 256, 0, s>>>(plan.tiles, plan.ntiles, nullptr, 0, nullptr, off,
                                                             plan.lane_info);
    return cudaGetLastError();
}

cudaError_t launch_tile_lane_starts_dev(const int4* tiles, const int64_t* d_ntiles, int64_t cap, const int* bad,
                                        const int32_t* off, uint16_t* lane_info, cudaStream_t s, int sm_count) {
    tile_lane_starts_kernel<<<sm_count * 8, 256, 0, s>>>(tiles, 0, d_ntiles, cap, bad, off, lane_info);
    return cudaGetLastError();
}

namespace {
// A tile's 256 merge items (kIpl per lane) in the order of the sweeps' loads: item i of lane l at
// (i / 4) * 128 + 4 * l + i % 4. Lane l of the tile's warp calls fn(position, nonzero or -1 for a row end
// or -2 past the tile) for each of its items; a hub segment is all nonzeros.
template <class F>
__device__ __forceinline__ void for_tile_items(const int4& T, int info, int lane, F fn) {
    const int nrows = T.y, nnz = T.w;
    const int total = nrows < 0 ? nnz : nrows + nnz;
    int kk = lane * kIpl - (nrows < 0 ? 0 : info & 0xFF);
#pragma unroll
    for (int i = 0; i < kIpl; ++i) {
        const int at = (i >> 2) * 128 + 4 * lane + (i & 3);
        const bool end = nrows >= 0 && ((info >> (8 + i)) & 1);
        if (lane * kIpl + i >= total) fn(at, -2);
        else if (end) fn(at, -1);
        else fn(at, kk++);
    }
}

__global__ void tile_items_kernel(RowPlanDev plan, const int32_t* __restrict__ col, const int32_t* __restrict__ perm,
                                  int32_t* __restrict__ items) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = w; t < plan.ntiles; t += nw) {
        const int4 T = __ldg(plan.tiles + t);
        int32_t* dst = items + static_cast<int64_t>(t) * kRowTileItems;
        for_tile_items(T, __ldg(plan.lane_info + t * 32 + lane), lane, [&](int at, int k) {
            int c = k == -1 ? kItemRowEnd : kItemNone;
            if (k >= 0) {
                c = __ldg(col + T.z + k);
                if (perm) c = __ldg(perm + c);
            }
            dst[at] = c;
        });
    }
}

__global__ void tile_values_kernel(RowPlanDev plan, const float* __restrict__ vals, const int32_t* __restrict__ arc,
                                   float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = w; t < plan.ntiles; t += nw) {
        const int4 T = __ldg(plan.tiles + t);
        float* dst = out + static_cast<int64_t>(t) * kRowTileItems;
        for_tile_items(T, __ldg(plan.lane_info + t * 32 + lane), lane, [&](int at, int k) {
            dst[at] = k >= 0 ? __ldg(vals + (arc ? __ldg(arc + T.z + k) : T.z + k)) : 0.0f;
        });
    }
}
}  // namespace

namespace {
// win[k].x: first tile of window k, i.e. the first tile whose row is at or past rows[k] (tiles ascend by row).
__global__ void window_tiles_kernel(RowPlanDev plan, const int32_t* __restrict__ rows, int nwin, int2* win) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nwin; k += gridDim.x * blockDim.x) {
        int lo = 0, hi = plan.ntiles;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(plan.tiles + mid).x < rows[k]) lo = mid + 1;
            else hi = mid;
        }
        win[k] = make_int2(lo, rows[k]);
    }
}
}  // namespace

cudaError_t launch_window_tiles(const RowPlanDev& plan, const int32_t* rows, int nwin, int2* win, cudaStream_t s) {
    if (nwin > 0) window_tiles_kernel<<<(nwin + 255) / 256, 256, 0, s>>>(plan, rows, nwin, win);
    return cudaGetLastError();
}

cudaError_t launch_tile_items(const RowPlanDev& plan, const int32_t* col, const int32_t* perm, int32_t* items,
                              cudaStream_t s, int sm_count) {
    if (plan.ntiles > 0) tile_items_kernel<<<sm_count * 8, 256, 0, s>>>(plan, col, perm, items);
    return cudaGetLastError();
}

cudaError_t launch_tile_values(const RowPlanDev& plan, const float* vals, const int32_t* arc, float* out, cudaStream_t s,
                               int sm_count) {
    if (plan.ntiles > 0) tile_values_kernel<<<sm_count * 8, 256, 0, s>>>(plan, vals, arc, out);
    return cudaGetLastError();
}

void rowgather_grid(int sm_count, int* gather_blocks, int* fix_blocks, int* block_threads) {
    *gather_blocks = sm_count;
    *fix_blocks = sm_count * 2;
    *block_threads = kBlock;
}

size_t rowgather_staging_bytes(bool sweeps) { return sizeof(float) * kWarps * kPadded * (sweeps ? 1 : 2); }

namespace {

// Lifts the kernel's dynamic shared-memory limit, once per device. Every thread sets the same limit, whatever
// its launch takes: a limit set to the launch's own size could be lowered by another thread ahead of the launch.
template <int MODE, bool CONV, bool BATCH>
cudaError_t prepare_rowgather() {
    static std::atomic<uint64_t> ready{0};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    const uint64_t bit = uint64_t{1} << (device & 63);
    if (e != cudaSuccess || (device < 64 && (ready.load() & bit))) return e;
    if constexpr (MODE == kModeSpmv)
        e = cudaFuncSetAttribute(spmv_gather_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatherSmem);
    else
        e = cudaFuncSetAttribute(rowgather_kernel<MODE, CONV, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kGatherSmem);
    if (e == cudaSuccess) ready.fetch_or(bit);
    return e;
}

}  // namespace

namespace {

// ---- the row plan, built on the device ------------------------------------------------------------
// Rows are tiled in fixed ranges of kPlanRange rows, one warp per range, by a greedy walk:
// consecutive rows share a tile while their merge items (rows + nonzeros) fit in kRowTileItems, and
// a row above kHubRowDegree becomes a hub cut into kRowTileItems segments (segments numbered from 0
// within the range, then offset by the earlier ranges' counts). A count pass, an exclusive scan of
// the per-range counts and a write pass produce the tiles in row order, so the plan is the same on
// every run. Offsets that are negative, decrease or pass E stop their range's walk and set bit 4 of
// the status flag; the walk never reads past off[V] and every write is checked against the capacity.
// The warp reads 32 rows at a time and finds the end of the open tile among them with one ballot, so a
// range takes about as many steps as it has tiles and groups of 32 rows. A thread per range walked
// 2,048 rows one after the other: 340 and 604 us for the two passes over 700,001 rows x 16 nonzeros, now 35
// and 45 us (55 and 73 without the next 32 rows loaded ahead).
constexpr int32_t kPlanRange = 2048;
constexpr int kPlanBlock = 128;

struct PlanCount {
    int64_t tiles = 0, small = 0, big = 0, segs = 0;
    __device__ void tile(int32_t, int32_t, int32_t, int32_t) { ++tiles; }
    __device__ void hub(int32_t, int32_t, int32_t, int32_t, int32_t nseg) {
        tiles += nseg;
        (nseg <= kSmallHubSegs ? small : big) += 1;
    }
};

struct PlanWrite {
    int64_t t, hs, hb, seg_base;  // next slots, and the range's first global segment id
    int64_t cap_tiles, cap_hubs;
    int4* tiles;
    int4* hubs_small;
    int4* hubs_big;
    __device__ void tile(int32_t row, int32_t nrows, int32_t nb, int32_t nnz) {
        if (lane_id() == 0 && t < cap_tiles) tiles[t] = make_int4(row, nrows, nb, nnz);
        ++t;
    }
    // Row [a, b) of the nonzeros in nseg segments, the first of them segment `first` of the range.
    __device__ void hub(int32_t row, int32_t a, int32_t b, int32_t first, int32_t nseg) {
        for (int32_t k = lane_id(); k < nseg; k += 32) {
            const int32_t sb = a + k * kRowTileItems;
            if (t + k < cap_tiles)
                tiles[t + k] = make_int4(row, static_cast<int32_t>(-(seg_base + first + k + 1)), sb,
                                         min(kRowTileItems, b - sb));
        }
        t += nseg;
        const int4 h = make_int4(row, static_cast<int32_t>(seg_base + first), nseg, 0);
        if (nseg <= kSmallHubSegs) {
            if (lane_id() == 0 && hs < cap_hubs) hubs_small[hs] = h;
            ++hs;
        } else {
            if (lane_id() == 0 && hb < cap_hubs) hubs_big[hb] = h;
            ++hb;
        }
    }
};

// The greedy walk of a warp over rows [r0, r1); returns the number of hub segments, or -1 on bad offsets.
template <class Sink>
__device__ int32_t plan_range(const int32_t* __restrict__ off, int32_t r0, int32_t r1, int64_t E, Sink& sk) {
    const int lane = lane_id();
    int32_t cur_row = r0, cur_rows = 0, cur_nb = 0, cur_end = 0, segs = 0;  // the open tile, the same in every lane
    int32_t na = 0, nb = 0;  // the lane's row of the next 32, loaded a step ahead
    auto fetch = [&](int32_t c) {
        na = c + lane < r1 ? __ldg(off + c + lane) : 0;
        nb = c + lane < r1 ? __ldg(off + c + lane + 1) : 0;
    };
    fetch(r0);
    for (int32_t c = r0; c < r1; c += 32) {
        const int n = min(32, r1 - c);
        const int32_t r = c + lane;
        const int32_t a = na, b = nb;
        fetch(c + 32);
        if (__any_sync(kFullMask, lane < n && (a < 0 || b < a || b > E))) return -1;
        const bool hub = lane < n && b - a > kHubRowDegree;
        int p = 0;  // next row of the 32
        while (p < n) {
            if (cur_rows == 0) {
                cur_row = c + p;
                cur_nb = __shfl_sync(kFullMask, a, p);
            }
            // Rows that do not fit in the open tile; the first of them, or a hub, ends it.
            const int64_t items = static_cast<int64_t>(b) - cur_nb + (r - cur_row + 1);
            const unsigned m = __ballot_sync(kFullMask, lane < n && lane >= p && (hub || items > kRowTileItems));
            const int q = m ? __ffs(m) - 1 : n;
            if (q > p) {
                cur_rows += q - p;
                cur_end = __shfl_sync(kFullMask, b, q - 1);
            }
            p = q;
            if (q == n) break;
            if (cur_rows > 0) sk.tile(cur_row, cur_rows, cur_nb, cur_end - cur_nb);
            cur_rows = 0;
            if (__shfl_sync(kFullMask, static_cast<int>(hub), q)) {
                const int32_t ha = __shfl_sync(kFullMask, a, q), hb = __shfl_sync(kFullMask, b, q);
                const int32_t nseg = segments_of(hb - ha, kRowTileItems);
                sk.hub(c + q, ha, hb, segs, nseg);
                segs += nseg;
                p = q + 1;
            }
        }
    }
    if (cur_rows > 0) sk.tile(cur_row, cur_rows, cur_nb, cur_end - cur_nb);
    return segs;
}

__device__ __forceinline__ int32_t range_end(int32_t r0, int32_t V) {
    const int64_t end = static_cast<int64_t>(r0) + kPlanRange;
    return static_cast<int32_t>(end < V ? end : V);
}

// counts[4][nranges]: tiles, small hubs, big hubs, segments of each range.
__global__ void __launch_bounds__(kPlanBlock) plan_count_kernel(const int32_t* __restrict__ off, int32_t V, int64_t E,
                                                                int64_t* __restrict__ counts, int32_t nranges, int* bad) {
    const int32_t k = (blockIdx.x * kPlanBlock + threadIdx.x) >> 5;
    if (k >= nranges) return;
    PlanCount c;
    const int32_t r0 = k * kPlanRange;
    const int32_t segs = plan_range(off, r0, range_end(r0, V), E, c);
    if (lane_id() != 0) return;
    if (segs < 0) {
        atomicOr(bad, 4);
        c = PlanCount();
    } else {
        c.segs = segs;
    }
    counts[k] = c.tiles;
    counts[nranges + k] = c.small;
    counts[2 * static_cast<int64_t>(nranges) + k] = c.big;
    counts[3 * static_cast<int64_t>(nranges) + k] = c.segs;
}

// In-place exclusive scan of each of the four count rows; totals[0..3] receive the sums. One block.
__global__ void __launch_bounds__(1024) plan_scan_kernel(int64_t* counts, int32_t nranges, int64_t* totals) {
    __shared__ int64_t s_part[4][1024];
    const int t = threadIdx.x;
    const int32_t per = (nranges + 1023) / 1024;
    const int64_t lo = static_cast<int64_t>(t) * per;
    const int64_t hi = lo + per < nranges ? lo + per : static_cast<int64_t>(nranges);
    for (int q = 0; q < 4; ++q) {
        int64_t acc = 0;
        for (int64_t i = lo; i < hi; ++i) acc += counts[q * static_cast<int64_t>(nranges) + i];
        s_part[q][t] = acc;
    }
    __syncthreads();
    if (t < 128) {  // a warp per row
        const int q = t >> 5, lane = t & 31;
        int64_t run = 0;
        for (int i = lane; i < 1024; i += 32) {
            const int64_t v = s_part[q][i];
            int64_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t u = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= o) incl += u;
            }
            s_part[q][i] = run + incl - v;
            run += __shfl_sync(kFullMask, incl, 31);
        }
        if (lane == 0) totals[q] = run;
    }
    __syncthreads();
    for (int q = 0; q < 4; ++q) {
        int64_t run = s_part[q][t];
        for (int64_t i = lo; i < hi; ++i) {
            int64_t* p = counts + q * static_cast<int64_t>(nranges) + i;
            const int64_t v = *p;
            *p = run;
            run += v;
        }
    }
}

__global__ void __launch_bounds__(kPlanBlock) plan_write_kernel(const int32_t* __restrict__ off, int32_t V, int64_t E,
                                                                const int64_t* __restrict__ bases, int32_t nranges,
                                                                int4* tiles, int64_t cap_tiles, int4* hubs_small,
                                                                int4* hubs_big, int64_t cap_hubs) {
    const int32_t k = (blockIdx.x * kPlanBlock + threadIdx.x) >> 5;
    if (k >= nranges) return;
    PlanWrite w;
    w.t = bases[k];
    w.hs = bases[nranges + k];
    w.hb = bases[2 * static_cast<int64_t>(nranges) + k];
    w.seg_base = bases[3 * static_cast<int64_t>(nranges) + k];
    w.cap_tiles = cap_tiles;
    w.cap_hubs = cap_hubs;
    w.tiles = tiles;
    w.hubs_small = hubs_small;
    w.hubs_big = hubs_big;
    const int32_t r0 = k * kPlanRange;
    plan_range(off, r0, range_end(r0, V), E, w);
}

int32_t plan_ranges(int32_t V) { return V > 0 ? static_cast<int32_t>((static_cast<int64_t>(V) + kPlanRange - 1) / kPlanRange) : 0; }

}  // namespace

// Tiles of a valid CSR: consecutive normal tiles of one run (no hub or range start between them)
// hold more than kRowTileItems merge items per pair, so there are at most 2(V+E)/257 + runs of them;
// a hub of degree d >= 256 gives ceil(d/256) <= d/256 + 1 segments; hubs <= E/256 and runs <=
// hubs + ranges. Hence tiles <= (2V + 5E)/256 + ranges + 1.
RowPlanCaps row_plan_caps(int32_t V, int64_t E) {
    RowPlanCaps c;
    const int64_t ranges = plan_ranges(V);
    c.tiles = (2 * static_cast<int64_t>(V) + 5 * E) / 256 + ranges + 2;
    c.hubs = E / 256 + 1;
    c.scratch_bytes = sizeof(int64_t) * (4 * static_cast<size_t>(ranges > 0 ? ranges : 1) + 4);
    return c;
}

cudaError_t launch_build_row_plan(const int32_t* off, int32_t V, int64_t E, const RowPlanCaps& caps, int4* tiles,
                                  int4* hubs_small, int4* hubs_big, void* scratch, int64_t* totals, int* bad,
                                  cudaStream_t s) {
    const int32_t nr = plan_ranges(V);
    if (nr == 0) return cudaMemsetAsync(totals, 0, 4 * sizeof(int64_t), s);
    int64_t* counts = static_cast<int64_t*>(scratch);
    const int blocks = (nr + kPlanBlock / 32 - 1) / (kPlanBlock / 32);
    plan_count_kernel<<<blocks, kPlanBlock, 0, s>>>(off, V, E, counts, nr, bad);
    plan_scan_kernel<<<1, 1024, 0, s>>>(counts, nr, totals);
    plan_write_kernel<<<blocks, kPlanBlock, 0, s>>>(off, V, E, counts, nr, tiles, caps.tiles, hubs_small, hubs_big,
                                                    caps.hubs);
    return cudaGetLastError();
}

namespace {

// The kernels of a sweep are chained (launch_chained). Same box, 20 sweeps of R-MAT 22 / 608,712 vertices,
// gradient of R-MAT 20 / 50,001 vertices x 8: unchained 3.13 / 0.70, 8.29 / 2.73 ms; gather and fix-up
// chained 3.04 / 0.61, 7.62 / 2.20 ms. Letting the fix-up start ahead of the gather's end cost more than
// it gave (3.15 / 0.72, 8.58 / 2.39 ms).
// A sweep: the gather kernel, then the hub fix-up kernel (which for PageRank also reduces the
// dangling partials). Folding the fix-up into the gather behind a grid barrier (one cooperative
// launch) measured only 0.6 % faster on R-MAT 22: the fix-up's round trips stay on the critical path.
template <int MODE, bool CONV, bool BATCH>
cudaError_t launch_row_sweep(const RowGatherLaunch& L, DevStatus* st, cudaStream_t stream, int sm_count,
                             LaunchHook* hook) {
    int gb, fb, bt;
    rowgather_grid(sm_count, &gb, &fb, &bt);
    // At least one hot entry: the SpMV gather reads entry 0 for cold columns, the sweeps keep a zero.
    const size_t smem = rowgather_staging_bytes(MODE != kModeSpmv) + sizeof(float) * (static_cast<size_t>(L.hot) + 1);
    cudaError_t err = prepare_rowgather<MODE, CONV, BATCH>();
    if (err != cudaSuccess) return err;
    {
        HookScope hs(hook, DPG_KERNEL_ROWGATHER, stream);
        if constexpr (MODE == kModeSpmv) {
            if (L.chained) {
                err = launch_chained(spmv_gather_kernel, gb, bt, smem, stream, L);
            } else {
                spmv_gather_kernel<<<gb, bt, smem, stream>>>(L);
                err = cudaGetLastError();
            }
        } else {
            err = launch_chained(rowgather_kernel<MODE, CONV, BATCH>, gb, bt, smem, stream, L);
        }
    }
    if (err != cudaSuccess) return err;
    if (MODE == kModeSpmv && L.plan.nhub_small + L.plan.nhub_big == 0) return cudaSuccess;
    {
        HookScope hs(hook, DPG_KERNEL_FIXUP, stream);
        err = launch_chained(hub_fixup_kernel<MODE>, fb, kFixBlock, 0, stream, L, gb * (bt / 32), st);
    }
    return err;
}

}  // namespace

cudaError_t launch_spmv(const RowGatherLaunch& L, DevStatus* st, cudaStream_t stream, int sm_count,
                        LaunchHook* hook) {
    return launch_row_sweep<kModeSpmv, false, false>(L, st, stream, sm_count, hook);
}

cudaError_t launch_weighted_sweep(const RowGatherLaunch& L, DevStatus* st, cudaStream_t stream, int sm_count,
                                  LaunchHook* hook) {
    return L.rank_prev ? launch_row_sweep<kModeWeighted, true, false>(L, st, stream, sm_count, hook)
                       : launch_row_sweep<kModeWeighted, false, false>(L, st, stream, sm_count, hook);
}

cudaError_t launch_pagerank_sweep(const RowGatherLaunch& L, DevStatus* st, cudaStream_t stream, int sm_count,
                                  LaunchHook* hook) {
    if (L.vgraph) return launch_row_sweep<kModePagerank, false, true>(L, st, stream, sm_count, hook);
    return L.rank_prev ? launch_row_sweep<kModePagerank, true, false>(L, st, stream, sm_count, hook)
                       : launch_row_sweep<kModePagerank, false, false>(L, st, stream, sm_count, hook);
}

cudaError_t launch_pagerank_init(const RowGatherLaunch& L, float init_rank, float* rank_prev, DevStatus* st,
                                 cudaStream_t stream, int sm_count, LaunchHook* hook) {
    int gb, fb, bt;
    rowgather_grid(sm_count, &gb, &fb, &bt);
    {
        HookScope hs(hook, DPG_KERNEL_INIT, stream);
        // Same number of warps as the gather grid, so dpart[] lines up one slot per warp.
        pr_init_kernel<<<gb * (bt / kInitBlock), kInitBlock, 0, stream>>>(L, init_rank, rank_prev);
    }
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    // A fix-up pass over no hubs reduces the initial dangling partials into dsum_out.
    RowGatherLaunch F = L;
    F.nonstop = nullptr;
    F.plan.nhub_small = 0;
    F.plan.nhub_big = 0;
    {
        HookScope hs(hook, DPG_KERNEL_INIT, stream);
        hub_fixup_kernel<kModePagerank><<<fb, kFixBlock, 0, stream>>>(F, gb * (bt / 32), st);
    }
    return cudaGetLastError();
}

}  // namespace dpg
