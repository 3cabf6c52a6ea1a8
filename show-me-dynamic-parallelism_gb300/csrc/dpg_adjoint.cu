// Batched right-hand sides and the SpMV adjoint: Y = A X, dX = A^T G, dA[e] = <G[row(e)], X[col(e)]>.
//
// No counterpart in the reference (its SpMV, apps/SpMV/src/SpMV_kernel.cu:81-96, multiplies one
// vector). With nrhs columns stored row-major ([V][nrhs] FP32), every nonzero touches whole rows of
// 4 * nrhs bytes.
//   rows_kernel           Y[row] = sum over the row's nonzeros of val * X[col] (Y = A X), or, over the
//                         transposed CSR, both gradients in one pass (dX = A^T G and dA). Takes nrhs
//                         a multiple of 4 with 16-byte aligned row blocks, and any nrhs up to 32.
//   spmm_rows_kernel      Y = A X for the other shapes, a warp per row
//   arc_dot_kernel        dA[e] = <G[row], X[col(e)]> for the other shapes
// Rows of more than kGroupRow nonzeros are listed in a plan (built on the device) as items of at most
// kSpmmSegment nonzeros; a row of several items writes partial rows that a fix-up adds in segment
// order. The others are read straight from the offsets. Every sum has a fixed order.
#include <cuda_runtime.h>

#include <algorithm>

#include "dpg_kernels.h"

namespace dpg {
namespace {

constexpr int kBlock = 256;

template <int NV>
__device__ __forceinline__ void load_row(const float* __restrict__ M, int64_t r, int nrhs, int lane, float (&v)[NV]) {
    const float* p = M + r * nrhs;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const int j = lane + 32 * q;
        v[q] = j < nrhs ? __ldg(p + j) : 0.0f;
    }
}

// The warp's k-th job of a plan: the listed items first, then the rows of at most kGroupRow nonzeros
// (a longer row reads as empty with row -1: its items were listed).
__device__ __forceinline__ int4 plan_job(const SpmmPlanDev& P, int64_t k) {
    if (k < P.nitems) return __ldg(P.items + k);
    const int v = static_cast<int>(k - P.nitems);
    const int b = __ldg(P.off + v), e = __ldg(P.off + v + 1);
    return e - b > kGroupRow ? make_int4(-1, 0, 0, -1) : make_int4(v, b, e, -1);
}

// One warp per job {row, arc begin, arc end, segment or -1}; 4 nonzeros in flight.
template <int NV>
__global__ void __launch_bounds__(kBlock) spmm_rows_kernel(SpmmPlanDev P,
                                                           const int32_t* __restrict__ col, const float* __restrict__ val,
                                                           const float* __restrict__ X, int nrhs, float* __restrict__ Y,
                                                           float* __restrict__ partial) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int64_t njobs = static_cast<int64_t>(P.nitems) + P.V;
    for (int64_t k = w; k < njobs; k += nw) {
        const int4 I = plan_job(P, k);
        if (I.x < 0) continue;
        float acc[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) acc[q] = 0.0f;
        int e = I.y;
        for (; I.z - e >= 4; e += 4) {
            int c[4];
            float a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = __ldg(col + e + u);
                a[u] = __ldg(val + e + u);
            }
            float xv[4][NV];
#pragma unroll
            for (int u = 0; u < 4; ++u) load_row<NV>(X, c[u], nrhs, lane, xv[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int q = 0; q < NV; ++q) acc[q] = fmaf(a[u], xv[u][q], acc[q]);
        }
        for (; e < I.z; ++e) {
            const int c = __ldg(col + e);
            const float a = __ldg(val + e);
            float xv[NV];
            load_row<NV>(X, c, nrhs, lane, xv);
#pragma unroll
            for (int q = 0; q < NV; ++q) acc[q] = fmaf(a, xv[q], acc[q]);
        }
        float* dst = I.w < 0 ? Y + static_cast<int64_t>(I.x) * nrhs : partial + static_cast<int64_t>(I.w) * nrhs;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const int j = lane + 32 * q;
            if (j < nrhs) dst[j] = acc[q];
        }
    }
}

// Split rows: Y[row] = sum of its segments' partial rows, in segment order; with TREE (segments shorter than
// kSpmmSegment, so more of them) every eight are added as a tree first and eight of those sums set aside, which
// keeps the chain of roundings shorter than that of segments of kSpmmSegment. Warp per split row.
template <int NV, bool TREE = false>
__global__ void __launch_bounds__(kBlock) spmm_fixup_kernel(const int4* __restrict__ hubs, int nhubs,
                                                            const float* __restrict__ partial, int nrhs,
                                                            float* __restrict__ Y) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int h = w; h < nhubs; h += nw) {
        const int4 H = __ldg(hubs + h);
        float acc[NV], aside[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) acc[q] = aside[q] = 0.0f;
        for (int s0 = 0; s0 < H.z; s0 += 8) {  // 8 partial rows in flight, added in segment order
            float pv[8][NV];
#pragma unroll
            for (int u = 0; u < 8; ++u) load_row<NV>(partial, H.y + min(s0 + u, H.z - 1), nrhs, lane, pv[u]);
            if constexpr (TREE) {
#pragma unroll
                for (int q = 0; q < NV; ++q) {
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (s0 + u >= H.z) pv[u][q] = 0.0f;
                    acc[q] += ((pv[0][q] + pv[1][q]) + (pv[2][q] + pv[3][q])) + ((pv[4][q] + pv[5][q]) + (pv[6][q] + pv[7][q]));
                    if (s0 % 64 == 56) {
                        aside[q] += acc[q];
                        acc[q] = 0.0f;
                    }
                }
            } else {
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int q = 0; q < NV; ++q)
                        if (s0 + u < H.z) acc[q] += pv[u][q];
            }
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const int j = lane + 32 * q;
            if (j < nrhs) Y[static_cast<int64_t>(H.x) * nrhs + j] = TREE ? aside[q] + acc[q] : acc[q];
        }
    }
}

// One column: dA[e] = G[row] * X[col(e)]: a warp per listed item, 8 lanes per other row (most rows of a power-law graph
// hold a few arcs: R-MAT 22 0.37 ms, 0.53 with a warp per row).
__global__ void __launch_bounds__(kBlock) arc_dot1_kernel(SpmmPlanDev P, const int32_t* __restrict__ col,
                                                          const float* __restrict__ X, const float* __restrict__ G,
                                                          float* __restrict__ dA) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (gridDim.x * blockDim.x) >> 5;
    for (int64_t k = w; k < P.nitems; k += nw) {
        const int4 I = __ldg(P.items + k);
        const float g = __ldg(G + I.x);
        for (int t = lane; t < I.z - I.y; t += 32) dA[I.y + t] = g * __ldg(X + __ldg(col + I.y + t));
    }
    for (int64_t v = w * 4 + (lane >> 3); v < P.V; v += nw * 4) {
        const int b = __ldg(P.off + v), n = __ldg(P.off + v + 1) - b;
        if (n > kGroupRow) continue;  // its items are listed
        const float g = __ldg(G + v);
        for (int t = lane & 7; t < n; t += 8) dA[b + t] = g * __ldg(X + __ldg(col + b + t));
    }
}

// dA[e] = <G[row], X[col(e)]> for the item's arcs; the warp keeps G[row] in registers.
template <int NV>
__global__ void __launch_bounds__(kBlock) arc_dot_kernel(SpmmPlanDev P,
                                                         const int32_t* __restrict__ col, const float* __restrict__ X,
                                                         const float* __restrict__ G, int nrhs, float* __restrict__ dA) {
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int64_t njobs = static_cast<int64_t>(P.nitems) + P.V;
    for (int64_t k = w; k < njobs; k += nw) {
        const int4 I = plan_job(P, k);
        if (I.x < 0) continue;
        float g[NV];
        load_row<NV>(G, I.x, nrhs, lane, g);
        int e = I.y;
        for (; I.z - e >= 4; e += 4) {
            float xv[4][NV];
#pragma unroll
            for (int u = 0; u < 4; ++u) load_row<NV>(X, __ldg(col + e + u), nrhs, lane, xv[u]);
            float d[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                d[u] = 0.0f;
#pragma unroll
                for (int q = 0; q < NV; ++q) d[u] = fmaf(g[q], xv[u][q], d[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) d[u] = warp_sum_f32(d[u]);
            if (lane < 4) {
                const float mine = lane == 0 ? d[0] : lane == 1 ? d[1] : lane == 2 ? d[2] : d[3];
                dA[e + lane] = mine;
            }
        }
        for (; e < I.z; ++e) {
            float xv[NV];
            load_row<NV>(X, __ldg(col + e), nrhs, lane, xv);
            float d = 0.0f;
#pragma unroll
            for (int q = 0; q < NV; ++q) d = fmaf(g[q], xv[q], d);
            d = warp_sum_f32(d);
            if (lane == 0) dA[e] = d;
        }
    }
}

__global__ void gather_values_kernel(const float* __restrict__ v, const int32_t* __restrict__ idx, int64_t n,
                                     float* __restrict__ out) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[i] = __ldg(v + __ldg(idx + i));
}

// ---- rows in groups of lanes -----------------------------------------------------------------------
// A gathered row of nrhs floats is Q vectors of VEC floats (float4, or single floats for widths and
// alignments that do not allow it), one per lane of LQ lanes (the power of two from Q up). A group of
// GL = max(8, LQ) lanes works through rows of its own (at most kGroupRow nonzeros), with 8 / LQ arcs
// side by side when LQ < 8, A arcs per step, and moves to its next row in the step after the last
// arc, whatever the other groups do. The indexes of the next step and the offsets of the next row are
// loaded one step ahead, so a step costs one round trip (the gathered rows). The listed items of
// longer rows are taken by whole warps, the groups interleaved.
// Summation order: a lane adds its arcs in order; the groups' (and side-by-side arcs') sums meet in a
// fixed butterfly.
struct RowsLaunch {
    SpmmPlanDev P;
    const int32_t* col;   // row of `in` that each arc gathers
    const int32_t* arc;   // kBwdArcs: index of each arc in val and dA
    const float* val;     // (kForward, kBwdSlots: in the order of col)
    const float* in;      // gathered matrix (X, or G for the backward)
    const float* X;       // backward: dA = <gathered row, X[own row]>
    int nrhs;
    float* out;           // Y or dX; null: skip (backward)
    float* partial;
    float* dA;            // backward; null: skip (kBwdSlots: in the order of col)
};
enum RowsMode { kForward, kBwdArcs, kBwdSlots };

template <int VEC>
struct RowVec;
template <>
struct RowVec<4> {
    float4 v;
    __device__ __forceinline__ static RowVec zero() { return {make_float4(0.f, 0.f, 0.f, 0.f)}; }
    // Zero unless `on`: one predicated load. As a conditional expression it became a branch whose
    // zeroing side waited for the loads in flight of the other lanes (R-MAT 22 x 64 backward: 8.5 -> 6.3
    // ms, with two vectors per lane).
    __device__ __forceinline__ static RowVec load_if(bool on, const float* p) {
        RowVec r = zero();
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
            : "+f"(r.v.x), "+f"(r.v.y), "+f"(r.v.z), "+f"(r.v.w) : "l"(p), "r"(static_cast<int>(on)));
        return r;
    }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = v; }
    __device__ __forceinline__ void fma(float a, const RowVec& x) {
        v.x = fmaf(a, x.v.x, v.x);
        v.y = fmaf(a, x.v.y, v.y);
        v.z = fmaf(a, x.v.z, v.z);
        v.w = fmaf(a, x.v.w, v.w);
    }
    __device__ __forceinline__ float dot(const RowVec& x, float d) const {
        return fmaf(v.w, x.v.w, fmaf(v.z, x.v.z, fmaf(v.y, x.v.y, fmaf(v.x, x.v.x, d))));
    }
    __device__ __forceinline__ void add(const RowVec& x) {
        v.x += x.v.x;
        v.y += x.v.y;
        v.z += x.v.z;
        v.w += x.v.w;
    }
    __device__ __forceinline__ void add_xor(int m) {
        v.x += __shfl_xor_sync(kFullMask, v.x, m);
        v.y += __shfl_xor_sync(kFullMask, v.y, m);
        v.z += __shfl_xor_sync(kFullMask, v.z, m);
        v.w += __shfl_xor_sync(kFullMask, v.w, m);
    }
};
template <>
struct RowVec<1> {
    float v;
    __device__ __forceinline__ static RowVec zero() { return {0.f}; }
    __device__ __forceinline__ static RowVec load_if(bool on, const float* p) {
        RowVec r = zero();
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}"
            : "+f"(r.v) : "l"(p), "r"(static_cast<int>(on)));
        return r;
    }
    __device__ __forceinline__ void store(float* p) const { *p = v; }
    __device__ __forceinline__ void fma(float a, const RowVec& x) { v = fmaf(a, x.v, v); }
    __device__ __forceinline__ float dot(const RowVec& x, float d) const { return fmaf(v, x.v, d); }
    __device__ __forceinline__ void add(const RowVec& x) { v += x.v; }
    __device__ __forceinline__ void add_xor(int m) { v += __shfl_xor_sync(kFullMask, v, m); }
};

// CTAs per SM the kernel is compiled for and launched with.
// Measured on the same box against the kernels before it (a warp per row: a chain of three dependent
// loads for every row, most of which have fewer than 4 arcs; float4 rows for multiples of 32 only):
//   Y = A X, 200,003 rows x 16, 20 columns 185 -> 70 us; R-MAT 20 x 1 / 3 / 64 / 100 / 128 columns
//   678 -> 118, 682 -> 147, 830 -> 631, 1284 -> 1024, 1385 -> 1056 us
//   backward, 237,987 rows x 32, 1 / 20 columns 445 -> 119, 949 -> 233 us; R-MAT 20 x 32 / 96 columns
//   997 -> 866, 1851 -> 1711 us; R-MAT 22 x 64 columns 5.78 -> 5.63 ms
// Gathered vectors in flight per lane and CTAs per SM: 8 vectors, or 3 or 5 CTAs, were slower on most
// of these (backward R-MAT 22 x 64: 6.0 ms with 8, 6.3 with 3 or 5). More vectors per lane and 8-lane
// groups for the wide rows (fewer shuffles) were slower too: 6.3 ms, and 1.66 against 1.06 ms for Y = A X
// with 128 columns.
constexpr int kRowLoads = 4;
constexpr int rows_blocks(int vec) { return vec == 1 ? 5 : 4; }

// Arc positions are unsigned: near 2^31 nonzeros a step may reach past INT32_MAX.
// Indexes of one step of a group: lane l holds arcs p + l, p + 8 + l, ... (zero past the end).
template <int R, int MODE>
struct StepIdx {
    int c[R];
    int a[R];    // kBwdArcs: arc
    float w[R];  // else: value
    __device__ __forceinline__ void load(const RowsLaunch& L, unsigned p, unsigned e, int gl) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const unsigned t = p + 8 * r + gl;
            const bool in = t < e;
            c[r] = in ? __ldg(L.col + t) : 0;
            if (MODE == kBwdArcs) a[r] = in ? __ldg(L.arc + t) : 0;
            else w[r] = in ? __ldg(L.val + t) : 0.0f;
        }
    }
};

template <int VEC, int LQ, int MODE>
__global__ void __launch_bounds__(kBlock, rows_blocks(VEC)) rows_kernel(RowsLaunch L) {
    using V = RowVec<VEC>;
    constexpr bool BWD = MODE != kForward;
    constexpr int GL = LQ < 8 ? 8 : LQ;                 // lanes of a group
    constexpr int NG = 32 / GL;                         // groups of a warp
    constexpr int AP = LQ < 8 ? 8 / LQ : 1;             // arcs side by side in a group
    constexpr int NB = 8 / AP;                          // batches of AP arcs in 8 arcs
    constexpr int R = LQ == 1 ? 4 : LQ == 2 ? 2 : 1;    // index loads per lane and step
    constexpr int A = 8 * R;                            // arcs per step
    constexpr int HB = NB < kRowLoads ? NB : kRowLoads;  // gathered vectors in flight per lane
    const int lane = threadIdx.x & 31;
    const int grp = lane / GL, gl = lane & 7, gbase = grp * GL;  // gl: the arc of 8 whose indexes the lane loads
    const int q0 = lane % LQ, sub = (lane % GL) / LQ;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const bool live = q0 < L.nrhs / VEC;
    V acc, xj;

    auto load_own = [&](int row, bool any) {  // backward: X[row], of a row that has arcs
        if (!BWD) return;
        xj = V::load_if(any && L.dA && live, L.X + static_cast<int64_t>(row) * L.nrhs + VEC * q0);
    };
    // The arcs [p, min(p + A, e)) of the group.
    auto step = [&](unsigned p, unsigned e, const StepIdx<R, MODE>& I) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float wv = 0.0f;
            if (MODE == kBwdArcs) wv = p + 8 * r + gl < e ? __ldg(L.val + I.a[r]) : 0.0f;
            else wv = I.w[r];
            float d[NB];
#pragma unroll
            for (int h = 0; h < NB; h += HB) {
                // Slots past the end load nothing and hold zeros, value and row (an Inf in a row that
                // no arc touches must not reach 0 * Inf).
                V x[HB];
#pragma unroll
                for (int i = 0; i < HB; ++i) {
                    const int u = (h + i) * AP + sub;
                    const int row = __shfl_sync(kFullMask, I.c[r], gbase + u);
                    const bool in = p + 8 * r + u < e;
                    x[i] = V::load_if(in && live, L.in + static_cast<int64_t>(row) * L.nrhs + VEC * q0);
                }
#pragma unroll
                for (int i = 0; i < HB; ++i) {
                    const int u = (h + i) * AP + sub;
                    const float a = __shfl_sync(kFullMask, wv, gbase + u);
                    acc.fma(a, x[i]);
                    if (BWD) d[h + i] = x[i].dot(xj, 0.0f);
                }
            }
            if (BWD && L.dA) {
                // Sum of each arc's dot over its LQ lanes: every exchange halves the arcs a lane still
                // holds, down to one, whose sum the lanes left then complete.
                int batch = 0;
#pragma unroll
                for (int m = LQ / 2, n = NB / 2; m > 0; m >>= 1, n >>= 1) {
                    if (n > 0) {
                        const bool up = (q0 & m) != 0;
                        if (up) batch += n;
#pragma unroll
                        for (int k = 0; k < n; ++k) {
                            const float send = up ? d[k] : d[k + n];
                            const float keep = up ? d[k + n] : d[k];
                            d[k] = keep + __shfl_xor_sync(kFullMask, send, m);
                        }
                    } else {
                        d[0] += __shfl_xor_sync(kFullMask, d[0], m);
                    }
                }
                const int u = batch * AP + sub;
                unsigned arc = p + 8 * r + u;
                if (MODE == kBwdArcs) arc = __shfl_sync(kFullMask, I.a[r], gbase + u);
                if (p + 8 * r + u < e && (LQ <= NB || q0 % (LQ / NB) == 0)) L.dA[arc] = d[0];
            }
        }
    };

    // Listed items, a warp each.
    for (int it = w; it < L.P.nitems; it += nw) {
        const int4 I = __ldg(L.P.items + it);
        acc = V::zero();
        load_own(I.x, true);
        StepIdx<R, MODE> cur, nxt;
        const unsigned end = I.z;
        cur.load(L, I.y + grp * A, end, gl);
        // Every 64 arcs of a lane the sum so far is set aside, which keeps the chain of roundings short.
        V total = V::zero();
        for (unsigned base = I.y, k = 1; base < end; base += NG * A, ++k) {
            nxt.load(L, base + (NG + grp) * A, end, gl);
            step(base + grp * A, end, cur);
            cur = nxt;
            if (k * A % (64 * AP) == 0) {
                total.add(acc);
                acc = V::zero();
            }
        }
        if (!L.out) continue;
        acc.add(total);
#pragma unroll
        for (int m = LQ; m < 32; m <<= 1) acc.add_xor(m);
        if (grp == 0 && sub == 0 && live)
            acc.store((I.w < 0 ? L.out + static_cast<int64_t>(I.x) * L.nrhs
                               : L.partial + static_cast<int64_t>(I.w) * L.nrhs) + VEC * q0);
    }

    // The other rows, a group each. A listed row reads as empty and is not stored.
    const int64_t ngroups = static_cast<int64_t>(nw) * NG;
    auto range = [&](int64_t v, unsigned& b, unsigned& e, bool& mine) {
        mine = v < L.P.V;
        b = mine ? __ldg(L.P.off + v) : 0;
        e = mine ? __ldg(L.P.off + v + 1) : 0;
        if (e - b > kGroupRow) {
            e = b;
            mine = false;
        }
    };
    int64_t v = static_cast<int64_t>(w) * NG + grp;
    unsigned p, e, nb, ne;
    bool mine, nmine;
    range(v, p, e, mine);
    range(v + ngroups, nb, ne, nmine);
    StepIdx<R, MODE> cur, nxt;
    cur.load(L, p, e, gl);
    acc = V::zero();
    load_own(static_cast<int>(v), mine && p < e);
    while (__any_sync(kFullMask, v < L.P.V)) {
        const bool last = p + A >= e;
        nxt.load(L, last ? nb : p + A, last ? ne : e, gl);
        unsigned nnb = 0, nne = 0;
        bool nnmine = false;
        if (last) range(v + 2 * ngroups, nnb, nne, nnmine);
        step(p, e, cur);
        if (AP > 1 && __any_sync(kFullMask, last)) {
            V t = acc;
#pragma unroll
            for (int m = LQ; m < 8; m <<= 1) t.add_xor(m);
            if (last) acc = t;
        }
        if (last) {
            if (mine && L.out && sub == 0 && live) acc.store(L.out + v * L.nrhs + VEC * q0);
            v += ngroups;
            p = nb;
            e = ne;
            mine = nmine;
            nb = nnb;
            ne = nne;
            nmine = nnmine;
            acc = V::zero();
            load_own(static_cast<int>(v), mine && p < e);
        } else {
            p += A;
        }
        cur = nxt;
    }
}

// ---- arc values between CSR order and transposed order -----------------------------------------------
// A permutation of E values in two passes over blocks of kPermBlock that fit in shared memory, every
// global access a run: arcs are cut into chunks and transposed slots into buckets of kPermBlock each,
// and a middle order holds the values by bucket, then chunk. Position i of a chunk (in middle order)
// is arc arc_in[i] of the chunk and middle position mid[i]; middle position t of a bucket is slot
// slot_in[t] of the bucket. The chunk pass moves runs of about kPermBlock^2 / E values to or from the
// middle order, the bucket pass whole blocks. What it replaces: one random 4-byte access per arc, a
// DRAM line each (45 G/s): the 64-column backward of R-MAT 22 took 5.6 ms with its value reads and
// gradient writes at random, of which the pass itself is 3.2 ms. Permuting through windows of slots
// that fit in L2 (one pass, random writes there) took 1.0 ms per permutation, this 0.40 ms; the call
// went from 5.65 to 4.14 ms. Blocks of 28,672 / 24,576 / 20,480 values, two CTAs per SM: 4.22 / 4.14 / 4.23
// ms; 32,768 in one CTA with its loads ahead: 4.77 ms (same box).
constexpr int kPermThreads = 1024;

// slot_of[arc] = transposed slot.
__global__ void __launch_bounds__(kBlock) invert_kernel(const int32_t* __restrict__ arc, int64_t E, int32_t* slot_of) {
    for (int64_t p = static_cast<int64_t>(blockIdx.x) * kBlock + threadIdx.x; p < E;
         p += static_cast<int64_t>(gridDim.x) * kBlock)
        slot_of[__ldg(arc + p)] = static_cast<int32_t>(p);
}

// counts[bucket][chunk]: arcs of the chunk whose slot lies in the bucket.
__global__ void __launch_bounds__(kPermThreads) perm_count_kernel(const int32_t* __restrict__ slot_of, int64_t E,
                                                                  int nblk, int32_t* __restrict__ counts) {
    extern __shared__ int s_n[];
    for (int c = blockIdx.x; c < nblk; c += gridDim.x) {
        for (int i = threadIdx.x; i < nblk; i += kPermThreads) s_n[i] = 0;
        __syncthreads();
        const int64_t e0 = static_cast<int64_t>(c) * kPermBlock;
        const int n = static_cast<int>(E - e0 < kPermBlock ? E - e0 : kPermBlock);
        for (int i = threadIdx.x; i < n; i += kPermThreads) atomicAdd(s_n + __ldg(slot_of + e0 + i) / kPermBlock, 1);
        __syncthreads();
        for (int i = threadIdx.x; i < nblk; i += kPermThreads) counts[static_cast<int64_t>(i) * nblk + c] = s_n[i];
        __syncthreads();
    }
}

// Sum over the block's threads before this one (kPermThreads threads).
__device__ __forceinline__ int block_exclusive(int v, int* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int incl = warp_inclusive_scan(v);
    __syncthreads();
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += s_warp[w];
    return before + incl - v;
}

// counts[bucket][chunk] becomes the middle position of the run's first value: a bucket's slots fill it
// exactly, so each row is scanned on its own from bucket * kPermBlock.
__global__ void __launch_bounds__(kPermThreads) perm_scan_kernel(int nblk, int32_t* __restrict__ counts) {
    __shared__ int s_warp[32];
    for (int b = blockIdx.x; b < nblk; b += gridDim.x) {
        int32_t* row = counts + static_cast<int64_t>(b) * nblk;
        const int per = (nblk + kPermThreads - 1) / kPermThreads;
        const int lo = min(nblk, static_cast<int>(threadIdx.x) * per), hi = min(nblk, lo + per);
        int sum = 0;
        for (int i = lo; i < hi; ++i) sum += row[i];
        int64_t run = static_cast<int64_t>(b) * kPermBlock + block_exclusive(sum, s_warp);
        for (int i = lo; i < hi; ++i) {
            const int v = row[i];
            row[i] = static_cast<int32_t>(run);
            run += v;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kPermThreads) perm_place_kernel(const int32_t* __restrict__ slot_of, int64_t E,
                                                                  int nblk, const int32_t* __restrict__ starts,
                                                                  int32_t* __restrict__ mid,
                                                                  uint16_t* __restrict__ arc_in,
                                                                  uint16_t* __restrict__ slot_in) {
    extern __shared__ int s_n[];
    int* s_first = s_n;         // middle position of the chunk's run in each bucket
    int* s_next = s_n + nblk;   // next free one
    __shared__ int s_warp[32];
    for (int c = blockIdx.x; c < nblk; c += gridDim.x) {
        const int64_t e0 = static_cast<int64_t>(c) * kPermBlock;
        const int n = static_cast<int>(E - e0 < kPermBlock ? E - e0 : kPermBlock);
        // Run lengths again (the starts of the next chunk are those of this one plus its length, but
        // the last chunk has no next), then each run's first position in the chunk.
        for (int i = threadIdx.x; i < nblk; i += kPermThreads) s_next[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += kPermThreads) atomicAdd(s_next + __ldg(slot_of + e0 + i) / kPermBlock, 1);
        __syncthreads();
        const int per = (nblk + kPermThreads - 1) / kPermThreads;
        const int lo = min(nblk, static_cast<int>(threadIdx.x) * per), hi = min(nblk, lo + per);
        int sum = 0;
        for (int b = lo; b < hi; ++b) sum += s_next[b];
        int local = block_exclusive(sum, s_warp);
        for (int b = lo; b < hi; ++b) {
            const int first = starts[static_cast<int64_t>(b) * nblk + c];
            const int len = s_next[b];
            s_first[b] = first - local;  // middle position minus position in the chunk, the same for the run
            s_next[b] = first;
            local += len;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += kPermThreads) {
            const int p = __ldg(slot_of + e0 + i);
            const int b = p / kPermBlock;
            const int t = atomicAdd(s_next + b, 1);
            const int64_t k = e0 + (t - s_first[b]);
            mid[k] = t;
            arc_in[k] = static_cast<uint16_t>(i);
            slot_in[t] = static_cast<uint16_t>(p - b * kPermBlock);
        }
        __syncthreads();
    }
}

// Block by block: the block's linear values into shared memory, then out[mid ? mid[i] : i] = value
// idx[i] of the block. Two CTAs per SM: while one loads, the other writes.
__global__ void __launch_bounds__(kPermThreads, 2) perm_out_kernel(const float* __restrict__ in, int64_t E, int nblk,
                                                                   const uint16_t* __restrict__ idx,
                                                                   const int32_t* __restrict__ mid,
                                                                   float* __restrict__ out) {
    extern __shared__ float s_v[];
    for (int c = blockIdx.x; c < nblk; c += gridDim.x) {
        const int64_t e0 = static_cast<int64_t>(c) * kPermBlock;
        const int n = static_cast<int>(E - e0 < kPermBlock ? E - e0 : kPermBlock);
#pragma unroll 7
        for (int i = threadIdx.x; i < n; i += kPermThreads) s_v[i] = __ldcs(in + e0 + i);
        __syncthreads();
#pragma unroll 7
        for (int i = threadIdx.x; i < n; i += kPermThreads)
            out[mid ? __ldcs(mid + e0 + i) : e0 + i] = s_v[__ldcs(idx + e0 + i)];
        __syncthreads();
    }
}

// The other way: value idx[i] of the block = in[mid ? mid[i] : i], then the block goes out linearly.
__global__ void __launch_bounds__(kPermThreads, 2) perm_in_kernel(const float* __restrict__ in, int64_t E, int nblk,
                                                                  const uint16_t* __restrict__ idx,
                                                                  const int32_t* __restrict__ mid,
                                                                  float* __restrict__ out) {
    extern __shared__ float s_v[];
    for (int c = blockIdx.x; c < nblk; c += gridDim.x) {
        const int64_t e0 = static_cast<int64_t>(c) * kPermBlock;
        const int n = static_cast<int>(E - e0 < kPermBlock ? E - e0 : kPermBlock);
#pragma unroll 7
        for (int i = threadIdx.x; i < n; i += kPermThreads)
            s_v[__ldcs(idx + e0 + i)] = __ldcs(in + (mid ? __ldcs(mid + e0 + i) : e0 + i));
        __syncthreads();
#pragma unroll 7
        for (int i = threadIdx.x; i < n; i += kPermThreads) out[e0 + i] = s_v[i];
        __syncthreads();
    }
}

template <int NV>
cudaError_t run_spmm(const SpmmPlanDev& P, const int32_t* col, const float* val, const float* X, int nrhs, float* Y,
                     float* partial, cudaStream_t s, int sm_count, LaunchHook* hook) {
    {
        HookScope hs(hook, DPG_KERNEL_ROWGATHER, s);
        spmm_rows_kernel<NV><<<sm_count * 8, kBlock, 0, s>>>(P, col, val, X, nrhs, Y, partial);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || P.nhubs == 0) return e;
    {
        HookScope hs(hook, DPG_KERNEL_FIXUP, s);
        spmm_fixup_kernel<NV><<<sm_count * 4, kBlock, 0, s>>>(P.hubs, P.nhubs, partial, nrhs, Y);
    }
    return cudaGetLastError();
}

template <int NV>
cudaError_t run_arc_dot(const SpmmPlanDev& P, const int32_t* col, const float* X, const float* G, int nrhs, float* dA,
                        cudaStream_t s, int sm_count, LaunchHook* hook) {
    HookScope hs(hook, DPG_KERNEL_ROWGATHER, s);
    arc_dot_kernel<NV><<<sm_count * 8, kBlock, 0, s>>>(P, col, X, G, nrhs, dA);
    return cudaGetLastError();
}

}  // namespace

namespace {

// Rows of more than kGroupRow nonzeros into the item list, the whole warp writing one row's segments
// at a time. Positions come from atomics: the order of the lists changes nothing in the results.
__global__ void __launch_bounds__(kBlock) spmm_plan_kernel(const int32_t* __restrict__ off, int32_t V, int segment,
                                                           int4* items, int4* hubs, int32_t* counts) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t v0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x - lane; v0 < V; v0 += stride) {
        const int64_t v = v0 + lane;
        const int b = v < V ? __ldg(off + v) : 0;
        const int e = v < V ? __ldg(off + v + 1) : 0;
        const int d = e - b;
        const int n = d > kGroupRow ? segments_of(d, segment) : 0;
        int pos = 0, seg = -1;
        if (n > 0) pos = atomicAdd(counts, n);
        if (n > 1) {
            seg = atomicAdd(counts + 2, n);
            hubs[atomicAdd(counts + 1, 1)] = make_int4(static_cast<int>(v), seg, n, 0);
        }
        unsigned m = __ballot_sync(kFullMask, n > 0);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1u;
            const int rb = __shfl_sync(kFullMask, b, src), re = __shfl_sync(kFullMask, e, src);
            const int rn = __shfl_sync(kFullMask, n, src), rp = __shfl_sync(kFullMask, pos, src);
            const int rs = __shfl_sync(kFullMask, seg, src);
            for (int k = lane; k < rn; k += 32) {
                const int sb = rb + k * segment;
                items[rp + k] = make_int4(static_cast<int>(v0) + src, sb, segment_end(sb, re, segment), rs < 0 ? -1 : rs + k);
            }
        }
    }
}

}  // namespace

// A warp takes the arcs of an item 16 at a time with up to 64 columns and 8 at a time with more, two round trips
// each, so an item of 512 is a chain of 64 or 128 round trips; in a small matrix that is the whole call, while most
// warps have nothing. The items are halved until there could be one for each of the 32 warps of every SM.
// R-MAT, same box, items of 512 / this rule (and the kernels before this layout, of 4 groups per item): backward of
// 64 columns, 2,048 vertices x 8 37 / 18 us (27), 10,007 x 16 49 / 29 (37), 60,001 x 16 74 / 68 (101); of 128 columns
// 51 / 22 (27), 57 / 33 (40), 108 / 96 (144); 200,003 x 16 has 512 either way. Narrow widths take 32 to 128 arcs a
// step, and the longer fix-up costs them more than that: 3 columns, 25,013 x 16 26.6 / 28.7.
int32_t spmm_short_segment(int64_t E, int sm_count) {
    int32_t segment = kSpmmSegment;
    while (segment > kGroupRow && E / segment < static_cast<int64_t>(sm_count) * 32) segment /= 2;
    return segment;
}

// A listed row of d nonzeros has ceil(d / segment) <= d / segment + 1 items.
int64_t spmm_plan_max_items(int64_t E, int32_t segment) { return E / segment + E / (kGroupRow + 1) + 1; }
int64_t spmm_plan_max_hubs(int64_t E, int32_t segment) { return E / (segment + 1) + 1; }

cudaError_t launch_spmm_plan(const int32_t* off, int32_t V, int32_t segment, int4* items, int4* hubs, int32_t* counts,
                             cudaStream_t s, int sm_count) {
    const cudaError_t e = cudaMemsetAsync(counts, 0, 3 * sizeof(int32_t), s);
    if (e != cudaSuccess || V <= 0) return e;
    const int64_t blocks = (static_cast<int64_t>(V) + kBlock - 1) / kBlock;
    spmm_plan_kernel<<<static_cast<int>(std::min<int64_t>(blocks, sm_count * 8)), kBlock, 0, s>>>(off, V, segment, items,
                                                                                                  hubs, counts);
    return cudaGetLastError();
}

cudaError_t launch_spmm(const SpmmPlanDev& P, const int32_t* col, const float* val, const float* X, int nrhs, float* Y,
                        float* partial, cudaStream_t s, int sm_count, LaunchHook* hook) {
    if (nrhs <= 32) return run_spmm<1>(P, col, val, X, nrhs, Y, partial, s, sm_count, hook);
    if (nrhs <= 64) return run_spmm<2>(P, col, val, X, nrhs, Y, partial, s, sm_count, hook);
    return run_spmm<4>(P, col, val, X, nrhs, Y, partial, s, sm_count, hook);
}

cudaError_t launch_arc_dot(const SpmmPlanDev& P, const int32_t* col, const float* X, const float* G, int nrhs,
                           float* dA, cudaStream_t s, int sm_count, LaunchHook* hook) {
    if (nrhs == 1) {
        HookScope hs(hook, DPG_KERNEL_ROWGATHER, s);
        arc_dot1_kernel<<<sm_count * 8, kBlock, 0, s>>>(P, col, X, G, dA);
        return cudaGetLastError();
    }
    if (nrhs <= 32) return run_arc_dot<1>(P, col, X, G, nrhs, dA, s, sm_count, hook);
    if (nrhs <= 64) return run_arc_dot<2>(P, col, X, G, nrhs, dA, s, sm_count, hook);
    return run_arc_dot<4>(P, col, X, G, nrhs, dA, s, sm_count, hook);
}

bool spmm_rows_ok(int nrhs, const void* a, const void* b, const void* c, const void* d) {
    if (nrhs <= 32) return true;
    if (nrhs % 4 != 0 || nrhs > 128) return false;
    for (const void* p : {a, b, c, d})
        if (p && reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
    return true;
}

namespace {

template <int VEC, int LQ, int MODE>
cudaError_t run_rows(const RowsLaunch& L, bool tree, cudaStream_t s, int sm_count, LaunchHook* hook) {
    {
        HookScope hs(hook, DPG_KERNEL_ROWGATHER, s);
        const int64_t need = std::max((static_cast<int64_t>(L.P.V) + 31) / 32, (static_cast<int64_t>(L.P.nitems) + 7) / 8);
        const int grid = static_cast<int>(std::min<int64_t>(need, static_cast<int64_t>(sm_count) * rows_blocks(VEC)));
        rows_kernel<VEC, LQ, MODE><<<grid, kBlock, 0, s>>>(L);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || L.P.nhubs == 0 || !L.out) return e;
    HookScope hs(hook, DPG_KERNEL_FIXUP, s);
    auto fixup = L.nrhs <= 32   ? spmm_fixup_kernel<1>
                 : L.nrhs <= 64 ? (tree ? spmm_fixup_kernel<2, true> : spmm_fixup_kernel<2>)
                                : (tree ? spmm_fixup_kernel<4, true> : spmm_fixup_kernel<4>);
    fixup<<<sm_count * 4, kBlock, 0, s>>>(L.P.hubs, L.P.nhubs, L.partial, L.nrhs, L.out);
    return cudaGetLastError();
}

template <int VEC, int MODE>
cudaError_t pick_rows(const RowsLaunch& L, bool tree, cudaStream_t s, int sm_count, LaunchHook* hook) {
    const int Q = L.nrhs / VEC;
    if (Q <= 1) return run_rows<VEC, 1, MODE>(L, tree, s, sm_count, hook);
    if (Q <= 2) return run_rows<VEC, 2, MODE>(L, tree, s, sm_count, hook);
    if (Q <= 4) return run_rows<VEC, 4, MODE>(L, tree, s, sm_count, hook);
    if (Q <= 8) return run_rows<VEC, 8, MODE>(L, tree, s, sm_count, hook);
    if (Q <= 16) return run_rows<VEC, 16, MODE>(L, tree, s, sm_count, hook);
    return run_rows<VEC, 32, MODE>(L, tree, s, sm_count, hook);
}

template <int MODE>
cudaError_t pick_vec(const RowsLaunch& L, bool tree, cudaStream_t s, int sm_count, LaunchHook* hook) {
    if (L.P.V <= 0) return cudaSuccess;
    bool vec4 = L.nrhs % 4 == 0;
    for (const void* p : {static_cast<const void*>(L.in), static_cast<const void*>(L.X), static_cast<const void*>(L.out),
                          static_cast<const void*>(L.partial)})
        vec4 = vec4 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
    return vec4 ? pick_rows<4, MODE>(L, tree, s, sm_count, hook) : pick_rows<1, MODE>(L, tree, s, sm_count, hook);
}

}  // namespace

cudaError_t launch_spmm_group(const SpmmPlanDev& P, const int32_t* col, const float* val, const float* X, int nrhs,
                              float* Y, float* partial, cudaStream_t s, int sm_count, LaunchHook* hook) {
    const RowsLaunch L = {P, col, nullptr, val, X, nullptr, nrhs, Y, partial, nullptr};
    return pick_vec<kForward>(L, false, s, sm_count, hook);
}

cudaError_t launch_spmv_bwd_group(const SpmmPlanDev& TP, bool tree, const int32_t* tcol, const int32_t* tarc, const float* val,
                                  const float* X, const float* G, int nrhs, float* dX, float* partial, float* dA,
                                  cudaStream_t s, int sm_count, LaunchHook* hook) {
    const RowsLaunch L = {TP, tcol, tarc, val, G, X, nrhs, dX, partial, dA};
    return tarc ? pick_vec<kBwdArcs>(L, tree, s, sm_count, hook) : pick_vec<kBwdSlots>(L, tree, s, sm_count, hook);
}

size_t perm_scratch_bytes(int64_t E) {
    const size_t nblk = static_cast<size_t>((E + kPermBlock - 1) / kPermBlock);
    return 4 * (static_cast<size_t>(E) + nblk * nblk);
}

cudaError_t launch_build_perm(const int32_t* tarc, int64_t E, void* scratch, const ArcPerm& P, cudaStream_t s,
                              int sm_count) {
    const int nblk = static_cast<int>((E + kPermBlock - 1) / kPermBlock);
    int32_t* slot_of = static_cast<int32_t*>(scratch);
    int32_t* counts = slot_of + E;
    // The limit of the largest permutation, whatever this one takes (two threads may set it at once).
    constexpr int kMaxBlocks = static_cast<int>((kPermMaxArcs + kPermBlock - 1) / kPermBlock);
    cudaError_t e = cudaFuncSetAttribute(perm_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * kMaxBlocks);
    if (e != cudaSuccess) return e;
    invert_kernel<<<sm_count * 8, kBlock, 0, s>>>(tarc, E, slot_of);
    const int grid = std::min(nblk, sm_count * 2);
    perm_count_kernel<<<grid, kPermThreads, 4 * nblk, s>>>(slot_of, E, nblk, counts);
    perm_scan_kernel<<<grid, kPermThreads, 0, s>>>(nblk, counts);
    perm_place_kernel<<<grid, kPermThreads, 8 * nblk, s>>>(slot_of, E, nblk, counts, P.mid, P.arc_in, P.slot_in);
    return cudaGetLastError();
}

cudaError_t launch_permute(const ArcPerm& P, int64_t E, bool to_slots, const float* in, float* tmp, float* out,
                           cudaStream_t s, int sm_count, LaunchHook* hook) {
    constexpr int smem = kPermBlock * sizeof(float);
    const int nblk = static_cast<int>((E + kPermBlock - 1) / kPermBlock);
    const int grid = std::min(nblk, 2 * sm_count);
    cudaError_t e = cudaFuncSetAttribute(perm_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(perm_in_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    {
        HookScope hs(hook, DPG_KERNEL_INIT, s);
        if (to_slots) perm_out_kernel<<<grid, kPermThreads, smem, s>>>(in, E, nblk, P.arc_in, P.mid, tmp);
        else perm_out_kernel<<<grid, kPermThreads, smem, s>>>(in, E, nblk, P.slot_in, nullptr, tmp);
    }
    HookScope hs(hook, DPG_KERNEL_INIT, s);
    if (to_slots) perm_in_kernel<<<grid, kPermThreads, smem, s>>>(tmp, E, nblk, P.slot_in, nullptr, out);
    else perm_in_kernel<<<grid, kPermThreads, smem, s>>>(tmp, E, nblk, P.arc_in, P.mid, out);
    return cudaGetLastError();
}

cudaError_t launch_gather_values(const float* v, const int32_t* idx, int64_t n, float* out, cudaStream_t s,
                                 int sm_count) {
    if (n > 0) gather_values_kernel<<<sm_count * 8, kBlock, 0, s>>>(v, idx, n, out);
    return cudaGetLastError();
}

}  // namespace dpg
