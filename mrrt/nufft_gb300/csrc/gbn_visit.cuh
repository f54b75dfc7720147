// Adjoint table interpolation (samples -> grid) over plan-time visit lists.
// Replaces the reference's scatters (serial per coil on the CPU,
// mrrt/nufft/_extensions/c/nufft_table.template.c:144-531, 924-1206; global
// atomicAdd per tap on the GPU, mrrt/nufft/cuda/jinja/table_*_adjoint.jinja)
// with an "owner computes" decomposition and register accumulation.
//
// The grid is cut into register blocks of 16 cells (4 x 4, one z-plane; 16 in
// 1-D); a warp holds a block's 16 complex sums in every lane, lane = (visit
// slot, coil), LS coils per chunk.  Which samples touch a block, and with
// which coefficients, is fixed by the coordinates, so the plan stores it:
//
//   * visits: for each work item (a tile's entries, or a part of them) and
//     each block of the tile, in entry order, the samples whose window
//     touches the block, padded to a multiple of four;
//   * each visit's coefficients clipped to the block and zero-padded: B0
//     values of axis 0, then (2-D, 3-D) B1 values w of the other axes, w = c1
//     or c1 c2.  Rows the window misses hold -0, so that a row is skipped by
//     a test of its bits and not by its value.
//
// At run time nothing is searched or sorted: a warp streams visits.  (The
// kernel this replaces staged a tile's entries chunk by chunk with two
// barriers each, and every warp balloted which of them touched its block:
// 515 warp instructions a sample at the 2-D 32-coil workload, 101 of them
// the multiply-adds.)  Measured, spread alone, before -> now, plus the pass
// that lays the values out: 128^3 kooshball, 8 coils 4892 -> 1860 + 109 us;
// 64-frame series, 8 coils 949 -> 398 + 64; 2-D 256^2, 32 coils 143 -> 92 +
// 24; 128^2, one coil 29 -> 18; 192^2 double, 4 coils 345 -> 216.  Bound by
// instruction issue (3-D: 80% of the issue slots, 45% of them multiply-adds).
//
// The sample values come coil-minor, [sample][coil], with conj(sample phase)
// applied (values_kernel: one transposition per call), so that one visit's
// coils are one segment: read straight from [coil][sample], a 32-coil visit
// touches 32 sectors.  Small batches (use_values in gbn_plan.cu) read the
// values in place and apply the phase on reading.
//
// Order of summation: entry order per slot, slots combined in a fixed
// pattern, warps sharing a block in warp order, parts of split tiles by
// reduce_kernel: the same in every run.
#pragma once

#include <cuda_runtime.h>

#include "gbn_device.cuh"
#include "gbn_internal.h"

namespace gbn {

template <int NDIM>
struct VisitBlock {
    static constexpr int B0 = SpreadBlock<NDIM>::B0, B1 = SpreadBlock<NDIM>::B1, B2 = SpreadBlock<NDIM>::B2;
    static constexpr int NB = B0 * B1;               // cells (B2 = 1: w carries axis 2)
    static constexpr int NC = B0 + (NDIM > 1 ? B1 : 0);   // coefficients per visit
    static_assert(B2 == 1 && NB == 16, "register blocks of 16 cells, one z-plane");
};

// Origin of register block `blk` within its tile (blocks of axis 0 fastest).
template <int NDIM, typename R>
__host__ __device__ __forceinline__ void block_origin(const Geom<R>& g, int blk, int& b0, int& b1, int& b2) {
    typedef VisitBlock<NDIM> VB;
    const int n0 = g.T[0] / VB::B0, n1 = NDIM > 1 ? g.T[1] / VB::B1 : 1;
    b0 = (blk % n0) * VB::B0;
    b1 = NDIM > 1 ? ((blk / n0) % n1) * VB::B1 : 0;
    b2 = NDIM > 2 ? blk / (n0 * n1) : 0;
}
// The same from the table the launcher put in the parameters (no division).
template <typename R>
__device__ __forceinline__ void block_origin_of(const VisitParams<R>& p, int blk, int& b0, int& b1, int& b2) {
    const short4 o = p.borg[blk];
    b0 = o.x;
    b1 = o.y;
    b2 = o.z;
}

__device__ __forceinline__ bool is_neg_zero(float v) { return __float_as_uint(v) == 0x80000000u; }
__device__ __forceinline__ bool is_neg_zero(double v) {
    return (unsigned long long)__double_as_longlong(v) == 0x8000000000000000ull;
}

// N values, 16 bytes at a time (16-byte aligned records, global or shared).
template <int N>
__device__ __forceinline__ void load_run(const float* src, float (&o)[N]) {
    static_assert(N % 4 == 0, "whole vectors");
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(src + i);
        o[i] = v.x;
        o[i + 1] = v.y;
        o[i + 2] = v.z;
        o[i + 3] = v.w;
    }
}
template <int N>
__device__ __forceinline__ void load_run(const double* src, double (&o)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const double2 v = *reinterpret_cast<const double2*>(src + i);
        o[i] = v.x;
        o[i + 1] = v.y;
    }
}

template <int N>
__device__ __forceinline__ void store_run(float* dst, const float (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = v[i];
    }
}
template <int N>
__device__ __forceinline__ void store_run(double* dst, const double (&v)[N]) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 2) *reinterpret_cast<double2*>(dst + i) = make_double2(v[i], v[i + 1]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = v[i];
    }
}

// Asynchronous copy of BYTES (8 or 16) source bytes, of none and zeros if not
// valid.
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(n) : "memory");
}

// Coefficient k of a visit to the block at (b0, b1, b2) of a window starting
// at ls; coef(d, j) gives tap j of axis d.
template <typename R, int NDIM, bool CX, typename F>
__device__ __forceinline__ typename Cx<R>::T clipped_coef(const Geom<R>& g, short4 ls, int b0, int b1, int b2, int k,
                                                          F coef) {
    typedef VisitBlock<NDIM> VB;
    typedef typename Cx<R>::T C;
    // one path for both axes: lanes of a warp hold coefficients of either
    const int d = NDIM > 1 && k >= VB::B0 ? 1 : 0;
    const int j = d ? b1 + (k - VB::B0) - ls.y : b0 + k - ls.x;
    if (j < 0 || j >= g.J[d]) return cmake<R>(d ? (R)-0.0 : (R)0, (R)0);
    C w = coef(d, j);
    if (NDIM > 2 && d) {
        const C c2 = coef(2, b2 - ls.z);
        w = CX ? cmul_fixed(w, c2) : cmake<R>(mul_rn(w.x, c2.x), (R)0);
    }
    return w;
}

// What the coefficients of a visit to list entry e (-1: padding) are computed
// from.
template <typename R, int NDIM>
struct VisitEntry {
    short4 ls;
    R t[3];
    int idx;   // sample index, -1: padding
    __device__ __forceinline__ void load(const SampleList<R>& s, int e, unsigned* check) {
        idx = -1;
        ls = make_short4(0, 0, 0, 0);
#pragma unroll
        for (int d = 0; d < NDIM; ++d) t[d] = (R)0;
        if (e < 0 || !GBN_INB(check, e < s.len, CHK_LIST)) return;
        idx = s.idx[e];
        ls = s.ls[e];
#pragma unroll
        for (int d = 0; d < NDIM; ++d) t[d] = s.t[d][e];
    }
};

// The part-th of P equal runs of the coefficients of a visit to the block at (b0, b1, b2),
// from the tables, into out: the numbers a plan that keeps them has stored.
// P lanes share a visit, and a lane reads the entry once for all of its
// coefficients.  Spread alone: 256 x 256, 4 and 8 coils 47 and 76 us, 60 x 72 x
// 45, 3 and 8 coils 380 and 462.  (A lane to each coefficient, which read the
// entry and, of w = c1 c2, the table for c2 anew, and where the samples are read
// in place each coil lane for itself: 222 and 226, 1331 and 1467.)
template <typename R, int NDIM, bool CX, int P>
__device__ __forceinline__ void table_visit(const Geom<R>& g, const VisitEntry<R, NDIM>& v, int b0, int b1, int b2,
                                            int part, R* out) {
    typedef VisitBlock<NDIM> VB;
    typedef typename Cx<R>::T C;
    int first[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < NDIM; ++d) first[d] = first_tap(v.t[d], g.J[d]);
    auto tap = [&](int d, R td, int k) {
        R cr, ci = (R)0;
        table_coef<R, CX>(g, d, td, k, cr, ci);
        return cmake<R>(cr, CX ? -ci : (R)0);
    };
    C c2 = cmake<R>((R)0, (R)0);
    if (NDIM > 2) c2 = tap(2, v.t[2], first[2] + b2 - v.ls.z);
    constexpr int NK = VB::NC / P, W = CX ? 2 : 1;
    R co[NK * W];
#pragma unroll
    for (int i = 0; i < NK; ++i) {
        const int k = part * NK + i, d = NDIM > 1 && k >= VB::B0 ? 1 : 0;
        const int j = d ? b1 + (k - VB::B0) - v.ls.y : b0 + k - v.ls.x;
        const bool in = v.idx >= 0 && j >= 0 && j < g.J[d];
        C c = cmake<R>(d ? (R)-0.0 : (R)0, (R)0);
        // a tap past the window is computed too (its table index is clamped) and
        // dropped: behind a branch each, the taps' loads waited for one another
        if (NDIM > 1 || in) {
            C w = tap(d, d ? v.t[1] : v.t[0], (d ? first[1] : first[0]) + j);
            if (NDIM > 2 && d) w = CX ? cmul_fixed(w, c2) : cmake<R>(mul_rn(w.x, c2.x), (R)0);
            if (in) c = w;
        }
        co[i * W] = c.x;
        if (CX) co[i * W + W - 1] = c.y;
    }
    store_run(out + part * NK * W, co);
}

// The same from the sample's coefficients, J_0 + J_1 + J_2 at rec (imaginary
// parts behind them).
template <typename R, int NDIM, bool CX, int P>
__device__ __forceinline__ void record_visit(const Geom<R>& g, bool on, short4 ls, const R* rec, int b0, int b1, int b2,
                                             int part, R* out) {
    typedef VisitBlock<NDIM> VB;
    typedef typename Cx<R>::T C;
    const int at1 = g.J[0], at2 = g.J[0] + (NDIM > 1 ? g.J[1] : 0), jsum = at2 + (NDIM > 2 ? g.J[2] : 0);
    auto tap = [&](int j) { return cmake<R>(rec[j], CX ? -rec[jsum + j] : (R)0); };
    C c2 = cmake<R>((R)0, (R)0);
    if (NDIM > 2 && on) c2 = tap(at2 + b2 - ls.z);
    constexpr int NK = VB::NC / P, W = CX ? 2 : 1;
    R co[NK * W];
#pragma unroll
    for (int i = 0; i < NK; ++i) {
        const int k = part * NK + i;
        C c = cmake<R>(NDIM > 1 && k >= VB::B0 ? (R)-0.0 : (R)0, (R)0);
        if (on)
            c = clipped_coef<R, NDIM, CX>(g, ls, b0, b1, b2, k,
                                          [&](int d, int j) { return d == 2 ? c2 : tap((d ? at1 : 0) + j); });
        co[i * W] = c.x;
        if (CX) co[i * W + W - 1] = c.y;
    }
    store_run(out + part * NK * W, co);
}

// ---- plan time ---------------------------------------------------------------

// The tile's block at (b0, b1, b2) holds cells of the grid (tile edges may
// reach past it); the others are never written and have no visits.
template <int NDIM, typename R>
__device__ __forceinline__ bool block_in_grid(const Geom<R>& g, int tile, int b0, int b1, int b2) {
    int org[3] = {0, 0, 0};
    tile_origin<NDIM>(tile, g.nt, g.T, org);
    return org[0] + b0 < g.K[0] && (NDIM < 2 || org[1] + b1 < g.K[1]) && (NDIM < 3 || org[2] + b2 < g.K[2]);
}

// A window starting at s (tile coordinates) touches the block at (b0, b1, b2).
template <int NDIM, typename R>
__device__ __forceinline__ bool visits_block(const Geom<R>& g, short4 s, int b0, int b1, int b2) {
    typedef VisitBlock<NDIM> VB;
    bool hit = s.x < b0 + VB::B0 && s.x + g.J[0] > b0;
    if (NDIM > 1) hit = hit && s.y < b1 + VB::B1 && s.y + g.J[1] > b1;
    if (NDIM > 2) hit = hit && s.z < b2 + VB::B2 && s.z + g.J[2] > b2;
    return hit;
}

// Entries e with base + 32 u + lane = e of a count-long run that touch the
// block, as one mask per u; the starts' loads are independent of each other.
constexpr int VISIT_UNROLL = 4;

template <typename R, int NDIM>
__device__ __forceinline__ void block_hits(const VisitBuildParams<R>& p, int first, int count, int base, int lane, int b0,
                                           int b1, int b2, unsigned (&mask)[VISIT_UNROLL]) {
    short4 s[VISIT_UNROLL];
#pragma unroll
    for (int u = 0; u < VISIT_UNROLL; ++u)
        if (base + 32 * u + lane < count) s[u] = p.s.ls[(int64_t)first + base + 32 * u + lane];
#pragma unroll
    for (int u = 0; u < VISIT_UNROLL; ++u)
        mask[u] = __ballot_sync(0xffffffffu,
                                base + 32 * u + lane < count && visits_block<NDIM>(p.g, s[u], b0, b1, b2));
}

// Visits per (item, block), rounded up to whole groups of four: one CTA per
// item, one warp per block.
template <typename R, int NDIM>
__global__ void __launch_bounds__(256) visit_count_kernel(const VisitBuildParams<R> p) {
    const int item = blockIdx.x, blk = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 it = p.items[item];
    const bool ok = GBN_INB(p.g.check, it.z >= 0 && it.w >= 0 && it.z + (int64_t)it.w <= p.s.len, CHK_LIST);
    int b0, b1, b2;
    block_origin<NDIM>(p.g, blk, b0, b1, b2);
    int n = 0;
    const int count = ok && block_in_grid<NDIM>(p.g, it.y, b0, b1, b2) ? it.w : 0;
    for (int base = 0; base < count; base += 32 * VISIT_UNROLL) {
        unsigned mask[VISIT_UNROLL];
        block_hits<R, NDIM>(p, it.z, count, base, lane, b0, b1, b2, mask);
#pragma unroll
        for (int u = 0; u < VISIT_UNROLL; ++u) n += __popc(mask[u]);
    }
    if (lane == 0) p.count[(int64_t)item * p.nblk + blk] = (n + 3) & ~3;
}

// The visits as list positions; padding is -1.
template <typename R, int NDIM>
__global__ void __launch_bounds__(256) visit_fill_kernel(const VisitBuildParams<R> p) {
    const int item = blockIdx.x, blk = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 it = p.items[item];
    if (!GBN_INB(p.g.check, it.z >= 0 && it.w >= 0 && it.z + (int64_t)it.w <= p.s.len, CHK_LIST)) return;
    int b0, b1, b2;
    block_origin<NDIM>(p.g, blk, b0, b1, b2);
    int64_t at = p.start[(int64_t)item * p.nblk + blk];
    // device binning sizes the lists by a bound on the sum of the counts
    const int64_t stop = p.start[(int64_t)item * p.nblk + blk + 1], end = min(stop, (int64_t)p.nvisits);
    if (!GBN_INB(p.g.check, stop <= p.nvisits, CHK_LIST)) return;
    const int count = block_in_grid<NDIM>(p.g, it.y, b0, b1, b2) ? it.w : 0;
    for (int base = 0; base < count; base += 32 * VISIT_UNROLL) {
        unsigned mask[VISIT_UNROLL];
        block_hits<R, NDIM>(p, it.z, count, base, lane, b0, b1, b2, mask);
#pragma unroll
        for (int u = 0; u < VISIT_UNROLL; ++u) {
            const int64_t pos = at + __popc(mask[u] & ((1u << lane) - 1u));
            if ((mask[u] >> lane & 1u) && pos < end) p.vidx[pos] = it.z + base + 32 * u + lane;
            at += __popc(mask[u]);
        }
    }
    if (at + lane < end) p.vidx[at + lane] = -1;
}

// Their coefficients, a thread to each, copied from the gather's record of
// the sample (the same numbers: a sample's coefficients do not depend on the
// block), and the sample indices in place of the positions.  A visit waits
// for a chain of loads (position, sample, record's place, record), so an
// item's visits, up to some thousands, go to the threads of up to
// VISIT_SLICES CTAs, VISIT_UNROLL at a time; most items need one.  128^3
// kooshball, 10^8 visits: 3.4 ms for 7.5 GB; computed from the tables, two
// scattered reads a coefficient, 9.9.  (With the warp of each block making
// them where it found the visits, a lane to a visit, the 330,000 visits of a
// 512 x 512 grid took 90 us in place of 34.)
constexpr int VISIT_SLICES = 4;

template <typename R, int NDIM, bool CX>
__global__ void __launch_bounds__(256) visit_coef_kernel(const VisitBuildParams<R> p) {
    typedef VisitBlock<NDIM> VB;
    typedef typename Cx<R>::T C;
    constexpr int NC = VB::NC, PER = 256 / NC;   // visits a CTA takes at a time
    const Geom<R>& g = p.g;
    const int item = blockIdx.x;
    const long long* st = p.start + (int64_t)item * p.nblk;
    const int64_t first = st[0];
    const int n = (int)(min(st[p.nblk], (long long)p.nvisits) - first);
    if ((int)blockIdx.y * PER * VISIT_UNROLL >= n) return;   // the whole CTA
    // origins and first visits of the item's blocks
    __shared__ int4 block[8];
    if ((int)threadIdx.x < p.nblk) {
        int4 o;
        block_origin<NDIM>(g, threadIdx.x, o.x, o.y, o.z);
        o.w = (int)(st[threadIdx.x] - first);
        block[threadIdx.x] = o;
    }
    __syncthreads();
    const int64_t fo = p.foff[p.items[item].x];
    const int k = threadIdx.x % NC;
    int* vidx = p.vidx + first;
    R* vco = p.vco + first * NC * (CX ? 2 : 1);
    for (int v0 = blockIdx.y * PER * VISIT_UNROLL; v0 < n; v0 += PER * VISIT_UNROLL * VISIT_SLICES) {
        int e[VISIT_UNROLL], idx[VISIT_UNROLL], blk[VISIT_UNROLL];
        C c[VISIT_UNROLL];
#pragma unroll
        for (int u = 0; u < VISIT_UNROLL; ++u) {
            const int v = v0 + u * PER + threadIdx.x / NC;
            e[u] = v < n ? vidx[v] : -1;
            blk[u] = 0;
        }
        for (int b = 1; b < p.nblk; ++b) {
            const int at = block[b].w;
#pragma unroll
            for (int u = 0; u < VISIT_UNROLL; ++u) blk[u] += at <= v0 + u * PER + (int)threadIdx.x / NC;
        }
#pragma unroll
        for (int u = 0; u < VISIT_UNROLL; ++u) {
            if (!GBN_INB(g.check, e[u] < p.s.len, CHK_LIST)) e[u] = -1;
            idx[u] = e[u] < 0 ? -1 : p.s.idx[e[u]];
            if (!GBN_INB(g.check, fo + idx[u] < p.samples, CHK_LIST)) e[u] = idx[u] = -1;
            c[u] = cmake<R>(!CX && k >= VB::B0 ? (R)-0.0 : (R)0, (R)0);
            if (e[u] >= 0) {
                const int4 o = block[blk[u]];
                int at = p.place[fo + idx[u]];
                if (!GBN_INB(g.check, at >= 0 && at < p.samples, CHK_LIST)) at = 0;
                const R* r = p.rec + (int64_t)at * p.stride;
                c[u] = clipped_coef<R, NDIM, CX>(g, p.s.ls[e[u]], o.x, o.y, o.z, k, [&](int d, int j) {
                    j += (d > 0 ? g.J[0] : 0) + (d > 1 ? g.J[1] : 0);
                    return cmake<R>(r[j], CX ? -r[p.jsum + j] : (R)0);
                });
            }
        }
        __syncwarp();   // a visit's lanes, one warp, have read its position
#pragma unroll
        for (int u = 0; u < VISIT_UNROLL; ++u) {
            const int v = v0 + u * PER + threadIdx.x / NC;
            if (v >= n) continue;
            if (k == 0) vidx[v] = idx[u];
            if (CX) reinterpret_cast<C*>(vco)[(int64_t)v * NC + k] = c[u];
            else vco[(int64_t)v * NC + k] = c[u].x;
        }
    }
}

// ---- per call ----------------------------------------------------------------

// Samples [frame][coil][m] -> values [frame][m][coil] times conj(phase).  A
// CTA transposes 64 consecutive samples of 32 coils at a time through shared
// memory: 512-byte reads along m, contiguous writes along (m, coil).
constexpr int VAL_SAMPLES = 64, VAL_COILS = 32;

template <typename R>
__global__ void __launch_bounds__(256) values_kernel(const ValuesParams<R> p) {
    typedef typename Cx<R>::T C;
    __shared__ C sm[VAL_SAMPLES * (VAL_COILS + 1)];
    const int64_t m0 = (int64_t)blockIdx.x * VAL_SAMPLES;
    const int ns = (int)min((int64_t)VAL_SAMPLES, p.M - m0);
    const int c0 = blockIdx.y * VAL_COILS;
    const int nc = min(VAL_COILS, p.n - c0);
    const int sl = threadIdx.x % VAL_SAMPLES, cg = threadIdx.x / VAL_SAMPLES;
    constexpr int NG = 256 / VAL_SAMPLES;
    if (sl < ns) {
        const int64_t m = m0 + sl;
        int f = 0, hi = p.F;   // foff[f] <= m < foff[hi]
        while (hi - f > 1) {
            const int mid = (f + hi) >> 1;
            if (p.foff[mid] <= m) f = mid;
            else hi = mid;
        }
        const int64_t fo = p.foff[f], Mf = p.foff[f + 1] - fo;
        const C* src = p.y + fo * p.coils + (m - fo) + (int64_t)(p.first + c0) * Mf;
        const C ph = p.ph ? p.ph[m] : cmake<R>((R)1, (R)0);
        for (int c = cg; c < nc; c += 4 * NG) {
            C v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = cmake<R>((R)0, (R)0);
                if (c + u * NG < nc &&
                    GBN_INB(p.check, fo * p.coils + (m - fo) + (int64_t)(p.first + c0 + c + u * NG) * Mf < p.M * p.coils,
                            CHK_SAMPLE_READ))
                    v[u] = src[(int64_t)(c + u * NG) * Mf];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c + u * NG < nc) sm[sl * (VAL_COILS + 1) + c + u * NG] = p.ph ? cmulc(v[u], ph) : v[u];
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < ns * nc; q += 256) {
        const int s = q / nc, c = q - s * nc;
        const int64_t o = (m0 + s) * p.row + c0 + c;
        if (GBN_INB(p.check, o < p.out_elems, CHK_SCRATCH)) p.out[o] = sm[s * (VAL_COILS + 1) + c];
    }
}

// ---- accumulation ------------------------------------------------------------

// Add row k1 of one visit: value v, coefficients co.
template <typename R, int NDIM, bool CX>
__device__ __forceinline__ void add_row(typename Cx<R>::T (&acc)[VisitBlock<NDIM>::NB], typename Cx<R>::T v,
                                        const R (&co)[VisitBlock<NDIM>::NC * (CX ? 2 : 1)], int k1) {
    typedef typename Cx<R>::T C;
    constexpr int B0 = VisitBlock<NDIM>::B0;
    C tv = v;
    if constexpr (CX) {
        if (NDIM > 1) tv = cmul_fixed(cmake<R>(co[2 * (B0 + k1)], co[2 * (B0 + k1) + 1]), v);
#pragma unroll
        for (int k0 = 0; k0 < B0; ++k0) {
            const C t = cmul_fixed(cmake<R>(co[2 * k0], co[2 * k0 + 1]), tv);
            acc[k1 * B0 + k0].x = add_rn(acc[k1 * B0 + k0].x, t.x);
            acc[k1 * B0 + k0].y = add_rn(acc[k1 * B0 + k0].y, t.y);
        }
    } else {
        if (NDIM > 1) {
            tv.x = mul_rn(co[B0 + k1], v.x);
            tv.y = mul_rn(co[B0 + k1], v.y);
        }
        // scalar multiply-adds: as many per cycle as packed ones, and no
        // register moves to form the (c, c) pairs
#pragma unroll
        for (int k0 = 0; k0 < B0; ++k0) {
            acc[k1 * B0 + k0].x = fma_rn(co[k0], tv.x, acc[k1 * B0 + k0].x);
            acc[k1 * B0 + k0].y = fma_rn(co[k0], tv.y, acc[k1 * B0 + k0].y);
        }
    }
}

// Sum a block over the warp's slots by a halving exchange: each slot ends up
// with KEEP consecutive cells, from cell q0 on, in acc[0..KEEP).
template <typename R, int LS, int NB>
__device__ __forceinline__ int combine_slots(typename Cx<R>::T (&acc)[NB], int slot) {
    typedef typename Cx<R>::T C;
    constexpr int SW = 32 / LS;
    int q0 = 0;
#pragma unroll
    for (int s = 0; (1 << s) < SW; ++s) {
        const int half = NB >> (s + 1);
        if (half >= 1) {
            const bool up = (slot >> s) & 1;
#pragma unroll
            for (int i = 0; i < (half >= 1 ? half : 1); ++i) {
                const C lo = acc[i], hi = acc[i + half];
                const C send = up ? lo : hi, keep = up ? hi : lo;
                acc[i].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, LS << s);
                acc[i].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, LS << s);
            }
            if (up) q0 += half;
        } else {   // 32 slots, 16 cells: the last stage adds the pair
            acc[0].x += __shfl_xor_sync(0xffffffffu, acc[0].x, LS << s);
            acc[0].y += __shfl_xor_sync(0xffffffffu, acc[0].y, LS << s);
        }
    }
    return q0;
}

// Where the blocks of an item go, for one lane: the grid (with
// conj(phase_before)), or the scratch slot of a split tile.  Formed once per
// item, so that a block costs an offset from the launcher's tables and a few
// adds, and its phases come in one load ahead of use; with origins, bounds
// and 64-bit strides worked out for each block, and the phases loaded where
// they were used, the adjoint took 182 us instead of 168 at 256 x 256 with
// 32 coils, 5000 instead of 4860 (with the forward) at 128^3 with 8, and 511
// instead of 449 (with the forward) at 60 x 72 x 45 with 3.
template <typename R, int NDIM, int LS>
struct BlockSink {
    typedef typename Cx<R>::T C;
    typedef VisitBlock<NDIM> VB;
    static constexpr int B0 = VB::B0, NB = VB::NB, SW = 32 / LS;
    static constexpr int KEEP = SW >= NB ? 1 : NB / SW;   // cells of a block this lane writes
    C* dst;               // cell 0 of the tile, this lane's coil
    int64_t pcell;        // cell 0 of the tile in the phase table
    int tile;
    bool direct, phased, whole, on;

    __device__ __forceinline__ BlockSink(const VisitParams<R>& p, int4 it, int slot_id, int chunk, int lane) {
        const Geom<R>& g = p.g;
        const int coil = lane % LS, c = chunk * LS + coil;
        int org[3] = {0, 0, 0};
        tile = it.y;
        tile_origin<NDIM>(tile, g.nt, g.T, org);
        direct = slot_id < 0;
        phased = direct && p.apply_pb;
        whole = org[0] + g.T[0] <= g.K[0] && (NDIM < 2 || org[1] + g.T[1] <= g.K[1]) &&
                (NDIM < 3 || org[2] + g.T[2] <= g.K[2]);
        on = c < p.coils && !(SW > NB && ((lane / LS) >> 4));
        if (direct) {
            dst = p.grid + it.x * g.gsf + c * g.gsp + org[0] * g.gs0 + (NDIM > 1 ? org[1] * g.gs1 : 0) +
                  (NDIM > 2 ? org[2] * g.gs2 : 0);
        } else {
            dst = p.scratch + ((int64_t)slot_id * p.chunks + chunk) * p.tile_cells * LS + coil;
        }
        pcell = org[0] + (int64_t)g.K[0] * ((NDIM > 1 ? org[1] : 0) + (int64_t)g.K[1] * (NDIM > 2 ? org[2] : 0));
    }

    // Extents of block blk that lie in the grid.
    __device__ __forceinline__ void extent(const VisitParams<R>& p, int blk, int& n0, int& n1) const {
        n0 = B0;
        n1 = NB / B0;
        if (!whole) {
            int b0, b1, b2, org[3] = {0, 0, 0};
            tile_origin<NDIM>(tile, p.g.nt, p.g.T, org);
            block_origin_of(p, blk, b0, b1, b2);
            n0 = min(B0, p.g.K[0] - org[0] - b0);
            if (NDIM > 1) n1 = min(n1, p.g.K[1] - org[1] - b1);
            if (NDIM > 2 && org[2] + b2 >= p.g.K[2]) n0 = 0;
        }
    }

    // phase_before of the block's cell `lane` (lanes below NB), to be loaded
    // ahead of the block's sums
    __device__ __forceinline__ C phase(const VisitParams<R>& p, int blk, int lane) const {
        C ph = cmake<R>((R)1, (R)0);
        if (phased && lane < NB) {
            int n0, n1;
            extent(p, blk, n0, n1);
            if (lane % B0 < n0 && lane / B0 < n1) {
                if (p.g.ptab) {
                    ph = p.g.ptab[pcell + p.bcell[blk] + lane % B0 + (NDIM > 1 ? p.g.K[0] * (lane / B0) : 0)];
                } else {
                    int b0, b1, b2, org[3] = {0, 0, 0};
                    tile_origin<NDIM>(tile, p.g.nt, p.g.T, org);
                    block_origin_of(p, blk, b0, b1, b2);
                    const int k[3] = {org[0] + b0 + lane % B0, org[1] + b1 + lane / B0, org[2] + b2};
                    ph = phase_before(p.g, k);
                }
            }
        }
        return ph;
    }

    // Write a combined block; `zero`: no visits (zeros need no phase).
    __device__ __forceinline__ void flush(const VisitParams<R>& p, C (&acc)[NB], int q0, int blk, C ph,
                                          bool zero) const {
        if (phased && !zero) {
#pragma unroll
            for (int i = 0; i < KEEP; ++i) {
                C w;
                w.x = __shfl_sync(0xffffffffu, ph.x, q0 + i);
                w.y = __shfl_sync(0xffffffffu, ph.y, q0 + i);
                acc[i] = cmulc(acc[i], w);
            }
        }
        if (!on) return;
        int n0, n1;
        extent(p, blk, n0, n1);
        const Geom<R>& g = p.g;
        // strides fit 32 bits (the launcher has looked), three rows need not (unsigned:
        // signed products of 64 bits cost the series' adjoint 2 us of 680)
        const int s0 = direct ? (int)g.gs0 : LS, s1 = direct ? (int)g.gs1 : g.T[0] * LS;
        const bool vec = sizeof(R) == 4 && direct && g.gs0 == 1 && ((g.K[0] | g.gsf | g.gsp | g.gs1 | g.gs2) & 1) == 0;
        C* d = dst + (direct ? p.boff[blk] : p.bscr[blk] * LS);
        constexpr int STEP = KEEP >= 2 ? 2 : 1;
#pragma unroll
        for (int i = 0; i < KEEP; i += STEP) {
            const int q = q0 + i, k0 = q % B0, k1 = q / B0;
            const bool in0 = k0 < n0 && k1 < n1, in1 = STEP == 2 && k0 + 1 < n0 && k1 < n1;
            C* o = d + ((unsigned long long)(unsigned)k1 * (unsigned)s1 + (unsigned)(k0 * s0));
#ifdef GBN_CHECKED
            C* last = o + (in1 ? s0 : 0);
            if ((in0 || in1) && !(direct ? GBN_INB(p.g.check, o >= p.grid && last < p.grid + p.g.grid_elems, CHK_GRID_WRITE)
                                         : GBN_INB(p.g.check, o >= p.scratch && last < p.scratch + p.scratch_elems,
                                                   CHK_SCRATCH)))
                continue;
#endif
            if (in0 && in1 && vec) {
                store_pair(o, acc[i], acc[i + STEP - 1]);
            } else {
                if (in0) o[0] = acc[i];
                if (in1) o[s0] = acc[i + STEP - 1];
            }
        }
    }
};

// ---- values read in place: one (item, block) per warp ---------------------------
//
// Up to four coil lanes (two of a single-precision volume).  U visits per slot
// are in flight at a time.
constexpr int VISIT_THREADS = 128;   // four (item, block) units per CTA

template <typename R, int NDIM, bool CX, int LS, bool TAB>
__global__ void __launch_bounds__(VISIT_THREADS, 5) spread_unit_kernel(const VisitParams<R> p) {
    typedef typename Cx<R>::T C;
    typedef VisitBlock<NDIM> VB;
    constexpr int NB = VB::NB, NC = VB::NC * (CX ? 2 : 1), B1 = NDIM > 1 ? VB::B1 : 1;
    constexpr int SW = 32 / LS;
    // visits in flight per slot, fewer the more registers one takes
    constexpr int WORDS = (int)sizeof(R) / 4 * (CX ? 2 : 1) * (NDIM == 1 ? 2 : 1);
    constexpr int U = WORDS > 2 || SW > 8 ? 1 : (WORDS > 1 || SW > 4 ? 2 : 4);
    // coefficients and sample indices of 32 visits, a lane to each, where they
    // are computed on the way
    __shared__ __align__(16) R tab_co[TAB ? VISIT_THREADS : 1][NC];
    __shared__ int tab_id[TAB ? VISIT_THREADS : 1];
    const int own = TAB ? threadIdx.x & ~31 : 0;
    const Geom<R>& g = p.g;
    const int lane = threadIdx.x & 31;
    const unsigned unit = blockIdx.x * (VISIT_THREADS / 32) + (threadIdx.x >> 5);
    if (unit >= (unsigned)(p.nitems * p.nblk)) return;   // whole warps only; no barrier below
    const int item = (int)(unit / (unsigned)p.nblk), blk = (int)(unit - (unsigned)item * p.nblk);
    const int chunk = blockIdx.y;
    const int4 it = p.items[item];
    const int2 part = p.parts[item];
    const int f = it.x;
    const int64_t st = p.start[unit];
    const int n = (int)(min(p.start[unit + 1], (long long)p.nvisits) - st);
    if (!GBN_INB(g.check, st >= 0 && n >= 0, CHK_LIST)) return;
    const int c0 = chunk * LS;
    const int nc = min(LS, p.coils - c0);
    const int slot = lane / LS, coil = lane % LS;

    const int64_t fo = p.foff[f];
    const int Mf = (int)(p.foff[f + 1] - fo);
    // samples of this lane's coil (lanes past the last coil repeat it)
    const C* yb = p.y + fo * p.coils + (int64_t)(c0 + min(coil, nc - 1)) * Mf;
    const C* ph = p.ph ? p.ph + fo : nullptr;
    int b0, b1, b2;
    block_origin_of(p, blk, b0, b1, b2);

    C acc[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) acc[q] = cmake<R>((R)0, (R)0);
    const int* vidx = p.vidx + st;
    VisitEntry<R, NDIM> entry;   // of the 32 visits to come, and the entries after them
    int next = -1;
    if (TAB) {
        entry.load(p.s, lane < n ? vidx[lane] : -1, g.check);
        next = 32 + lane < n ? vidx[32 + lane] : -1;
    }
    for (int i0 = 0; i0 < n; i0 += U * SW) {
        if (TAB && (i0 & 31) == 0) {
            __syncwarp();   // the visits before these have been read
            tab_id[threadIdx.x] = entry.idx;
            table_visit<R, NDIM, CX, 1>(g, entry, b0, b1, b2, 0, tab_co[threadIdx.x]);
            entry.load(p.s, next, g.check);
            next = i0 + 64 + lane < n ? vidx[i0 + 64 + lane] : -1;
            __syncwarp();
        }
        // past the last visit, and for padding, the value is zero by selection:
        // an infinity or NaN must not meet a zero coefficient
        int id[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * SW + slot;
            id[u] = TAB ? tab_id[own + (i & 31)] : i < n ? vidx[i] : -1;
        }
        C v[U], w[U];
        R co[U][NC];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (TAB) load_run(tab_co[own + ((i0 + u * SW + slot) & 31)], co[u]);
            else load_run(p.vco + (st + min(i0 + u * SW + slot, n - 1)) * NC, co[u]);
            const int m = max(id[u], 0);
            v[u] = cmake<R>((R)0, (R)0);
            if (GBN_INB(g.check, m < Mf, CHK_SAMPLE_READ)) v[u] = yb[m];
            if (ph) w[u] = ph[m];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (ph) v[u] = cmulc(v[u], w[u]);
            if (id[u] < 0) v[u] = cmake<R>((R)0, (R)0);
        }
#pragma unroll
        for (int k1 = 0; k1 < B1; ++k1)
#pragma unroll
            for (int u = 0; u < U; ++u) add_row<R, NDIM, CX>(acc, v[u], co[u], k1);
    }
    const BlockSink<R, NDIM, LS> sink(p, it, part.x, chunk, lane);
    C phase = cmake<R>((R)1, (R)0);
    if (n > 0) phase = sink.phase(p, blk, lane);
    const int q0 = combine_slots<R, LS, NB>(acc, slot);
    sink.flush(p, acc, q0, blk, phase, n == 0);
}

// ---- coil-minor values: a warp streams visits through a shared-memory ring ------
//
// The visits of an item's blocks lie one after another, so a warp runs over
// a whole range of them, blocks in turn, with the copies (values and
// coefficients, cp.async into the warp's own ring, no barrier) running
// one stage ahead across block boundaries: with loads into registers
// the same sums waited 58% of the time on the four visits a lane could hold.
//
// An item of many entries is shared by the eight warps of a CTA, each taking
// an equal run of the visits wherever the block boundaries fall (a block cut
// by a run's end is completed by the warp that began it, from shared
// memory, in warp order); lighter items go one to a warp, eight to a CTA.
// Sharing costs a barrier and, where blocks are cut, an exchange; not sharing
// leaves the last warps alone with the heavy tiles of the k-space centre.
//
// Calls that may not allocate and whose values do not fit the fixed array have
// them copied from [coil][sample] value by value (INPLACE): the same sums in the
// same order.  Adjacent lanes copy a coil's values for adjacent visits, whose
// samples tend to be adjacent, into rows of one value more, which keeps the lanes
// on different banks.
constexpr int STREAM_WARPS = 8;

// Where a visit costs a warp more (double precision, coefficients computed on
// the way), the lighter items end a launch on their one warp each; they go to a
// CTA too, a block to each warp.  No block is cut, so no sum changes.  (With
// eight slots a stage's end decides which slot a visit goes to: not there.)
// 256 x 256, 8 coils: double 658 us in place of 804; computed coefficients 80
// in place of 96, complex 115 and 147, double 738 and 878.
template <typename R, int LS, bool TAB>
constexpr bool share_whole() { return (TAB || sizeof(R) == 8) && LS >= 8; }

template <typename R, int NDIM, bool CX, int LS, bool INPLACE>
struct StreamLayout {
    typedef typename Cx<R>::T C;
    static constexpr int NC = VisitBlock<NDIM>::NC * (CX ? 2 : 1);
    static constexpr int VROW = LS * (int)sizeof(C);            // bytes of one visit's values
    // values of a stage: at 32 coils two copies of eight visits each, 9 us of
    // 168 faster than one (256 x 256, 32 coils)
    static constexpr int VBYTES = LS == 32 && sizeof(C) == 8 ? 4096 : VROW < 64 ? 32 * VROW : 2048;
    static constexpr int RV = VBYTES / VROW;                    // visits per stage
    static constexpr int CBYTES = RV * NC * (int)sizeof(R);     // coefficients of a stage
    static constexpr int COFF = VBYTES + (INPLACE ? RV * (int)sizeof(C) : 0);   // where they begin
    static constexpr int STAGE = COFF + CBYTES;
    static constexpr int LSP = LS + (INPLACE ? 1 : 0);          // values from a visit's to the next's
    static constexpr int HEAD = 16 * LS * (int)sizeof(C);       // one combined block
    static constexpr int SINK = 32;                             // the item's BlockSink
    static constexpr int WARP = 2 * STAGE + HEAD + SINK;
    static constexpr int SMEM = STREAM_WARPS * WARP;
    static_assert(sizeof(BlockSink<R, 2, LS>) <= SINK, "sink");
    static_assert(RV % 4 == 0 && RV <= 32 && VROW <= 512 && COFF % 16 == 0 && STAGE % 16 == 0, "stage layout");
};

// CTAs per SM: what the registers of a block's sums leave (two in double
// precision: 1048 us at 192 x 192, 16 coils, against 1074 with one), and those
// of coefficients computed on the way (two: 60 x 72 x 45, complex, 3 coils 607
// us against 849 where 163 registers left one).
template <typename R, int NDIM, bool CX, int LS, bool TAB, bool INPLACE>
__global__ void __launch_bounds__(32 * STREAM_WARPS,
                                  TAB && sizeof(R) == 4 ? 2 : CX ? 1 : sizeof(R) == 8 || LS == 32 ? 2 : 3)
spread_stream_kernel(const VisitParams<R> p) {
    typedef typename Cx<R>::T C;
    typedef VisitBlock<NDIM> VB;
    typedef StreamLayout<R, NDIM, CX, LS, INPLACE> SL;
    constexpr int NB = VB::NB, NC = SL::NC, B1 = NDIM > 1 ? VB::B1 : 1, SW = 32 / LS, RV = SL::RV;
    constexpr int KEEP = NB / SW, GROUP = SW > 4 ? SW : 4;
    constexpr bool WHOLE = share_whole<R, LS, TAB>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geom<R>& g = p.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nshared = WHOLE ? p.nwhole : p.nshared;
    const bool shared_item = (int)blockIdx.x < nshared;
    const int item = shared_item ? (int)blockIdx.x : nshared + ((int)blockIdx.x - nshared) * STREAM_WARPS + warp;
    if (item >= p.nitems) return;   // only in a CTA of unshared items: no barrier there
    const int chunk = blockIdx.y;
    const int4 it = p.items[item];
    const int part = p.parts[item].x;
    const int f = it.x;
    const int c0 = chunk * LS;
    const int slot = lane / LS, coil = lane % LS;
    unsigned char* ring = smem_raw + warp * SL::WARP;
    C* head = reinterpret_cast<C*>(ring + 2 * SL::STAGE);

    // visit offsets of the item's blocks: lane b holds block b's, from base on
    const int nblk = p.nblk;
    const long long* st = p.start + (int64_t)item * nblk;
    const long long base = st[0];
    const int rel = (int)(min(st[min(lane, nblk)], (long long)p.nvisits) - base);
    const int N = __shfl_sync(0xffffffffu, rel, nblk);
    // this warp's run [lo, hi): the whole item, or its share; whole blocks
    // where the largest is close enough to an equal share
    int lo = 0, hi = N, per = N;
    bool whole = false;
    if (shared_item) {
        per = ((N + STREAM_WARPS - 1) / STREAM_WARPS + 3) & ~3;
        const int nxt = __shfl_down_sync(0xffffffffu, rel, 1);
        const int most = __reduce_max_sync(0xffffffffu, (unsigned)(lane < nblk ? nxt - rel : 0));
        whole = most <= per + 8 * SW || (WHOLE && item >= p.nshared);
        lo = whole ? __shfl_sync(0xffffffffu, rel, min(warp, nblk)) : min(N, warp * per);
        hi = whole ? __shfl_sync(0xffffffffu, rel, min(warp + 1, nblk)) : min(N, (warp + 1) * per);
    }
    const int64_t fo = p.foff[f];
    const int Mf = (int)(p.foff[f + 1] - fo);
    // the item's sink waits in shared memory: held in registers through the
    // sums it spilled at 80, and formed anew for each block it cost 2-3%
    BlockSink<R, NDIM, LS>* kept = reinterpret_cast<BlockSink<R, NDIM, LS>*>(ring + SL::WARP - SL::SINK);
    {
        const BlockSink<R, NDIM, LS> first(p, it, part, chunk, lane);
        if (lane == 0) *kept = first;   // coil 0 of the chunk
        __syncwarp();
    }
    auto sink = [&]() {   // for this lane's coil
        BlockSink<R, NDIM, LS> k = *kept;
        k.dst += coil * (k.direct ? g.gsp : (int64_t)1);
        k.on = c0 + coil < p.coils;
        return k;
    };

    // ---- copies: stage k holds visits lo + k RV ... of the run -----------------
    // A lane copies 16 bytes at a fixed place of every (512 / VROW)-th visit.
    const int row_bytes = p.row * (int)sizeof(C);
    const int off = lane * 16 % SL::VROW;
    const bool lane_ok = c0 * (int)sizeof(C) + off < row_bytes;
    const char* vsrc = reinterpret_cast<const char*>(p.vals + fo * p.row + c0) + (lane_ok ? off : 0);
    const C* ysrc = p.y + fo * p.coils + (int64_t)c0 * Mf;
    const int visit = TAB ? lane % RV : lane;
    const int* isrc = p.vidx + base + lo + visit;
    const char* csrc = reinterpret_cast<const char*>(p.vco + (base + lo) * NC) + lane * 16;
    int to_load = hi - lo - visit;                       // this lane's visits not yet read
    int to_copy = (hi - lo) * NC * (int)sizeof(R) - lane * 16;   // coefficient bytes not yet copied
    int issued = 0;                                      // visits whose copies were issued
    // index of the visit this lane reads for the stage to come (-1: none); with
    // TAB its list entry, visit lane % RV of the stage, and what it holds
    VisitEntry<R, NDIM> entry;
    int origin = 0;   // lane b: block b's, for the visits' blocks
    if (TAB) {
        const short4 o = p.borg[min(lane, 7)];
        origin = o.x | o.y << 8 | o.z << 16;
    }
    auto load_id = [&]() {
        const int id = (TAB || lane < RV) && to_load > 0 ? *isrc : -1;
        isrc += RV;
        to_load -= RV;
        return id;
    };
    auto issue = [&](unsigned char* sb, int id) {
        if (issued < hi - lo) {
            if (TAB) id = entry.idx;
            // no copy of a sample out of range, nor past the last coil: zeros
            if (!GBN_INB(g.check, id < Mf, CHK_SAMPLE_READ)) id = -1;
            if (INPLACE) {
#pragma unroll
                for (int j = 0; j < LS * RV / 32; ++j) {
                    const int c = j * (32 / RV) + lane / RV, m = __shfl_sync(0xffffffffu, id, lane % RV);
                    const bool ok = m >= 0 && c0 + c < p.coils;
                    cp_async_zfill<sizeof(C)>(sb + (lane % RV * SL::LSP + c) * sizeof(C),
                                              ysrc + (ok ? (int64_t)c * Mf + m : 0), ok);
                }
            } else {
#pragma unroll
                for (int j = 0; j < SL::VBYTES / 512; ++j) {
                    const int m = __shfl_sync(0xffffffffu, id, lane * 16 / SL::VROW + j * (512 / SL::VROW));
                    const bool ok = m >= 0 && lane_ok;
                    cp_async_zfill<16>(sb + lane * 16 + j * 512, vsrc + (ok ? (int64_t)m * row_bytes : 0), ok);
                }
            }
            if (TAB) {
                const int vi = lane % RV;
                int blk = 0;   // the block the visit belongs to: the last that begins at or before it
#pragma unroll
                for (int h = 4; h > 0; h /= 2)
                    if (__shfl_sync(0xffffffffu, rel, blk + h) <= lo + issued + vi) blk += h;
                const int o = __shfl_sync(0xffffffffu, origin, blk);
                const int b0 = o & 0xff, b1 = o >> 8 & 0xff, b2 = o >> 16;
                R* co = reinterpret_cast<R*>(sb + SL::COFF) + vi * NC;
                if (!GBN_INB(g.check, entry.idx < Mf, CHK_SAMPLE_READ)) entry.idx = -1;
                if (sizeof(R) == 8 && !INPLACE && p.rec) {
                    const R* rec = reinterpret_cast<const R*>(p.vals + (fo + max(entry.idx, 0)) * p.row) + p.rec;
                    record_visit<R, NDIM, CX, 32 / RV>(g, entry.idx >= 0, entry.ls, rec, b0, b1, b2, lane / RV, co);
                } else {
                    table_visit<R, NDIM, CX, 32 / RV>(g, entry, b0, b1, b2, lane / RV, co);
                }
            } else {
#pragma unroll
                for (int q = 0; q < SL::CBYTES; q += 512) {
                    if (SL::CBYTES - q < 512 && lane * 16 >= SL::CBYTES - q) break;
                    const bool ok = q < to_copy;
                    cp_async_zfill<16>(sb + SL::COFF + lane * 16 + q,
                                       ok ? csrc + q : reinterpret_cast<const char*>(p.vco), ok);
                }
                csrc += SL::CBYTES;
                to_copy -= SL::CBYTES;
            }
            issued += RV;
        }
        cp_async_commit();
    };
    int id = load_id();
    {
        const int nx = load_id();
        if (TAB) entry.load(p.s, id, g.check);
        issue(ring, id);
        id = nx;
        if (TAB) {
            entry.load(p.s, id, g.check);
            id = load_id();
        }
    }

    C acc[NB], phase = cmake<R>((R)1, (R)0);
    const unsigned char* sb = ring + SL::STAGE;   // the stage being read (none yet)
    const C* vp = nullptr;
    const R* cp = nullptr;
    int left = 0, pos = lo;                       // visits left in it; next visit of the run
    int pending = -1, pending_end = 0, q_pending = 0;
    for (int b = 0; b < nblk; ++b) {
        const int rb = __shfl_sync(0xffffffffu, rel, b), re = __shfl_sync(0xffffffffu, rel, b + 1);
        const bool owned = shared_item ? (whole ? b == warp
                                                : lo <= rb && (rb < hi || warp == STREAM_WARPS - 1))
                                       : true;
        const int end = min(re, hi);
        if (!owned && max(rb, lo) >= end) continue;
#pragma unroll
        for (int q = 0; q < NB; ++q) acc[q] = cmake<R>((R)0, (R)0);
        while (pos < end) {
            if (left == 0) {
                // the next stage has landed, for every lane; the buffer just
                // read takes the one after it
                cp_async_wait_all();
                __syncwarp();
                const int nx = load_id();
                unsigned char* done = const_cast<unsigned char*>(sb);
                sb = sb == ring ? ring + SL::STAGE : ring;
                issue(done, id);
                if (TAB) entry.load(p.s, id, g.check);
                id = nx;
                left = RV;
                vp = reinterpret_cast<const C*>(sb) + slot * SL::LSP + coil;
                cp = reinterpret_cast<const R*>(sb + SL::COFF) + slot * NC;
            }
            const int n = min(end - pos, left);
            pos += n;
            left -= n;
            // groups of four visits (blocks begin and end on whole groups)
#pragma unroll 1
            for (int q = n; q > 0; q -= GROUP) {
                unsigned rows = 0xffffu;
                if (NDIM > 1 && !CX && SW == 1) {
                    // one visit at a time: bit 4 u + k1 is set where visit u's
                    // window covers row k1; the warp skips the others
                    rows = __ballot_sync(0xffffffffu,
                                         lane < 16 && !is_neg_zero(cp[(lane >> 2) * NC + NC - B1 + (lane & 3)]));
                }
#pragma unroll
                for (int u = 0; u < GROUP / SW; ++u) {
                    if (GROUP > 4 && slot >= q) break;   // four visits left for eight slots
                    const C v = vp[u * SW * SL::LSP];
                    R co[NC];
                    load_run(cp + u * SW * NC, co);
#pragma unroll
                    for (int k1 = 0; k1 < B1; ++k1)
                        if (!(NDIM > 1 && !CX && SW == 1) || (rows >> (4 * u + k1) & 1))
                            add_row<R, NDIM, CX>(acc, v, co, k1);
                }
                const int step = GROUP > 4 ? min(q, GROUP) : GROUP;
                vp += step * SL::LSP;
                cp += step * NC;
            }
        }
        // loaded ahead of the exchange between slots, which hides part of it
        if (owned && re > rb) phase = sink().phase(p, b, lane);
        const int q0 = combine_slots<R, LS, NB>(acc, slot);
        if (!owned) {   // begun by an earlier warp: hand it over
#pragma unroll
            for (int i = 0; i < KEEP; ++i) head[(q0 + i) * LS + coil] = acc[i];
        } else if (re > hi) {   // continued by later warps (the last block of the run)
            pending = b;
            pending_end = re;
            q_pending = q0;
        } else {
            sink().flush(p, acc, q0, b, phase, re == rb);
        }
    }
    if (!shared_item || whole) return;   // the same for the whole CTA
    __syncthreads();
    if (pending >= 0) {
        for (int w = warp + 1; w < STREAM_WARPS && w * per < pending_end; ++w) {
            const C* h = reinterpret_cast<const C*>(smem_raw + w * SL::WARP + 2 * SL::STAGE);
#pragma unroll
            for (int i = 0; i < KEEP; ++i) acc[i] = cadd(acc[i], h[(q_pending + i) * LS + coil]);
        }
        sink().flush(p, acc, q_pending, pending, phase, false);
    }
}

// ---- launchers -----------------------------------------------------------------

template <typename R>
cudaError_t launch_visit_count(const VisitBuildParams<R>& p, cudaStream_t s) {
    if (p.nitems == 0) return cudaSuccess;
    const int threads = 32 * p.nblk;
    switch (p.g.ndim) {
        case 1: visit_count_kernel<R, 1><<<p.nitems, threads, 0, s>>>(p); break;
        case 2: visit_count_kernel<R, 2><<<p.nitems, threads, 0, s>>>(p); break;
        case 3: visit_count_kernel<R, 3><<<p.nitems, threads, 0, s>>>(p); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename R, int NDIM>
cudaError_t visit_fill_any(const VisitBuildParams<R>& p, cudaStream_t s) {
    visit_fill_kernel<R, NDIM><<<p.nitems, 32 * p.nblk, 0, s>>>(p);
    if (p.vco) {
        const dim3 grid((unsigned)p.nitems, VISIT_SLICES);
        if (p.cx) visit_coef_kernel<R, NDIM, true><<<grid, 256, 0, s>>>(p);
        else visit_coef_kernel<R, NDIM, false><<<grid, 256, 0, s>>>(p);
    }
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_visit_fill(const VisitBuildParams<R>& p, cudaStream_t s) {
    if (p.nitems == 0) return cudaSuccess;
    if (p.nblk < 1 || p.nblk > 8) return cudaErrorInvalidValue;
    switch (p.g.ndim) {
        case 1: return visit_fill_any<R, 1>(p, s);
        case 2: return visit_fill_any<R, 2>(p, s);
        case 3: return visit_fill_any<R, 3>(p, s);
    }
    return cudaErrorInvalidValue;
}

template <typename R>
cudaError_t launch_values(const ValuesParams<R>& p, cudaStream_t s) {
    if (p.M == 0 || p.n == 0) return cudaSuccess;
    const int64_t bx = (p.M + VAL_SAMPLES - 1) / VAL_SAMPLES;
    const int64_t by = (p.n + VAL_COILS - 1) / VAL_COILS;
    if (bx > INT32_MAX || by > 65535) return cudaErrorInvalidValue;
    values_kernel<R><<<dim3((unsigned)bx, (unsigned)by), 256, 0, s>>>(p);
    return cudaGetLastError();
}

template <typename R, int NDIM, bool CX, int LS, bool TAB, bool INPLACE>
cudaError_t stream_launch(const VisitParams<R>& p0, cudaStream_t s) {
    VisitParams<R> p = p0;
    if (INPLACE && p.ph && p.s.len > 0) return cudaErrorInvalidValue;   // the values hold the phase
    // An item goes to one warp up to 32 entries per slot (a longer one would
    // outlast the rest of a small launch), more where each warp of three CTAs on
    // each of 152 SMs would have many times that to do anyway.  (Where fewer CTAs
    // fit, complex kernels above all, this shares items sooner than that asks.)
    const int64_t load = p.s.len * p.chunks / (3 * STREAM_WARPS * 152) / 8;
    int q = LS >= 32 ? 0 : LS >= 16 ? 1 : 2;
    while (q < SPREAD_HEAVY_LEVELS - 1 && (SPREAD_SHARE_ENTRIES << q) < load) ++q;
    p.nshared = p.nheavy[q];
    p.nwhole = max(p.nshared, p.nheavy[0]);
    const int shared = share_whole<R, LS, TAB>() ? p.nwhole : p.nshared;
    const int64_t ctas = shared + ((int64_t)p.nitems - shared + STREAM_WARPS - 1) / STREAM_WARPS;
    if (ctas > INT32_MAX || p.nchunk > 65535) return cudaErrorInvalidValue;
    constexpr size_t smem = StreamLayout<R, NDIM, CX, LS, INPLACE>::SMEM;
    const auto kernel = spread_stream_kernel<R, NDIM, CX, LS, TAB, INPLACE>;
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    kernel<<<dim3((unsigned)ctas, (unsigned)p.nchunk), 32 * STREAM_WARPS, smem, s>>>(p);
    return cudaGetLastError();
}

template <typename R, int NDIM, bool CX, int LS, bool TAB>
cudaError_t unit_launch(const VisitParams<R>& p, cudaStream_t s) {
    const int64_t units = (int64_t)p.nitems * p.nblk;
    const int64_t ctas = (units + VISIT_THREADS / 32 - 1) / (VISIT_THREADS / 32);
    if (units > INT32_MAX || p.nchunk > 65535) return cudaErrorInvalidValue;
    spread_unit_kernel<R, NDIM, CX, LS, TAB><<<dim3((unsigned)ctas, (unsigned)p.nchunk), VISIT_THREADS, 0, s>>>(p);
    return cudaGetLastError();
}

template <typename R, int NDIM, bool CX, int LS, bool TAB>
cudaError_t stream_values(const VisitParams<R>& p, cudaStream_t s) {
    if (p.vals) return stream_launch<R, NDIM, CX, LS, TAB, false>(p, s);
    if constexpr (LS <= inplace_lanes<R>()) return stream_launch<R, NDIM, CX, LS, TAB, true>(p, s);
    return cudaErrorInvalidValue;
}

template <typename R, int NDIM, bool CX, bool TAB>
cudaError_t visit_lanes(const VisitParams<R>& p, cudaStream_t s) {
    switch (p.LS) {
        case 1: return unit_launch<R, NDIM, CX, 1, TAB>(p, s);
        case 2: return unit_launch<R, NDIM, CX, 2, TAB>(p, s);
        case 4:
            if constexpr (sizeof(R) == 4 && NDIM == 3) return stream_values<R, NDIM, CX, 4, TAB>(p, s);
            else return unit_launch<R, NDIM, CX, 4, TAB>(p, s);
        case 8: return stream_values<R, NDIM, CX, 8, TAB>(p, s);
        // volumes have eight lanes at most
        case 16: if constexpr (NDIM < 3) return stream_values<R, NDIM, CX, 16, TAB>(p, s); break;
        case 32: if constexpr (NDIM < 3) return stream_values<R, NDIM, CX, 32, TAB>(p, s); break;
    }
    return cudaErrorInvalidValue;
}

template <typename R, int NDIM, bool CX>
cudaError_t visit_any(const VisitParams<R>& p, cudaStream_t s) {
    return p.vco ? visit_lanes<R, NDIM, CX, false>(p, s) : visit_lanes<R, NDIM, CX, true>(p, s);
}

template <typename R>
cudaError_t launch_spread_visits(const VisitParams<R>& p0, cudaStream_t s) {
    if (p0.nitems == 0 || p0.coils == 0) return cudaSuccess;
    VisitParams<R> p = p0;
    if (p.nblk < 1 || p.nblk > 8 || p.g.gs0 > INT32_MAX / 4 || p.g.gs1 > INT32_MAX) return cudaErrorInvalidValue;
    for (int b = 0; b < p.nblk; ++b) {
        int b0, b1, b2;
        if (p.g.ndim == 1) block_origin<1>(p.g, b, b0, b1, b2);
        else if (p.g.ndim == 2) block_origin<2>(p.g, b, b0, b1, b2);
        else block_origin<3>(p.g, b, b0, b1, b2);
        p.borg[b] = make_short4((short)b0, (short)b1, (short)b2, 0);
        p.boff[b] = b0 * p.g.gs0 + (p.g.ndim > 1 ? b1 * p.g.gs1 : 0) + (p.g.ndim > 2 ? b2 * p.g.gs2 : 0);
        p.bscr[b] = b0 + p.g.T[0] * (b1 + p.g.T[1] * b2);
        p.bcell[b] = b0 + (int64_t)p.g.K[0] * (b1 + (int64_t)p.g.K[1] * b2);
    }
    const bool cx = p.g.hi[0] != nullptr;
    switch (p.g.ndim * 2 + (cx ? 1 : 0)) {
        case 2: return visit_any<R, 1, false>(p, s);
        case 3: return visit_any<R, 1, true>(p, s);
        case 4: return visit_any<R, 2, false>(p, s);
        case 5: return visit_any<R, 2, true>(p, s);
        case 6: return visit_any<R, 3, false>(p, s);
        case 7: return visit_any<R, 3, true>(p, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace gbn
