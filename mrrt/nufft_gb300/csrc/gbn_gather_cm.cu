// Forward table interpolation (grid -> samples) on a coil-minor grid, for
// real single-precision kernels of width 4, 5 or 6.
//
// The same decomposition as gbn_gather.cu (a CTA stages a tile with its halo
// for LS coils in shared memory and interpolates the tile's samples there).
// What bounded it was not the interpolation: of 666 warp instructions a sample
// at a 3-D kooshball some 560 staged cells (divisions for the cell's place, a
// sincos for its phase, an 8-byte load, multiply and store per coil), and a
// further 22 shuffles a sample handed its prepared coefficients round.  Here
//   * the grid comes coil-minor and with phase_before applied (the last FFT
//     pass does both), so staging is 16-byte asynchronous copies of whole
//     row segments (8-byte ones for an odd coil count);
//   * a sample's window place, output index, phase and coefficients are one
//     plan-time record; each warp streams the records of its share of the
//     samples through a small ring in shared memory and reads them as
//     broadcasts;
//   * a lane takes two adjacent coils, so the tap loop reads 16 bytes a lane.
//     With 8 coils or fewer, groups of lanes share a sample and take every
//     2nd, 4th or 8th of its taps along axis 0, so that the eight lanes of a
//     wavefront read adjacent cells, each bank once (one lane per sample, as
//     one coil had it, reads 32 unrelated cells).
// What it spends: the taps are 72 wavefronts of shared memory a sample at J 6,
// 2-D, 32 coils (108 in 3-D with 8) of 91 (148) in all.  The data pipe is busy
// 69% (80%) of the time, at 23% of the warps: the rest is waiting, staging and
// interpolation being in sequence within a CTA.
#include <cuda_runtime.h>

#include <algorithm>

#include "gbn_device.cuh"
#include "gbn_internal.h"

namespace gbn {

namespace {

constexpr int CM_THREADS = 256, CM_WARPS = CM_THREADS / 32;

template <int NDIM, int J, int LS>
struct CmLayout {
    static constexpr int VC = LS > 1 ? 2 : 1;               // coils per lane
    static constexpr int LL = LS / VC;                      // lanes over the coils
    static constexpr int TSP = LS >= 16 ? 1 : 8 / LL;       // lane groups over a sample's taps
    static constexpr int GL = LL * TSP;                     // lanes per sample
    static constexpr int SW = 32 / GL;                      // samples a warp serves at a time
    static constexpr int NC = (NDIM * J + 3) / 4 * 4;       // coefficients of a record
    static constexpr int REC = 16 + 4 * NC;                 // bytes of a record
    static constexpr int B = 2 * SW;                        // records per ring stage
    static constexpr int RING = 2 * B * REC;                // bytes per warp
};

// The values of VC adjacent coils.
template <int VC> struct Vals;
template <> struct Vals<2> { typedef float4 T; };
template <> struct Vals<1> { typedef float2 T; };
__device__ __forceinline__ void add_scaled(float4& a, float c, const float4& v) {
    a.x = fmaf(c, v.x, a.x);
    a.y = fmaf(c, v.y, a.y);
    a.z = fmaf(c, v.z, a.z);
    a.w = fmaf(c, v.w, a.w);
}
__device__ __forceinline__ void add_scaled(float2& a, float c, const float2& v) {
    a.x = fmaf(c, v.x, a.x);
    a.y = fmaf(c, v.y, a.y);
}
__device__ __forceinline__ float2 first_coil(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 first_coil(const float2& v) { return v; }
__device__ __forceinline__ float2 second_coil(const float4& v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 second_coil(const float2& v) { return v; }
__device__ __forceinline__ float2 add_lane(float2 v, float2 send, int lanes) {
    v.x += __shfl_xor_sync(0xffffffffu, send.x, lanes);
    v.y += __shfl_xor_sync(0xffffffffu, send.y, lanes);
    return v;
}

// Bytes of a staged tile, rounded up: the record rings behind it are read 16
// bytes at a time (an odd number of one-coil cells is not a multiple of 16).
__host__ __device__ constexpr size_t tile_bytes(size_t cells, int LS) {
    return (cells * LS * sizeof(float2) + 15) & ~(size_t)15;
}

template <int CB>
__device__ __forceinline__ void cp_async_fill(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? CB : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(CB), "r"(n) : "memory");
}

template <int N>
__device__ __forceinline__ void load_coefs(const float* src, float (&o)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(src + i);
        o[i] = v.x;
        o[i + 1] = v.y;
        o[i + 2] = v.z;
        o[i + 3] = v.w;
    }
}

// The records of n list entries from e0 on, computed instead of copied (plans
// that keep no coefficients): the plan-time values, by the same arithmetic.
template <int NDIM, int J, int NC>
__device__ __noinline__ void compute_records(const GatherParams<float>& p, int64_t e0, int n, float* out) {
    const Geom<float>& g = p.g;
    constexpr int STRIDE = 4 + NC;
    for (int q = threadIdx.x & 31; q < n * (NDIM * J + 1); q += 32) {
        const int r = q / (NDIM * J + 1), k = q - r * (NDIM * J + 1);
        const int64_t e = e0 + r;
        float* rec = out + r * STRIDE;
        if (k == 0) {
            int cell = 0, mul = 1;
            for (int a = 0; a < NDIM; ++a) {
                cell += mul * (wrapk(first_tap(p.s.t[a][e], J), g.K[a]) % g.T[a]);
                mul *= g.T[a] + J - 1;
            }
            const float2 ph = p.s.ph ? p.s.ph[e] : make_float2(1.f, 0.f);
            *reinterpret_cast<int4*>(rec) = make_int4(cell, p.s.idx[e], __float_as_int(ph.x), __float_as_int(ph.y));
        } else {
            const int d = (k - 1) / J, j = (k - 1) - d * J;
            const float t = p.s.t[d][e];
            float ci;
            table_coef<float, false>(g, d, t, first_tap(t, J) + j, rec[3 + k], ci);
        }
    }
}

template <int NDIM, int J, int LS, int CB, bool TAB>
__global__ void __launch_bounds__(CM_THREADS) gather_cm_kernel(const GatherParams<float> p) {
    typedef CmLayout<NDIM, J, LS> L;
    typedef typename Vals<L::VC>::T V;
    constexpr int VC = L::VC, LL = L::LL, TSP = L::TSP, GL = L::GL, SW = L::SW, B = L::B, REC = L::REC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geom<float>& g = p.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int4 it = p.items[blockIdx.x];
    const int f = it.x, start = it.z, count = it.w;
    if (!GBN_INB(g.check, start >= 0 && count >= 0 && start + (int64_t)count <= p.s.len, CHK_LIST)) return;
    const int c0 = blockIdx.y * LS;
    const int nc = min(LS, p.coils - c0);
    int org[3] = {0, 0, 0};
    tile_origin<NDIM>(it.y, g.nt, g.T, org);
    int Rd[3];
    const int cells = region_dims(g, NDIM, Rd);
    V* S = reinterpret_cast<V*>(smem_raw);                                 // [cell][LL], VC coils each
    unsigned char* ring = smem_raw + tile_bytes(cells, LS) + warp * L::RING;

    // ---- this warp's samples: an equal share, whole rounds of SW ----------------
    const int share = ((count + CM_WARPS - 1) / CM_WARPS + SW - 1) / SW * SW;
    const int s0 = min(count, warp * share), ns = min(count, (warp + 1) * share) - s0;
    const char* rsrc = reinterpret_cast<const char*>(p.s.rec) + (int64_t)(start + s0) * REC;
    auto issue_records = [&](int k) {   // stage k: records k B ... of the share
        if constexpr (TAB) {
            compute_records<NDIM, J, L::NC>(p, (int64_t)start + s0 + k * B, min(B, ns - k * B),
                                            reinterpret_cast<float*>(ring + (k & 1) * (B * REC)));
        } else {
            const int left = (ns - k * B) * REC;
            for (int q = lane * 16; q < B * REC; q += 512)
                if (q < left) cp_async<16>(ring + (k & 1) * (B * REC) + q, rsrc + (int64_t)k * (B * REC) + q);
        }
    };
    issue_records(0);

    // ---- stage the tile and its halo --------------------------------------------
    // Grid offsets of the region's rows first, one per thread; then a thread
    // keeps its place along axis 0 (and so its wrapped offset) and copies it
    // from every row: a load of the row's offset, an add and a copy each.
    const int nrows = Rd[1] * (NDIM > 2 ? Rd[2] : 1);
    int64_t* rowoff = reinterpret_cast<int64_t*>(smem_raw + tile_bytes(cells, LS) + CM_WARPS * L::RING);
    for (int r = threadIdx.x; r < nrows; r += CM_THREADS) {
        const int y = NDIM > 2 ? r % Rd[1] : r, z = NDIM > 2 ? r / Rd[1] : 0;
        int64_t o = f * g.gsf + c0 + (int64_t)wrapk(org[1] + y, g.K[1]) * g.gs1;
        if (NDIM > 2) o += (int64_t)wrapk(org[2] + z, g.K[2]) * g.gs2;
        rowoff[r] = o;
    }
    __syncthreads();
    {
        constexpr int PC = LS * 8 / CB;   // copies per cell
        const int Q = Rd[0] * PC;
        int tpr = 32;                     // threads per row
        while (tpr < Q && tpr < CM_THREADS) tpr *= 2;
        const int part = threadIdx.x % PC * CB;
        const bool part_ok = part < nc * 8;
        for (int q = threadIdx.x % tpr; q < Q; q += tpr) {
            const int64_t x = (int64_t)wrapk(org[0] + q / PC, g.K[0]) * g.gs0;
            const char* src = reinterpret_cast<const char*>(p.grid + x) + part;
            unsigned char* dst = smem_raw + q * CB;
#pragma unroll 4
            for (int r = threadIdx.x / tpr; r < nrows; r += CM_THREADS / tpr) {
                const bool ok = part_ok && GBN_INB(g.check, rowoff[r] + x + (part + CB) / 8 <= g.grid_elems,
                                                   CHK_GRID_READ);
                cp_async_fill<CB>(dst + (size_t)r * Rd[0] * (LS * 8),
                                  ok ? src + rowoff[r] * 8 : reinterpret_cast<const char*>(p.grid), ok);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();

    // ---- interpolate --------------------------------------------------------------
    const int grp = lane / GL, th = TSP > 1 ? (lane / LL) % TSP : 0, cl = lane % LL;   // coils VC cl, ...
    const int64_t fo = p.foff[f];
    const int Mf = (int)(p.foff[f + 1] - fo);
    if (!GBN_INB(g.check, (fo + Mf) * p.coils <= g.sample_elems, CHK_SAMPLE_WRITE)) return;
    // the coil this lane writes: where lane groups share a sample, the first
    // VC of them one each; else both
    const int wc = TSP > 1 ? VC * cl + th % VC : VC * cl;
    const bool writes = TSP == 1 || th < VC;
    float2* yb = p.y + fo * p.coils + (int64_t)(c0 + wc) * Mf;
    const int rs = Rd[0] * LL, ps = Rd[0] * Rd[1] * LL;
    constexpr int JH = (J + TSP - 1) / TSP;   // taps of a lane along axis 0
    int pidx = -1;                            // held output (per coil), waiting for its neighbour
    float2 pa = make_float2(0.f, 0.f), pb = make_float2(0.f, 0.f);
    auto put = [&](float2* y, int idx, float2 held, float2 v, bool pair) {
        if (pair)
            store_pair(y + idx - 1, held, v);
        else
            y[idx] = v;
    };
    for (int k = 0; k * B < ns; ++k) {
        if (k > 0) {
            cp_async_wait_all();
            __syncwarp();
        }
        if ((k + 1) * B < ns) issue_records(k + 1);
        const unsigned char* buf = ring + (k & 1) * (B * REC);
        // a lane group takes adjacent list entries in turn, as few turns as the
        // stage's entries need
        const int have = min(B, ns - k * B), turns = (have + SW - 1) / SW;
#pragma unroll 1
        for (int u = 0; u < turns; ++u) {
            const int e = grp * turns + u;
            const bool on = e < have;
            const unsigned char* rec = buf + (on ? e : 0) * REC;
            const int4 meta = *reinterpret_cast<const int4*>(rec);   // region cell, index, phase
            const float* coef = reinterpret_cast<const float*>(rec + 16);
            float q[L::NC];
            load_coefs(coef, q);
            float qx[JH];   // this lane's taps along axis 0: th, th + TSP, ...
#pragma unroll
            for (int j = 0; j < JH; ++j) qx[j] = TSP > 1 ? coef[j * TSP + th] : q[j];
            const V* w = S + (meta.x + th) * LL + cl;
            V acc = {};
#pragma unroll
            for (int j2 = 0; j2 < (NDIM > 2 ? J : 1); ++j2) {
                V plane = {};
#pragma unroll
                for (int j1 = 0; j1 < J; ++j1) {
                    const V* r = w + j2 * ps + j1 * rs;
                    V row = {};
#pragma unroll
                    for (int j = 0; j < JH; ++j) {
                        // lanes whose next tap lies past the window leave the cell
                        // there alone: it must not enter, not even times zero
                        if (j * TSP + TSP <= J)
                            add_scaled(row, qx[j], r[j * TSP * LL]);
                        else if (j * TSP + th < J)
                            add_scaled(row, qx[j], r[j * TSP * LL]);
                    }
                    add_scaled(plane, q[J + j1], row);
                }
                if (NDIM > 2)
                    add_scaled(acc, q[2 * J + j2 < L::NC ? 2 * J + j2 : 0], plane);
                else
                    acc = plane;
            }
            float2 va = first_coil(acc), vb = second_coil(acc);
            if (TSP > 1) {
                // sum over the lane groups; with two coils each pair of groups
                // first splits them
                if (VC == 2) va = add_lane(th & 1 ? vb : va, th & 1 ? va : vb, LL);
#pragma unroll
                for (int o = VC * LL; o < GL; o *= 2) va = add_lane(va, va, o);
            }
            if (!writes) continue;
            if (!on || wc >= nc) continue;
            const int idx = meta.y;
            if (!GBN_INB(g.check, idx >= 0 && idx < Mf, CHK_SAMPLE_WRITE)) continue;
            if (p.apply_ph) {
                const float2 ph = make_float2(__int_as_float(meta.z), __int_as_float(meta.w));
                va = cmul(va, ph);
                if (TSP == 1) vb = cmul(vb, ph);
            }
            // samples idx, idx + 1 (idx even) in consecutive entries leave as
            // one 16-byte store per coil
            const bool two = TSP == 1 && VC == 2 && wc + 1 < nc;
            if (pidx >= 0 && idx == pidx + 1) {
                put(yb, idx, pa, va, (reinterpret_cast<uintptr_t>(yb + pidx) & 15) == 0);
                if ((reinterpret_cast<uintptr_t>(yb + pidx) & 15) != 0) yb[pidx] = pa;
                if (two) {
                    float2* y2 = yb + Mf;
                    const bool al = (reinterpret_cast<uintptr_t>(y2 + pidx) & 15) == 0;
                    put(y2, idx, pb, vb, al);
                    if (!al) y2[pidx] = pb;
                }
                pidx = -1;
            } else {
                if (pidx >= 0) {
                    yb[pidx] = pa;
                    if (two) yb[Mf + pidx] = pb;
                    pidx = -1;
                }
                if ((idx & 1) == 0) {
                    pidx = idx;
                    pa = va;
                    pb = vb;
                } else {
                    yb[idx] = va;
                    if (two) yb[Mf + idx] = vb;
                }
            }
        }
    }
    if (pidx >= 0 && wc < nc) {
        yb[pidx] = pa;
        if (TSP == 1 && VC == 2 && wc + 1 < nc) yb[Mf + pidx] = pb;
    }
}

template <int NDIM, int J, int LS, int CB, bool TAB = false>
cudaError_t cm_launch(const GatherParams<float>& p, cudaStream_t s) {
    int Rd[3] = {1, 1, 1};
    size_t cells = 1;
    for (int d = 0; d < NDIM; ++d) {
        Rd[d] = p.g.T[d] + p.g.J[d] - 1;
        cells *= (size_t)Rd[d];
    }
    const size_t nrows = (size_t)Rd[1] * (NDIM > 2 ? Rd[2] : 1);
    const size_t smem = tile_bytes(cells, LS) + CM_WARPS * (size_t)CmLayout<NDIM, J, LS>::RING +
                        nrows * sizeof(int64_t);
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(gather_cm_kernel<NDIM, J, LS, CB, TAB>), smem);
    if (e != cudaSuccess) return e;
    gather_cm_kernel<NDIM, J, LS, CB, TAB><<<dim3(p.nitems, p.chunks), CM_THREADS, smem, s>>>(p);
    return cudaGetLastError();
}

template <int NDIM, int J, int LS>
cudaError_t cm_bytes(const GatherParams<float>& p, cudaStream_t s) {
    if (!p.s.rec) return cm_launch<NDIM, J, LS, 8, true>(p, s);
    // 16-byte copies where every cell's coils start on a 16-byte boundary
    if constexpr (LS > 1) {
        if (p.coils % 2 == 0 && (reinterpret_cast<uintptr_t>(p.grid) & 15) == 0) return cm_launch<NDIM, J, LS, 16>(p, s);
    }
    return cm_launch<NDIM, J, LS, 8>(p, s);
}

template <int NDIM, int LS>
cudaError_t cm_width(const GatherParams<float>& p, cudaStream_t s) {
    switch (p.g.J[0]) {
        case 4: return cm_bytes<NDIM, 4, LS>(p, s);
        case 5: return cm_bytes<NDIM, 5, LS>(p, s);
        case 6: return cm_bytes<NDIM, 6, LS>(p, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

// The grid is coil-minor with its phases and scale applied, the kernel real and
// of one width on every axis, and the staged tile fits.
bool gather_cm_supported(const GatherParams<float>& p) {
    const Geom<float>& g = p.g;
    if (g.hi[0] || g.ndim < 2 || g.gsp != 1 || g.gs0 != p.coils) return false;
    if (p.apply_pb || p.grid_scale != 1.f || p.chunks > 65535) return false;
    const int LS = p.ln.LS;
    if (LS > (g.ndim == 2 ? 32 : 8)) return false;
    size_t cells = 1;
    for (int d = 0; d < g.ndim; ++d) {
        if (g.J[d] != g.J[0]) return false;
        cells *= (size_t)(g.T[d] + g.J[d] - 1);
    }
    if (g.J[0] < 4 || g.J[0] > 6) return false;
    const size_t nrows = cells / (size_t)(g.T[0] + g.J[0] - 1);
    return tile_bytes(cells, LS) + nrows * sizeof(int64_t) + 20 * 1024 <= 227 * 1024;
}

cudaError_t launch_gather_cm(const GatherParams<float>& p, cudaStream_t s) {
    if (p.nitems == 0 || p.coils == 0) return cudaSuccess;
    switch (p.ln.LS * 4 + p.g.ndim) {
        case 6: return cm_width<2, 1>(p, s);
        case 7: return cm_width<3, 1>(p, s);
        case 10: return cm_width<2, 2>(p, s);
        case 11: return cm_width<3, 2>(p, s);
        case 18: return cm_width<2, 4>(p, s);
        case 19: return cm_width<3, 4>(p, s);
        case 34: return cm_width<2, 8>(p, s);
        case 35: return cm_width<3, 8>(p, s);
        case 66: return cm_width<2, 16>(p, s);
        case 130: return cm_width<2, 32>(p, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace gbn
