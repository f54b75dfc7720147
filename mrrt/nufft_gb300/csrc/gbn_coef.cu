// Plan-time preparation of the gather list, and the phase table.
//
// A sample's interpolation coefficients depend only on its coordinates, which
// are fixed per plan, so the gather reads them instead of interpolating the
// lookup tables for every call.  Table mode fills them with table_coef, the
// device function the kernels would use, so results are bitwise those of the
// table path.  Sparse-matrix mode fills them from the per-sample weights of
// the reference's precomputed interpolation matrix
// (mrrt/nufft/_nufft.py:750-877).  For the coil-minor gather
// (gbn_gather_cm.cu) an entry's record also holds its window's place in the
// staged tile, its output index and its phase.
//
// phase_before of every grid cell is as fixed (a sum rounded in the working
// precision, then a sincos): the table replaces a sincos per staged or
// written cell by a load.
#include <cuda_runtime.h>

#include "gbn_device.cuh"
#include "gbn_internal.h"

namespace gbn {

namespace {

// One thread per (entry, coefficient): consecutive threads write consecutive
// values (one CTA per work item, some hundred values each, took 27 us on a
// 65,536-sample trajectory).
template <typename R, bool CX>
__global__ void __launch_bounds__(256) coef_kernel(const CoefParams<R> p) {
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= p.s.len * p.jsum) return;
    const Geom<R>& g = p.g;
    const int64_t e = q / p.jsum;
    int j = (int)(q - e * p.jsum);
    const int k = j;
    int d = 0;
    while (d + 1 < g.ndim && j >= g.J[d]) {
        j -= g.J[d];
        ++d;
    }
    R cr, ci = (R)0;
    int f = 0;
    if (p.wr[0] || k == 0 || !p.place) {
        // the gather list is sorted by frame first, one entry per sample
        int hi = p.F;
        while (hi - f > 1) {
            const int mid = (f + hi) >> 1;
            if (p.foff[mid] <= e) f = mid;
            else hi = mid;
        }
    }
    if ((k == 0 || !p.place) && !GBN_INB(g.check, p.foff[f] + p.s.idx[e] < p.s.len, CHK_LIST)) return;
    if (k == 0 && p.place) p.place[p.foff[f] + p.s.idx[e]] = (int)e;
    if (p.wr[0]) {
        const int64_t w = (p.foff[f] + p.s.idx[e]) * g.J[d] + j;
        cr = p.wr[d][w];
        if (CX) ci = p.wi[d][w];
    } else {
        const R t = p.s.t[d][e];
        table_coef<R, CX>(g, d, t, first_tap(t, g.J[d]) + j, cr, ci);
    }
    R* rec = p.out + (p.place ? e : p.foff[f] + p.s.idx[e]) * p.stride;
    rec[p.off + k] = cr;
    if (CX) rec[p.off + p.jsum + k] = ci;
    if (sizeof(R) == 4 && !CX && k == 0 && p.place) {
        // the record's head: {cell of the window's start in the staged tile, index, phase}
        int cell = 0, mul = 1;
        for (int a = 0; a < g.ndim; ++a) {
            cell += mul * (wrapk(first_tap(p.s.t[a][e], g.J[a]), g.K[a]) % g.T[a]);
            mul *= g.T[a] + g.J[a] - 1;
        }
        float2 ph = make_float2(1.f, 0.f);
        if (p.s.ph) ph = make_float2((float)p.s.ph[e].x, (float)p.s.ph[e].y);
        *reinterpret_cast<int4*>(rec) = make_int4(cell, p.s.idx[e], __float_as_int(ph.x), __float_as_int(ph.y));
        for (int z = p.off + p.jsum; z < p.stride; ++z) rec[z] = (R)0;
    }
}

template <typename R>
__global__ void __launch_bounds__(256) phase_kernel(const Geom<R> g, typename Cx<R>::T* out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.Kprod) return;
    const int k[3] = {(int)(i % g.K[0]), (int)(i / g.K[0] % g.K[1]), (int)(i / g.K[0] / g.K[1])};
    out[i] = phase_before(g, k);
}

}  // namespace

template <typename R>
cudaError_t launch_coef(const CoefParams<R>& p, cudaStream_t s) {
    const int64_t n = p.s.len * p.jsum;
    if (n == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (p.cx)
        coef_kernel<R, true><<<blocks, 256, 0, s>>>(p);
    else
        coef_kernel<R, false><<<blocks, 256, 0, s>>>(p);
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_phase_table(const Geom<R>& g, typename Cx<R>::T* out, cudaStream_t s) {
    phase_kernel<R><<<(unsigned)((g.Kprod + 255) / 256), 256, 0, s>>>(g, out);
    return cudaGetLastError();
}

template cudaError_t launch_coef<float>(const CoefParams<float>&, cudaStream_t);
template cudaError_t launch_coef<double>(const CoefParams<double>&, cudaStream_t);
template cudaError_t launch_phase_table<float>(const Geom<float>&, float2*, cudaStream_t);
template cudaError_t launch_phase_table<double>(const Geom<double>&, double2*, cudaStream_t);

}  // namespace gbn
