// Sum of the partial tiles of the adjoint spread (gbn_visit.cuh): a tile of
// more entries than one work item takes is split into parts, each writing its
// partial sums to a scratch slot; this kernel adds them in part order, applies
// conj(phase_before) and writes the grid.
#include <cuda_runtime.h>

#include "gbn_device.cuh"
#include "gbn_internal.h"

namespace gbn {

int spread_threads(int ndim, const int* T) {
    int b[3];
    if (ndim == 1) { b[0] = SpreadBlock<1>::B0; b[1] = b[2] = 1; }
    else if (ndim == 2) { b[0] = SpreadBlock<2>::B0; b[1] = SpreadBlock<2>::B1; b[2] = 1; }
    else { b[0] = SpreadBlock<3>::B0; b[1] = SpreadBlock<3>::B1; b[2] = SpreadBlock<3>::B2; }
    int warps = 1;
    for (int d = 0; d < ndim; ++d) warps *= T[d] / b[d];
    return 32 * warps;
}

// Sum the parts of split tiles in part order and write the grid.  One
// thread per (coil, cell) of a tile; a tile's TT x LS elements are spread
// over `nsub` CTAs (blockIdx.x = tile * nsub + sub) so that the many small
// partial-sum reads are in flight at once.  The parts are loaded four at a
// time and added in part order, so the result is the same in every run.
template <typename R, int NDIM>
__global__ void __launch_bounds__(256) reduce_kernel(const ReduceParams<R> p, const int nsub) {
    typedef typename Cx<R>::T C;
    const Geom<R>& g = p.g;
    const int ti = blockIdx.x / nsub;
    const int sub = blockIdx.x - ti * nsub;
    const int4 tl = p.tiles[ti];
    const int f = tl.x, tile = tl.y, slot0 = tl.z, nparts = tl.w;
    const int LS = p.ln.LS, lsh = p.ln.lsh;
    const int c0 = blockIdx.y << lsh;
    const int nc = min(LS, p.coils - c0);
    int org[3] = {0, 0, 0}, ext[3] = {1, 1, 1}, Td[3] = {1, 1, 1};
    tile_origin<NDIM>(tile, g.nt, g.T, org);
#pragma unroll
    for (int d = 0; d < NDIM; ++d) {
        Td[d] = g.T[d];
        ext[d] = min(g.T[d], g.K[d] - org[d]);
    }
    const int TT = Td[0] * Td[1] * Td[2];
    const int q = sub * blockDim.x + threadIdx.x;
    if (q >= TT * LS) return;
    const int cell = q >> lsh, c = q & (LS - 1);   // coils fastest, as the partial sums lie
    if (c >= nc) return;
    int r[3];
    r[0] = cell % Td[0];
    r[1] = (cell / Td[0]) % Td[1];
    r[2] = cell / (Td[0] * Td[1]);
    bool inside = true;
#pragma unroll
    for (int d = 0; d < NDIM; ++d) inside = inside && (r[d] < ext[d]);
    if (!inside) return;
    const int64_t pstride = (int64_t)gridDim.y * LS * p.tile_cells;
    const int64_t s0 = (((int64_t)slot0 * gridDim.y + blockIdx.y) * p.tile_cells + cell) * LS + c;
    if (!GBN_INB(g.check, slot0 >= 0 && nparts >= 1 && s0 + (int64_t)(nparts - 1) * pstride < p.scratch_elems,
                 CHK_SCRATCH))
        return;
    const C* src = p.scratch + s0;
    C acc = cmake<R>((R)0, (R)0);
    int s = 0;
    for (; s + 4 <= nparts; s += 4) {
        const C v0 = src[(int64_t)s * pstride];
        const C v1 = src[(int64_t)(s + 1) * pstride];
        const C v2 = src[(int64_t)(s + 2) * pstride];
        const C v3 = src[(int64_t)(s + 3) * pstride];
        acc.x += v0.x; acc.y += v0.y;
        acc.x += v1.x; acc.y += v1.y;
        acc.x += v2.x; acc.y += v2.y;
        acc.x += v3.x; acc.y += v3.y;
    }
    for (; s < nparts; ++s) {
        const C v = src[(int64_t)s * pstride];
        acc.x += v.x;
        acc.y += v.y;
    }
    int k[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < NDIM; ++d) k[d] = org[d] + r[d];
    const int64_t off = k[0] * g.gs0 + (int64_t)k[1] * g.gs1 + (int64_t)k[2] * g.gs2;
    if (p.apply_pb) acc = cmulc(acc, phase_before(g, k));
    const int64_t gi = f * g.gsf + (c0 + c) * g.gsp + off;
    if (GBN_INB(g.check, gi >= 0 && gi < g.grid_elems, CHK_GRID_WRITE)) p.grid[gi] = acc;
}

template <typename R>
cudaError_t launch_reduce(const ReduceParams<R>& p, cudaStream_t s) {
    if (p.ntiles == 0 || p.coils == 0) return cudaSuccess;
    const int64_t tt = (int64_t)p.g.T[0] * (p.g.ndim > 1 ? p.g.T[1] : 1) * (p.g.ndim > 2 ? p.g.T[2] : 1);
    const int nsub = (int)((tt * p.ln.LS + 255) / 256);
    dim3 grid((unsigned)((int64_t)p.ntiles * nsub), (p.coils + p.ln.LS - 1) / p.ln.LS);
    switch (p.g.ndim) {
        case 1: reduce_kernel<R, 1><<<grid, 256, 0, s>>>(p, nsub); break;
        case 2: reduce_kernel<R, 2><<<grid, 256, 0, s>>>(p, nsub); break;
        case 3: reduce_kernel<R, 3><<<grid, 256, 0, s>>>(p, nsub); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template cudaError_t launch_reduce<float>(const ReduceParams<float>&, cudaStream_t);
template cudaError_t launch_reduce<double>(const ReduceParams<double>&, cudaStream_t);

}  // namespace gbn
