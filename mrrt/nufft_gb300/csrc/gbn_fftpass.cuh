// Pruned FFT passes of the oversampled transforms, one axis each, with the
// deapodisation, zero-pad, crop and phase_before folded in.
//
// The oversampled FFT (mrrt/nufft/_nufft.py:1330-1350 forward fftn of the
// zero-padded image, :1561-1572 adjoint ifftn before the crop) runs axis by
// axis.  A pass transforms columns of length L at a fixed element stride;
// half of every axis is zero padding, so a forward pass reads only the nin =
// N_d rows that hold data and an inverse pass writes only the nout = N_d rows
// used afterwards.
//
// Order.  The forward goes from the slowest axis to the contiguous one, the
// inverse back: an axis is widened only once the others before it are, so the
// passes with large element strides run on the small arrays,
//   3-D forward: image [N2][N1][N0] -> [K2][N1][N0] -> [K2][K1][N0] -> [K2][K1][K0],
// and the largest one, which moves half of all bytes, is along contiguous
// rows.  (Contiguous axis first, the last pass of a 256^3 grid of 8 coils had
// its elements 4 MB apart and took 505 us; 8 planes 512 KB apart, 291 us.)
// The grid and the arrays between are coil-minor ([...][k0][coil]); images
// are [coil][...], and the first pass of the forward and the last of the
// inverse do the transposition on the way: a CTA takes 4 adjacent positions of
// 4 coils, 32-byte segments on both sides.
//
// Algorithm: the four-step split L = L1 L2 of the Cooley-Tukey FFT,
//   X[k2 + L2 k1] = sum_n1 W_L1^(n1 k1) W_L^(n1 k2) sum_n2 x[n1 + L1 n2] W_L2^(n2 k2),
// with W_M = exp(-2 pi i / M) forward and its conjugate inverse.
//   step A: a thread per (column, n1) loads the L2 elements n1 + L1 n2,
//     transforms them in registers, multiplies by W_L^(n1 k2) and stores to
//     shared memory;
//   step B: a thread per (column, k2) reads its L1 values back, transforms
//     them in registers and stores elements k2 + L2 k1.
// Consecutive threads take consecutive columns (TC of them a CTA), or, where
// adjacent columns are whole rows apart (the contiguous axis with fewer than
// four coils: RM), consecutive elements of one.
// The register transforms are Stockham autosort FFTs (Govindaraju et al.,
// "High performance discrete Fourier transforms on graphics processors",
// SC 2008), radix 4, 2, 3 and 5 stages fully unrolled; their roots are compile-
// time constants in constant memory, the W_L^(n1 k2) twiddles a per-plan
// table computed on the host in double precision.  Single precision only;
// other lengths and double precision run through cuFFT.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gbn_device.cuh"
#include "gbn_fft.cuh"
#include "gbn_internal.h"

namespace gbn {

namespace {

// PLAIN: columns of arrays; IMAGE: one side is the image (forward in, inverse
// out); PHASE: forward, plain, the outputs times phase_before.
enum PassMode { PLAIN, IMAGE, PHASE };

template <int L1, int L2>
__host__ __device__ constexpr int row_block() {   // exchange values per column (RM), odd rows of L1
    return L2 * (L1 | 1) + ((2 - L2 * (L1 | 1)) % 16 + 16) % 16;
}
template <int L1, int L2, int TC, bool RM>
__host__ __device__ constexpr size_t exchange_bytes() {
    return (size_t)TC * (RM ? row_block<L1, L2>() : L1 * L2) * sizeof(float2);
}

// CTAs per SM asked of the compiler: as many as the register transforms leave
// room for, left to itself it may take 148 registers for loads in flight.  (At
// 128 in place of 96 registers the 256-point passes of a 128^3, 8-coil pair
// took 70 us more.)  96 for the longest transforms give a 256-thread CTA two,
// with room for loads in flight; with three the 512-point passes took 154 in
// place of 142 us (256^2, 32 coils, forward) and 196 in place of 182 (adjoint).
template <int L1, int L2, int TC>
__host__ __device__ constexpr int pass_ctas(PassMode mode) {
    const int big = L1 > L2 ? L1 : L2, threads = TC * L1;
    const int regs = (big <= 12 ? 48 : big <= 16 ? 64 : big <= 24 ? 80 : 96) +
                     // the phases held beside a column (16 x 12 spilled at 64)
                     (mode == PHASE && L2 == 12 ? 16 : 0);
    const int ctas = 65536 / (threads * regs);
    return ctas < 1 ? 1 : ctas > 16 ? 16 : ctas;
}

template <int L1, int L2, int TC, int SIGN, PassMode MODE, bool RM>
__global__ void __launch_bounds__(TC * L1, (pass_ctas<L1, L2, TC>(MODE))) fftpass_kernel(const FftPassParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sm = reinterpret_cast<float2*>(smem_raw);
    if (MODE != IMAGE && SIGN < 0 && p.state && blockIdx.x == 0 && threadIdx.x == 0) *p.state = MODE == PHASE;
    auto at = [](int col, int k2, int n1) {
        return RM ? col * row_block<L1, L2>() + k2 * (L1 | 1) + n1 : (k2 * L1 + n1) * TC + col;
    };
    // a column's first element on the array side (arr) and, IMAGE, on the
    // image side (img), its place in sn and maps, its row of the phase table
    struct Col {
        bool ok;
        int64_t in, out, img, map;
        int xy;
        unsigned a;
    };
    // `t`: position in the CTA, columns fastest on the array side; the image
    // side (`side`) takes positions fastest
    auto col_of = [&](int t, bool side, int& canon) {
        Col c;
        if constexpr (MODE == IMAGE) {
            const int cw = 1 << p.cwsh, tx = TC >> p.cwsh;
            const int xl = side ? t % tx : t >> p.cwsh, cl = side ? t / tx : t & (cw - 1);
            canon = (xl << p.cwsh) + cl;
            const unsigned ct = blockIdx.x % (unsigned)p.nct, r = blockIdx.x / (unsigned)p.nct;
            const unsigned xt = r % (unsigned)p.nxt, f = r / (unsigned)p.nxt;
            const int xy = (int)xt * tx + xl, co = (int)ct * cw + cl;
            c.ok = xy < p.Sxy && co < p.coils;
            c.xy = xy;
            const int64_t vol = (int64_t)p.Sxy * (SIGN < 0 ? p.nin : p.nout);
            c.map = co * vol + xy;
            c.img = (p.maps && SIGN < 0 ? f * vol : ((int64_t)f * p.coils + co) * vol) + xy;
            const int64_t arr = f * (SIGN < 0 ? p.pso : p.psi) + (int64_t)xy * p.coils + co;
            c.in = SIGN < 0 ? c.img : arr;
            c.out = SIGN < 0 ? arr : c.img;
            c.a = 0;
        } else {
            canon = t;
            const unsigned j = blockIdx.x * TC + t;
            c.a = j / (unsigned)p.S;
            const unsigned s = j - c.a * (unsigned)p.S;
            c.ok = j < (unsigned)p.ncols;
            c.in = c.a * p.psi + s;
            c.out = c.a * p.pso + s;
        }
        return c;
    };
    const int64_t si = MODE == IMAGE && SIGN < 0 ? p.Sxy : p.S, so = MODE == IMAGE && SIGN > 0 ? p.Sxy : p.S;

    // step A: (column, n1), L2-point transforms of elements n1 + L1 n2
    {
        const int t = RM ? threadIdx.x / L1 : threadIdx.x % TC, n1 = RM ? threadIdx.x % L1 : threadIdx.x / TC;
        int col;
        const Col c = col_of(t, SIGN < 0, col);
        float2 v[L2];
        // one running pointer: offsets formed per element from a 64-bit stride
        // cost the longer passes 40 to 60 registers
        const float2* src = p.in + c.in + n1 * si;
        const int64_t step = L1 * si;
        const int lim = c.ok ? p.nin : 0;
#pragma unroll
        for (int n2 = 0; n2 < L2; ++n2) {
            v[n2] = make_float2(0.f, 0.f);
            if (n1 + L1 * n2 < lim && GBN_INB(p.check, src >= p.in && src < p.in + p.in_elems,
                                              MODE == IMAGE && SIGN < 0 ? CHK_IMAGE : CHK_GRID_READ))
                v[n2] = *src;
            src += step;
        }
        if (MODE == IMAGE && SIGN < 0) {
            if (p.maps) {
                const float2* m = p.maps + c.map + n1 * si;
#pragma unroll
                for (int n2 = 0; n2 < L2; ++n2, m += step)
                    if (n1 + L1 * n2 < lim) v[n2] = cmul(v[n2], __ldg(m));
            }
            const float* w = p.sn + c.xy + n1 * si;
#pragma unroll
            for (int n2 = 0; n2 < L2; ++n2, w += step)
                if (n1 + L1 * n2 < lim) {
                    const float f = __ldg(w);
                    v[n2] = make_float2(v[n2].x * f, v[n2].y * f);
                }
        }
        stockham<L2, 1, SIGN>(v);
#pragma unroll
        for (int k2 = 1; k2 < L2; ++k2) {
            float2 w = __ldg(p.tw + n1 * k2);   // n1 k2 < L
            if (SIGN > 0) w.y = -w.y;
            v[k2] = cmul(v[k2], w);
        }
#pragma unroll
        for (int k2 = 0; k2 < L2; ++k2) sm[at(col, k2, n1)] = v[k2];
    }
    __syncthreads();
    // step B: (column, k2), L1-point transforms, elements k2 + L2 k1 out
    for (int q = threadIdx.x; q < TC * L2; q += TC * L1) {
        const int t = RM ? q / L2 : q % TC, k2 = RM ? q % L2 : q / TC;
        int col;
        const Col c = col_of(t, SIGN > 0, col);
        float2 u[L1];
#pragma unroll
        for (int n1 = 0; n1 < L1; ++n1) u[n1] = sm[at(col, k2, n1)];
        stockham<L1, 1, SIGN>(u);
        if (MODE == PHASE && c.ok) {
            const float2* ph = p.phase + (int64_t)(c.a % (unsigned)p.prows) * (L1 * L2) + k2;
#pragma unroll
            for (int k1 = 0; k1 < L1; ++k1) u[k1] = cmul(u[k1], __ldg(ph + L2 * k1));
            if (p.div != 1.f) {
#pragma unroll
                for (int k1 = 0; k1 < L1; ++k1) u[k1] = make_float2(u[k1].x / p.div, u[k1].y / p.div);
            }
        }
        float2* dst = p.out + c.out + k2 * so;
        const int64_t step = L2 * so;
        const int lim = c.ok ? p.nout : 0;
        const float* w = MODE == IMAGE && SIGN > 0 ? p.sn + c.xy + k2 * so : nullptr;
#pragma unroll
        for (int k1 = 0; k1 < L1; ++k1) {
            if (k2 + L2 * k1 < lim && GBN_INB(p.check, dst >= p.out && dst < p.out + p.out_elems,
                                              MODE == IMAGE && SIGN > 0 ? CHK_IMAGE : CHK_GRID_WRITE)) {
                if (MODE == IMAGE && SIGN > 0) {
                    const float f = __ldg(w);
                    float2 o = make_float2(u[k1].x * p.scale, u[k1].y * p.scale);
                    o.x *= f;
                    o.y *= f;
                    *dst = o;
                } else {
                    *dst = u[k1];
                }
            }
            dst += step;
            if (MODE == IMAGE && SIGN > 0) w += step;
        }
    }
}

template <int L1, int L2, int TC, int SIGN, PassMode MODE, bool RM>
cudaError_t pass_run(const FftPassParams& p, cudaStream_t s) {
    constexpr size_t smem = exchange_bytes<L1, L2, TC, RM>();
    cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(fftpass_kernel<L1, L2, TC, SIGN, MODE, RM>), smem);
    if (e != cudaSuccess) return e;
    FftPassParams q = p;
    int64_t ctas;
    if (MODE == IMAGE) {
        q.cwsh = p.coils >= 3 ? 2 : p.coils - 1;   // 4, 2 or 1 coils a CTA
        q.nct = (p.coils + (1 << q.cwsh) - 1) >> q.cwsh;
        const int tx = TC >> q.cwsh;
        q.nxt = (p.Sxy + tx - 1) / tx;
        ctas = (int64_t)q.nct * q.nxt * p.frames;
    } else {
        ctas = (p.ncols + TC - 1) / TC;
    }
    if (ctas > INT32_MAX || p.ncols > INT32_MAX) return cudaErrorInvalidValue;
    fftpass_kernel<L1, L2, TC, SIGN, MODE, RM><<<(unsigned)ctas, TC * L1, smem, s>>>(q);
    return cudaGetLastError();
}

template <int L1, int L2, int TC, int TR>
cudaError_t pass_launch(const FftPassParams& p, int sign, cudaStream_t s) {
    const bool rows = !p.sn && p.S < 4;   // the contiguous axis of fewer than four coils
    if (sign < 0) {
        if (p.sn) return pass_run<L1, L2, TC, -1, IMAGE, false>(p, s);
        if (p.phase)
            return rows ? pass_run<L1, L2, TR, -1, PHASE, true>(p, s) : pass_run<L1, L2, TC, -1, PHASE, false>(p, s);
        return rows ? pass_run<L1, L2, TR, -1, PLAIN, true>(p, s) : pass_run<L1, L2, TC, -1, PLAIN, false>(p, s);
    }
    if (p.sn) return pass_run<L1, L2, TC, 1, IMAGE, false>(p, s);
    return rows ? pass_run<L1, L2, TR, 1, PLAIN, true>(p, s) : pass_run<L1, L2, TC, 1, PLAIN, false>(p, s);
}

}  // namespace
}  // namespace gbn
