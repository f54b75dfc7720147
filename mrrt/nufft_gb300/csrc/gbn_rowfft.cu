// Row passes of the 2-D and 3-D oversampled FFTs with the deapodisation,
// zero-pad and crop folded in.
//
// The oversampled grid is coil-minor: cell (k0, k1, k2) of coil c of frame f at
// ((f K + cell) C + c), so that the interpolation kernels find a cell's coils
// in one segment.  Image rows are contiguous per coil; a CTA's rows are
// numbered coil first, so these passes do the transposition on the way.
//
// Forward (mrrt/nufft/_nufft.py:1325-1331, then the first axis of fftn): each
// image row x[f][c][n2][n1][:N0] is multiplied by sn[n2][n1][:N0], taken as
// the first N0 of K0 values (the rest zero, never stored or read) and
// transformed along memory axis 0 into its grid row.  This replaces the pad
// kernel's write of the zero-padded planes and the row FFT's read of them.
// Inverse (the first axis of ifftn, then :1561-1572): each grid row the crop
// keeps (n1 < N1, n2 < N2) is transformed back and only its first N0 outputs
// are formed into the image, scaled by scale * sn: the row FFT's write and
// the crop's read of the transformed rows are gone.
//
// Same four-step split as the strided passes (gbn_colfft.cu), with a CTA
// owning TR whole rows: step A transforms elements n1 + L1 n2 of a row, step B
// writes elements k2 + L2 k1.  On the image's side consecutive threads take
// consecutive elements of a row, on the grid's side the same element of
// consecutive coils (CM; a plain contiguous row with one coil).  The shared
// rows of the exchange are padded to L1 + 1 and each row's block to 2 modulo
// 16 values, so that both orders of reading hit distinct banks.
// Plain transforms only: the coil-map (SENSE) variants keep the pad / crop
// kernels around the cuFFT row pass.
#include <cuda_runtime.h>

#include <cstdint>

#include "gbn_device.cuh"
#include "gbn_fft.cuh"
#include "gbn_internal.h"

namespace gbn {

namespace {

template <int L1, int L2>
__host__ __device__ constexpr int row_block() {   // exchange values per row
    return L2 * (L1 + 1) + ((2 - L2 * (L1 + 1)) % 16 + 16) % 16;
}

template <int L1, int L2, int TR, int SIGN, bool CM>
__global__ void __launch_bounds__(TR * L1) rowfft_kernel(const RowFftParams p) {
    constexpr int LP = L1 + 1, RB = row_block<L1, L2>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* sm = reinterpret_cast<float2*>(smem_raw);
    const unsigned r0 = blockIdx.x * TR;
    // row r: coil fastest, then n1, n2, frame.  Offsets of its image row, its
    // sn row and its first grid value.
    struct Row {
        bool ok;
        int64_t x, g;
        int sn;
    };
    auto row_of = [&](unsigned r) {
        Row o;
        o.ok = r < (unsigned)p.rows;
        const unsigned t = r / (unsigned)p.coils, c = r - t * p.coils;
        const unsigned t1 = t / (unsigned)p.N1, n1 = t - t1 * p.N1;
        const unsigned f = t1 / (unsigned)p.N2, n2 = t1 - f * p.N2;
        o.sn = (int)((n2 * p.N1 + n1) * p.N0);
        o.x = ((int64_t)f * p.coils + c) * ((int64_t)p.N0 * p.N1 * p.N2) + o.sn;
        o.g = f * p.gsf + n2 * p.gs2 + n1 * p.gs1 + c;
        return o;
    };

    // step A: (row, n1), L2-point transforms of elements n1 + L1 n2
    {
        constexpr bool RF = CM && SIGN > 0;   // rows (coils) fastest
        const int n1 = RF ? threadIdx.x / TR : threadIdx.x % L1;
        const int rl = RF ? threadIdx.x % TR : threadIdx.x / L1;
        const Row r = row_of(r0 + rl);
        float2 v[L2];
#pragma unroll
        for (int n2 = 0; n2 < L2; ++n2) v[n2] = make_float2(0.f, 0.f);
        if (r.ok) {
            if (SIGN < 0) {
                // image row times sn, zero past N0
                const float* s = p.sn + r.sn;
#pragma unroll
                for (int n2 = 0; n2 < L2; ++n2) {
                    const int n = n1 + L1 * n2;
                    if (n < p.N0 && GBN_INB(p.check, r.x + n < p.in_elems, CHK_IMAGE)) {
                        const float2 x = p.in[r.x + n];
                        const float w = s[n];
                        v[n2] = make_float2(x.x * w, x.y * w);
                    }
                }
            } else {
                const int64_t gs = CM ? p.coils : 1;
#pragma unroll
                for (int n2 = 0; n2 < L2; ++n2) {
                    const int64_t i = r.g + (n1 + L1 * n2) * gs;
                    if (GBN_INB(p.check, i >= 0 && i < p.in_elems, CHK_GRID_READ)) v[n2] = p.in[i];
                }
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
        for (int k2 = 0; k2 < L2; ++k2) sm[rl * RB + k2 * LP + n1] = v[k2];
    }
    __syncthreads();
    // step B: (row, k2), L1-point transforms, elements k2 + L2 k1 out
    for (int q = threadIdx.x; q < TR * L2; q += TR * L1) {
        constexpr bool RF = CM && SIGN < 0;
        const int k2 = RF ? q / TR : q % L2, rl = RF ? q % TR : q / L2;
        float2 u[L1];
#pragma unroll
        for (int n1 = 0; n1 < L1; ++n1) u[n1] = sm[rl * RB + k2 * LP + n1];
        stockham<L1, 1, SIGN>(u);
        const Row r = row_of(r0 + rl);
        if (!r.ok) continue;
        if (SIGN < 0) {
            const int64_t gs = CM ? p.coils : 1;
#pragma unroll
            for (int k1 = 0; k1 < L1; ++k1) {
                const int64_t i = r.g + (k2 + L2 * k1) * gs;
                if (GBN_INB(p.check, i >= 0 && i < p.out_elems, CHK_GRID_WRITE)) p.out[i] = u[k1];
            }
        } else {
            // the crop: first N0 outputs, times scale, times sn
            const float* s = p.sn + r.sn;
#pragma unroll
            for (int k1 = 0; k1 < L1; ++k1) {
                const int k = k2 + L2 * k1;
                if (k < p.N0 && GBN_INB(p.check, r.x + k < p.out_elems, CHK_IMAGE)) {
                    float2 t = make_float2(u[k1].x * p.scale, u[k1].y * p.scale);
                    const float w = s[k];
                    t.x *= w;
                    t.y *= w;
                    p.out[r.x + k] = t;
                }
            }
        }
    }
}

template <int L1, int L2, int TR>
cudaError_t rowfft_launch(const RowFftParams& p, int sign, cudaStream_t s) {
    const size_t smem = (size_t)TR * row_block<L1, L2>() * sizeof(float2);
    const bool cm = p.coils > 1;
    const void* k = sign < 0 ? (cm ? reinterpret_cast<const void*>(rowfft_kernel<L1, L2, TR, -1, true>)
                                   : reinterpret_cast<const void*>(rowfft_kernel<L1, L2, TR, -1, false>))
                             : (cm ? reinterpret_cast<const void*>(rowfft_kernel<L1, L2, TR, 1, true>)
                                   : reinterpret_cast<const void*>(rowfft_kernel<L1, L2, TR, 1, false>));
    cudaError_t e = ensure_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    const unsigned ctas = (unsigned)((p.rows + TR - 1) / TR);
    if (sign < 0 && cm)
        rowfft_kernel<L1, L2, TR, -1, true><<<ctas, TR * L1, smem, s>>>(p);
    else if (sign < 0)
        rowfft_kernel<L1, L2, TR, -1, false><<<ctas, TR * L1, smem, s>>>(p);
    else if (cm)
        rowfft_kernel<L1, L2, TR, 1, true><<<ctas, TR * L1, smem, s>>>(p);
    else
        rowfft_kernel<L1, L2, TR, 1, false><<<ctas, TR * L1, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace

bool rowfft_supported(int L) { return colfft_supported(L); }

// Rows per CTA and splits measured on a GB300 (pad + forward, inverse + crop):
//   512, 32 planes x 256 rows: 16 x 32 with 8 rows 16.3 + 18.0 us, 16 rows
//     18.2 + 20.7 us (cuFFT's row pass alone 13.3 us each way, plus the pad
//     or crop kernel);
//   384, 512 planes x 192 rows: 16 x 24 with 8 rows 99.7 + 110.1 us, 16 rows
//     100.2 + 117.5 us (cuFFT's row pass alone 161.5 us).
cudaError_t launch_rowfft(const RowFftParams& p, int sign, cudaStream_t s) {
    if (p.coils <= 0 || p.rows <= 0 || p.rows > INT32_MAX || p.N1 <= 0 || p.N2 <= 0 || p.N0 <= 0 || p.N0 > p.L)
        return cudaErrorInvalidValue;
    switch (p.L) {
        case 64: return rowfft_launch<8, 8, 16>(p, sign, s);
        case 96: return rowfft_launch<8, 12, 16>(p, sign, s);
        case 128: return rowfft_launch<8, 16, 16>(p, sign, s);
        case 192: return rowfft_launch<16, 12, 16>(p, sign, s);
        case 256: return rowfft_launch<8, 32, 16>(p, sign, s);
        case 384: return rowfft_launch<16, 24, 8>(p, sign, s);
        case 512: return rowfft_launch<16, 32, 8>(p, sign, s);
        case 768: return rowfft_launch<32, 24, 8>(p, sign, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbn
