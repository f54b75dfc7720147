// FFT passes (gbn_fftpass.cuh): the supported lengths and the launch, with the
// kernels of the lengths of factors two and three.
#include "gbn_fftpass.cuh"

namespace gbn {

cudaError_t launch_fftpass_short(const FftPassParams& p, int sign, cudaStream_t s);
cudaError_t launch_fftpass_long(const FftPassParams& p, int sign, cudaStream_t s);

// The lengths with kernels: a selection of the products of two factors up to 32
// that divide 480, each a compile-time split.
bool fftpass_supported(int L) {
    switch (L) {
        case 64: case 96: case 128: case 192: case 256: case 384: case 512: case 768:
        case 60: case 72: case 90: case 100: case 120: case 144: case 150: case 160: case 180: case 200: case 240:
        case 288: case 300: case 320: case 360: case 400: case 450: case 480: case 576: case 600: case 640: case 720:
            return true;
        default:
            return false;
    }
}

cudaError_t launch_fftpass(const FftPassParams& p, int sign, cudaStream_t s) {
    if (p.nin < 0 || p.nin > p.L || p.nout < 0 || p.nout > p.L || p.S <= 0 || (p.sn && (p.coils < 1 || p.frames < 1)))
        return cudaErrorInvalidValue;
    if (!p.sn && p.ncols <= 0) return cudaErrorInvalidValue;
    // Splits measured on a GB300 as strided passes (forward + inverse, packed
    // butterflies):
    //   512, 16384 columns: 16 x 32 with 16 columns per CTA 57 us, 32 x 16
    //     with 8 columns 58 us, cuFFT 62 us;
    //   384, 196608 columns: 16 x 24 321 us, 24 x 16 337 us, cuFFT 694 us;
    //   256, 8 planes of 65536 columns: 8 x 32 554 us, 16 x 16 662 us,
    //     cuFFT 808 us;
    //   128, 4 planes of 32768 columns: 8 x 16 73 us, 16 x 8 81 us, cuFFT 134 us;
    //   192: 16 x 12 116 us, 8 x 24 120 us, cuFFT 214 us; 768: 32 x 24 109 us,
    //     24 x 32 128 us, cuFFT 255 us.
    // 1024 (32 x 32, one CTA per SM at 242 registers) ran slower than cuFFT
    // (152 against about 139 us at 16384 columns) and is left to cuFFT.
    switch (p.L) {
        case 64: return pass_launch<8, 8, 16, 16>(p, sign, s);
        case 96: return pass_launch<8, 12, 16, 16>(p, sign, s);
        case 128: return pass_launch<8, 16, 16, 16>(p, sign, s);
        case 192: return pass_launch<16, 12, 16, 16>(p, sign, s);
        case 256: return pass_launch<8, 32, 16, 16>(p, sign, s);
        case 384: return pass_launch<16, 24, 16, 8>(p, sign, s);
        case 512: return pass_launch<16, 32, 16, 8>(p, sign, s);
        case 768: return pass_launch<32, 24, 8, 8>(p, sign, s);
        case 60: case 72: case 90: case 100: case 120: case 144: case 150: case 160: case 180: case 200: case 240:
            return launch_fftpass_short(p, sign, s);
        default: return launch_fftpass_long(p, sign, s);
    }
}

}  // namespace gbn
