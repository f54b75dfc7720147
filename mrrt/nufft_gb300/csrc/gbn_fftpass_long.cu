// FFT passes (gbn_fftpass.cuh) of the longer lengths that are not 2^a or 3 2^a: a
// translation unit of its own so that the lengths compile in parallel.
#include "gbn_fftpass.cuh"

namespace gbn {

cudaError_t launch_fftpass_long(const FftPassParams& p, int sign, cudaStream_t s) {
    switch (p.L) {
        case 288: return pass_launch<12, 24, 16, 8>(p, sign, s);
        case 300: return pass_launch<15, 20, 16, 8>(p, sign, s);
        case 320: return pass_launch<16, 20, 16, 8>(p, sign, s);
        case 360: return pass_launch<15, 24, 16, 8>(p, sign, s);
        case 400: return pass_launch<20, 20, 16, 8>(p, sign, s);
        case 450: return pass_launch<15, 30, 16, 8>(p, sign, s);
        case 480: return pass_launch<20, 24, 16, 8>(p, sign, s);
        case 576: return pass_launch<24, 24, 8, 8>(p, sign, s);
        case 600: return pass_launch<20, 30, 8, 8>(p, sign, s);
        case 640: return pass_launch<20, 32, 8, 8>(p, sign, s);
        case 720: return pass_launch<24, 30, 8, 8>(p, sign, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbn
