// FFT passes (gbn_fftpass.cuh) of the shorter lengths that are not 2^a or 3 2^a: a
// translation unit of its own so that the lengths compile in parallel.
#include "gbn_fftpass.cuh"

namespace gbn {

cudaError_t launch_fftpass_short(const FftPassParams& p, int sign, cudaStream_t s) {
    switch (p.L) {
        case 60: return pass_launch<6, 10, 16, 16>(p, sign, s);
        case 72: return pass_launch<6, 12, 16, 16>(p, sign, s);
        case 90: return pass_launch<6, 15, 16, 16>(p, sign, s);
        case 100: return pass_launch<10, 10, 16, 16>(p, sign, s);
        case 120: return pass_launch<10, 12, 16, 16>(p, sign, s);
        case 144: return pass_launch<12, 12, 16, 16>(p, sign, s);
        case 150: return pass_launch<10, 15, 16, 16>(p, sign, s);
        case 160: return pass_launch<10, 16, 16, 16>(p, sign, s);
        case 180: return pass_launch<12, 15, 16, 16>(p, sign, s);
        case 200: return pass_launch<10, 20, 16, 16>(p, sign, s);
        case 240: return pass_launch<12, 20, 16, 16>(p, sign, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbn
