"""The library's FFT passes (gbn_fftpass.cuh) of every supported length against
cuFFT (plans made with GBN_FLAG_CUFFT_ONLY): both directions, odd image sizes,
coil counts on both sides of the passes' splits (one coil; rows of fewer than
four; a ragged last group of four), several frames, coil maps, 3-D.

Both factor the same transform differently in float32, so the forward and the
adjoint agree to float32 rounding: relative L2 2e-6, the tolerance of the
other FFT pass tests.
"""
import numpy as np
import pytest
import torch

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

LENGTHS = [60, 64, 72, 90, 96, 100, 120, 128, 144, 150, 160, 180, 192, 200, 240, 256, 288, 300, 320, 360, 384, 400,
           450, 480, 512, 576, 600, 640, 720, 768]


def _plans(N, K, coils, frames):
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    rng = np.random.default_rng(sum(K))
    J, M, nd = 4, 600, len(K)
    tm = (rng.uniform(0, 1, (M * frames, nd)) * np.asarray(K)).astype(np.float32)
    h = [kernel_table(N[d], J, K[d], 256, "real", np.float32) for d in range(nd)]
    sn = rng.uniform(0.5, 1.5, int(np.prod(N))).astype(np.float32)
    foff = np.arange(frames + 1, dtype=np.int64) * M
    pb = [np.pi * (n // 2) * 2 / k for n, k in zip(N, K)]
    return [GpuPlan(N, K, (J,) * nd, 256, np.float32, h, None, sn, tm, None, frame_offsets=foff, max_coils=coils,
                    pb_coef=pb, pb_order=list(range(nd)), ortho=coils == 3, cufft_only=flag) for flag in (False, True)]


def _check(N, K, coils, frames=1):
    plans = _plans(N, K, coils, frames)
    P = plans[0]
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((frames, coils, P.Nprod), dtype=torch.complex64, device="cuda", generator=g)
    maps = torch.randn((coils, P.Nprod), dtype=torch.complex64, device="cuda", generator=g)
    y = torch.randn(coils * P.M_total, dtype=torch.complex64, device="cuda", generator=g)
    calls = [
        (lambda Q, o: Q.forward(x, o, coils), torch.empty_like(y)),
        (lambda Q, o: Q.adjoint(y, o, coils), torch.empty_like(x)),
        (lambda Q, o: Q.forward_sense(x[:, 0].contiguous(), maps, o, coils), torch.empty_like(y)),
        (lambda Q, o: Q.adjoint_sense(y, maps, o, coils), torch.empty_like(x[:, 0].contiguous())),
    ]
    for call, out in calls:
        a, b = (call(Q, torch.empty_like(out)).cpu().numpy() for Q in plans)
        assert rel_l2(a, b) < 2e-6


@pytest.mark.parametrize("L", LENGTHS)
def test_2d_length(gpu_lib, L):
    _check((L // 2 - 1, 33), (L, 64), coils=1)
    _check((33, L // 2 + 1), (64, L), coils=5)


@pytest.mark.parametrize("N,K,coils,frames", [
    ((31, 45, 50), (60, 90, 100), 1, 1), ((36, 33, 32), (72, 64, 64), 3, 1), ((48, 30, 32), (96, 60, 64), 8, 1),
    ((50, 50), (100, 150), 2, 3), ((50, 49), (100, 96), 33, 2),
])
def test_coils_frames_3d(gpu_lib, N, K, coils, frames):
    _check(N, K, coils, frames)
