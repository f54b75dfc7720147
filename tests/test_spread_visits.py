"""Visit-list spread (gbn_visit.cuh) against the oracle, where its work split
can go wrong: every coil-lane count and a ragged last lane, items shared by a
CTA's warps with blocks cut between them (a dense point), empty blocks, grids
that are no multiple of the register blocks, windows wrapping at every edge.

Tolerances: single precision 1e-5 relative L2, double 1e-12, those of the
other interpolation tests.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _points(K, M, dense, seed):
    """Uniform samples over three periods, some on cell centres and period
    edges, and `dense` of them around one point next to the origin."""
    rng = np.random.default_rng(seed)
    tm = rng.uniform(-1.0, 2.0, (M, len(K))) * np.asarray(K)
    tm[:8] = 0.0
    tm[8:16] = np.round(tm[8:16])
    tm[16:24] = np.asarray(K) - 1e-3
    tm[24:24 + dense] = 1.25 + 0.5 * rng.random((dense, len(K)))
    return tm


def _plan(K, J, tm, rdt, phasing, coils, table_only=False):
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    N = tuple(k // 2 for k in K)
    tdt = np.result_type(rdt, np.complex64) if phasing == "complex" else rdt
    h = [kernel_table(N[d], J[d], K[d], 512, phasing, tdt) for d in range(len(K))]
    P = GpuPlan(N, K, J, 512, rdt, [np.real(t) for t in h],
                [np.imag(t) for t in h] if phasing == "complex" else None,
                np.ones(int(np.prod(N)), rdt), tm, None, max_coils=coils, phasing=phasing, table_only=table_only)
    return P, h


@pytest.mark.parametrize("K,J,coils,precision,phasing", [
    ((40, 38), (6, 6), 1, "single", "real"), ((37, 22), (6, 6), 2, "single", "real"),
    ((40, 38), (5, 4), 4, "single", "real"), ((40, 38), (6, 6), 5, "single", "real"),
    ((37, 22), (6, 6), 8, "single", "real"), ((40, 38), (8, 3), 9, "single", "real"),
    ((40, 38), (6, 6), 17, "single", "real"), ((37, 22), (6, 6), 33, "single", "real"),
    ((6, 7), (6, 6), 32, "single", "real"), ((150,), (6,), 48, "single", "real"), ((9,), (8,), 3, "single", "real"),
    ((18, 13, 10), (6, 6, 6), 8, "single", "real"), ((18, 13, 10), (5, 6, 4), 3, "single", "real"),
    ((40, 38), (6, 6), 6, "double", "real"), ((37, 22), (6, 5), 32, "double", "real"),
    ((40, 38), (6, 6), 4, "single", "complex"), ((37, 22), (6, 6), 3, "single", "complex"),
    ((150,), (6,), 4, "single", "real"), ((18, 13, 10), (6, 6, 6), 4, "single", "real"),
    ((40, 38), (6, 6), 12, "single", "complex"), ((18, 13, 10), (6, 6, 6), 2, "double", "complex"),
])
def test_spread_matches_oracle(gpu_lib, K, J, coils, precision, phasing):
    rdt = np.float32 if precision == "single" else np.float64
    cdt = np.result_type(rdt, np.complex64)
    M = 4000
    tm = _points(K, M, 2500, seed=sum(K) + coils).astype(rdt)
    P, h = _plan(K, J, tm, rdt, phasing, coils)
    rng = np.random.default_rng(3)
    y = (rng.standard_normal((coils, M)) + 1j * rng.standard_normal((coils, M))).astype(cdt)
    out = [torch.full((coils, int(np.prod(K))), 7.0, dtype=P.ctype, device="cuda") for _ in range(2)]
    yd = torch.from_numpy(y).cuda()
    for g in out:
        P.interp_adjoint(yd, g, coils)
    assert torch.equal(out[0], out[1])   # the order of summation is fixed
    ref = O.interp_adjoint(y.T, h, J, 512, tm, K)
    assert rel_l2(out[0].cpu().numpy().T, ref) < (1e-5 if precision == "single" else 1e-12)
    # coefficients computed on the way: the same sums
    T, _ = _plan(K, J, tm, rdt, phasing, coils, table_only=True)
    T.interp_adjoint(yd, out[1], coils)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("N,K,J,coils", [
    ((30, 33), (64, 72), 6, 1), ((30, 33), (64, 72), 5, 2), ((30, 33), (64, 72), 4, 3), ((30, 33), (64, 72), 6, 4),
    ((30, 33), (64, 72), 5, 7), ((30, 33), (64, 72), 6, 8), ((30, 33), (64, 72), 4, 13), ((30, 33), (64, 72), 6, 35),
    ((30, 33, 32), (60, 64, 64), 6, 1), ((30, 33, 32), (60, 64, 64), 4, 2), ((30, 33, 32), (60, 64, 64), 5, 3),
    ((30, 33, 32), (60, 64, 64), 6, 11),
])
def test_gather_matches_oracle(gpu_lib, N, K, J, coils):
    """Coil-minor gather (gbn_gather_cm.cu): the forward transform for every
    coil-lane count, odd and even coil counts (8- and 16-byte copies), ragged
    last chunks, kernel widths whose taps fill the lane groups unevenly, heavy
    and nearly empty tiles, against the oracle; the same bits without
    precomputed coefficients."""
    from mrrt.nufft_gb300 import NufftBase
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    rng = np.random.default_rng(coils)
    nd, M = len(N), 2500
    omega = rng.uniform(-np.pi, np.pi, (M, nd))
    omega[:700] = 0.3 + 0.02 * rng.random((700, nd))
    kw = dict(Nd=N, omega=omega, Jd=(J,) * nd, Kd=K)
    x = (rng.standard_normal(N + (coils,)) + 1j * rng.standard_normal(N + (coils,))).astype(np.complex64)
    y = NufftBase(max_coils=coils, **kw).fft(x)
    assert rel_l2(y, O.OracleNufft(**kw).fft(x).reshape(y.shape)) < 1e-5
    h = [kernel_table(N[d], J, K[d], 512, "real", np.float32) for d in range(nd)]
    tm = (omega / (2 * np.pi / np.asarray(K))).astype(np.float32)
    xt = torch.from_numpy(x).permute(*reversed(range(nd + 1))).contiguous().cuda()
    out = []
    for table_only in (False, True):
        P = GpuPlan(N, K, (J,) * nd, 512, np.float32, h, None, np.ones(int(np.prod(N)), np.float32), tm, None,
                    max_coils=coils, table_only=table_only)
        out.append(P.forward(xt, torch.empty((coils, M), dtype=torch.complex64, device="cuda"), coils))
    assert torch.equal(out[0], out[1])
