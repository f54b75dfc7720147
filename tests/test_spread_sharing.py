"""Which warps a spread tile's visits go to (gbn_visit.cuh): tiles of every
weight, from empty over those whose blocks go to a warp each to those whose
runs are cut between warps, against the oracle.

Tolerances: single precision 1e-5 relative L2, double 1e-12, those of the
other interpolation tests.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

L = 512


def _weights(K, seed):
    """Samples clustered so that the tiles hold from none to several hundred
    entries, with windows across the period's edges."""
    rng = np.random.default_rng(seed)
    nd = len(K)
    tm = [rng.uniform(0, 0.45, (900, nd)) * K]
    for n in (20, 40, 60, 90, 130, 200, 400, 900):
        tm.append((0.5 + 0.5 * rng.random(nd)) * K + rng.uniform(0, 5, (n, nd)))
    return np.concatenate(tm)


def plan_of(K, J, tm, rdt, phasing, coils, table_only=False, frame_offsets=None):
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    N = tuple(k // 2 for k in K)
    tdt = np.result_type(rdt, np.complex64) if phasing == "complex" else rdt
    h = [kernel_table(N[d], J, K[d], L, phasing, tdt) for d in range(len(K))]
    P = GpuPlan(N, K, (J,) * len(K), L, rdt, [np.real(t) for t in h],
                [np.imag(t) for t in h] if phasing == "complex" else None, np.ones(int(np.prod(N)), rdt),
                tm.astype(rdt), None, max_coils=coils, phasing=phasing, table_only=table_only,
                frame_offsets=frame_offsets)
    return P, h


@pytest.mark.parametrize("coils", [5, 8, 11, 32, 37])
@pytest.mark.parametrize("K,J", [((150, 141), 6), ((1500,), 5), ((37, 30, 26), 4)])
@pytest.mark.parametrize("rdt", [np.float32, np.float64])
def test_tiles_of_every_weight(gpu_lib, K, J, coils, rdt):
    tm = _weights(np.asarray(K), coils).astype(rdt)
    P, h = plan_of(K, J, tm, rdt, "real", coils)
    rng = np.random.default_rng(5)
    y = rng.standard_normal((coils, len(tm))) + 1j * rng.standard_normal((coils, len(tm)))
    y = y.astype(np.result_type(rdt, np.complex64))
    g = torch.full((coils, int(np.prod(K))), 7.0, dtype=P.ctype, device="cuda")
    P.interp_adjoint(torch.from_numpy(y).cuda(), g, coils)
    ref = O.interp_adjoint(y.T, h, (J,) * len(K), L, tm, K)
    assert rel_l2(g.cpu().numpy().T, ref) < (1e-5 if rdt == np.float32 else 1e-12)


@pytest.mark.parametrize("coils", [1, 3, 4, 5, 8, 19, 32])
@pytest.mark.parametrize("K,J,phasing", [((150, 141), 6, "real"), ((150, 141), 5, "complex"), ((1500,), 6, "real"),
                                         ((1500,), 8, "complex"), ((37, 30, 26), 6, "real"), ((37, 30, 26), 4, "complex")])
@pytest.mark.parametrize("rdt", [np.float32, np.float64])
def test_computed_coefficients(gpu_lib, K, J, phasing, coils, rdt):
    """Plans that keep no coefficients: the sums of those that do, bit for bit,
    in several frames (one empty), and with the samples read in place."""
    tm = _weights(np.asarray(K), coils)
    M = len(tm)
    fo = [0, M // 3, M // 3, M]
    P, _ = plan_of(K, J, tm, rdt, phasing, coils, frame_offsets=fo)
    T, _ = plan_of(K, J, tm, rdt, phasing, coils, table_only=True, frame_offsets=fo)
    g = torch.Generator(device="cuda").manual_seed(6)
    y = torch.randn(coils * M, dtype=P.ctype, device="cuda", generator=g)
    out = [torch.full((3 * coils, int(np.prod(K))), 7.0, dtype=P.ctype, device="cuda") for _ in range(2)]
    P.interp_adjoint(y, out[0], coils)
    T.interp_adjoint(y, out[1], coils)
    assert torch.equal(out[0], out[1])
    ys = [torch.empty_like(y) for _ in range(2)]
    P.interp_forward(out[0], ys[0], coils)
    T.interp_forward(out[0], ys[1], coils)
    assert torch.equal(ys[0], ys[1])
