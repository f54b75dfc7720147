"""The bounds-checked build (libgbnufft_checked.so) through the plan-time kernels
and the spread's variants: host and device planning, moved points, stored and
computed coefficients, sparse-mode weights, several frames, the fixed no-alloc
array.  Every index lies in its buffer (the status word stays zero) and the
results are the normal build's, bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

from tests.test_checked_build import _edge_tm, _status, checked  # noqa: F401

pytestmark = pytest.mark.gpu

L = 512


def _plan(K, J, tm, rdt, phasing, coils, lib, table_only, fo):
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    N = tuple(k // 2 for k in K)
    tdt = np.result_type(rdt, np.complex64) if phasing == "complex" else rdt
    h = [kernel_table(N[d], J, K[d], L, phasing, tdt) for d in range(len(K))]
    return GpuPlan(N, K, (J,) * len(K), L, rdt, [np.real(t) for t in h],
                   [np.imag(t) for t in h] if phasing == "complex" else None, np.ones(int(np.prod(N)), rdt), tm, None,
                   max_coils=coils, phasing=phasing, table_only=table_only, frame_offsets=fo, lib=lib)


@pytest.mark.parametrize("K,J,coils,rdt,phasing,table_only", [
    ((150,), 6, 9, np.float32, "real", False), ((150,), 5, 17, np.float64, "complex", True),
    ((64, 60), 6, 1, np.float32, "real", True), ((64, 60), 6, 8, np.float32, "real", False),
    ((64, 60), 4, 33, np.float32, "complex", True), ((40, 34), 6, 6, np.float64, "real", True),
    ((60, 64, 64), 6, 4, np.float32, "real", False), ((24, 20, 16), 5, 7, np.float64, "complex", False),
    ((24, 20, 16), 6, 3, np.float32, "real", True),
])
def test_paths(gpu_lib, checked, K, J, coils, rdt, phasing, table_only):  # noqa: F811
    nd, M = len(K), 2500
    fo = [0, 900, 900, M]
    tm = _edge_tm(K, M, seed=coils).astype(rdt)
    tm2 = np.ascontiguousarray(tm[::-1]) + rdt(0.37)
    F = len(fo) - 1
    g = torch.Generator(device="cuda").manual_seed(1)
    out = []
    for lib in (gpu_lib, checked):
        P = _plan(K, J, tm, rdt, phasing, coils, lib, table_only, fo)
        x = torch.randn((F * coils, P.Nprod), dtype=P.ctype, device="cuda", generator=g.manual_seed(1))
        y = torch.randn(coils * M, dtype=P.ctype, device="cuda", generator=g)
        res = []

        def run():
            res.append(P.forward(x, torch.empty_like(y), coils))
            res.append(P.adjoint(y, torch.empty_like(x), coils))
            grid = torch.empty(F * coils * P.Kprod, dtype=P.ctype, device="cuda")
            assert lib.gbn_interp_adjoint_noalloc(P.handle, ctypes.c_void_p(y.data_ptr()),
                                                  ctypes.c_void_p(grid.data_ptr()), coils,
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            res.append(grid)

        run()
        P.set_points_device(torch.from_numpy(tm2).cuda())
        run()
        P.set_points(tm, None)
        run()
        if not table_only:
            rng = np.random.default_rng(3)
            w = [rng.standard_normal((M, J)) for _ in range(2 * nd)]
            P.set_weights(w[:nd], w[nd:] if phasing == "complex" else None)
            run()
        torch.cuda.synchronize()
        if lib is checked:
            assert _status(P) == 0
        out.append(res)
    assert all(torch.equal(a, b) for a, b in zip(*out))
