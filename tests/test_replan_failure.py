"""A re-planning that fails (host-side injection of a failed allocation, or
invalid coordinates) leaves the plan with its old points or with none: then
every transform is refused on the host, nothing is launched, and a later
re-planning that succeeds gives the results of a new plan.

Equal plans run the same sums in the same order: results are the same bits.
"""
import ctypes

import numpy as np
import pytest
import torch

from mrrt.nufft_gb300 import _lib
from mrrt.nufft_gb300._lib import GBN_ERR_INVALID, GBN_ERR_NOMEM, GbnError

pytestmark = pytest.mark.gpu

N, K, J, M, COILS = (40, 36), (80, 72), (6, 6), 3000, 5


def _plan(tm, ph):
    from mrrt.nufft_gb300._kernels import kernel_deriv_table, kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    h = [kernel_table(N[d], J[d], K[d], 512, "real", np.float32) for d in range(2)]
    P = GpuPlan(N, K, J, 512, np.float32, h, None, np.ones(N[0] * N[1], np.float32), tm, ph, max_coils=COILS,
                pb_coef=[1.0, 0.5], pb_order=[0, 1])
    P.set_dtables([kernel_deriv_table(N[d], J[d], K[d], 512, np.float32) for d in range(2)])
    return P


def _points():
    """Few visits (every window starts on a register block) and many."""
    rng = np.random.default_rng(1)
    few = np.full((M, 2), 10.75, np.float32)
    many = (rng.uniform(-1, 2, (M, 2)) * K).astype(np.float32)
    ph = np.exp(1j * rng.uniform(0, 6, M)).astype(np.complex64)
    return few, many, ph


def _data():
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((COILS, N[1], N[0]), dtype=torch.complex64, device="cuda", generator=g)
    y = torch.randn((COILS, M), dtype=torch.complex64, device="cuda", generator=g)
    return x, y


def _results(P, x, y):
    return P.forward(x, torch.empty_like(y), COILS), P.adjoint(y, torch.empty_like(x), COILS)


def _check_refused(P, x, y):
    """Every entry point returns the error and leaves its output alone."""
    grid = torch.zeros((COILS, K[1], K[0]), dtype=torch.complex64, device="cuda")
    maps, img = torch.ones_like(x), torch.ones_like(x[0])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    gtm = torch.empty((M, 2), device="cuda")
    calls = [
        (lambda o: P.forward(x, o, COILS), y), (lambda o: P.adjoint(y, o, COILS), x),
        (lambda o: P.forward_host(x.cpu(), o, COILS), y.cpu()), (lambda o: P.adjoint_host(y.cpu(), o, COILS), x.cpu()),
        (lambda o: P.forward_sense(img, maps, o, COILS), y), (lambda o: P.adjoint_sense(y, maps, o, COILS), img),
        (lambda o: P.interp_forward(grid, o, COILS), y), (lambda o: P.interp_adjoint(y, o, COILS), grid),
        (lambda o: _lib.check(P.lib.gbn_interp_adjoint_noalloc(
            P.handle, ctypes.c_void_p(y.data_ptr()), ctypes.c_void_p(o.data_ptr()), COILS, stream)), grid),
        (lambda o: P.grad_tm(grid.data_ptr(), y, [0.0, 0.0], o, COILS), gtm),
    ]
    for call, like in calls:
        out = torch.full_like(like, 7.0)
        with pytest.raises(GbnError) as e:
            call(out)
        assert e.value.code == GBN_ERR_INVALID and "sample points" in str(e.value)
        torch.cuda.synchronize()
        assert bool((out == 7.0).all())


@pytest.mark.parametrize("device", [False, True])
def test_failed_replanning(gpu_lib, device):
    few, many, ph = _points()
    x, y = _data()
    old, new = _results(_plan(few, ph), x, y), _results(_plan(many, ph), x, y)
    refused = kept = 0

    def move(P):
        if device:
            P.set_points_device(torch.from_numpy(many).cuda(), torch.from_numpy(ph).cuda())
        else:
            P.set_points(many, ph)

    P = None
    try:
        for k in range(64):
            P = _plan(few, ph)
            assert all(torch.equal(a, b) for a, b in zip(_results(P, x, y), old))
            gpu_lib.gbn_debug_fail_alloc(k)
            try:
                move(P)
                break
            except GbnError as e:
                assert e.code == GBN_ERR_NOMEM, str(e)
            gpu_lib.gbn_debug_fail_alloc(-1)
            try:
                got = _results(P, x, y)
                assert all(torch.equal(a, b) for a, b in zip(got, old))
                kept += 1
            except GbnError:
                _check_refused(P, x, y)
                refused += 1
            move(P)
            got = _results(P, x, y)
            if not device:   # the host planner's lists and items are a new plan's
                assert all(torch.equal(a, b) for a, b in zip(got, new))
            else:
                assert all(torch.allclose(a, b, rtol=1e-4, atol=1e-4) for a, b in zip(got, new))
        else:
            pytest.fail("more than 64 allocations for a re-planning")
    finally:
        gpu_lib.gbn_debug_fail_alloc(-1)
    assert refused >= 3   # the items, the spread list, the visits
    got = _results(P, x, y)
    assert all(torch.allclose(a, b, rtol=1e-4, atol=1e-4) for a, b in zip(got, new))


def test_failed_weights(gpu_lib):
    few, many, ph = _points()
    x, y = _data()
    ref = _results(_plan(many, ph), x, y)
    w = [np.ones((M, 6), np.float32)] * 2
    P = _plan(many, ph)
    try:
        gpu_lib.gbn_debug_fail_alloc(0)
        with pytest.raises(GbnError) as e:
            P.set_weights(w)
        assert e.value.code == GBN_ERR_NOMEM
    finally:
        gpu_lib.gbn_debug_fail_alloc(-1)
    P.set_weights(None)
    assert all(torch.equal(a, b) for a, b in zip(_results(P, x, y), ref))


@pytest.mark.parametrize("device", [False, True])
def test_invalid_points_keep_the_old_ones(gpu_lib, device):
    few, many, ph = _points()
    x, y = _data()
    P = _plan(many, ph)
    ref = _results(P, x, y)
    bad = few.copy()
    bad[7, 1] = np.nan
    with pytest.raises(GbnError) as e:
        P.set_points_device(torch.from_numpy(bad).cuda()) if device else P.set_points(bad, None)
    assert e.value.code == GBN_ERR_INVALID
    assert all(torch.equal(a, b) for a, b in zip(_results(P, x, y), ref))


@pytest.mark.parametrize("on_device", [False, True])
def test_operator_after_a_failed_move(gpu_lib, on_device):
    """The operator forgets the trajectory of a move that failed: the old one
    is planned anew when it is asked for."""
    from mrrt.nufft_gb300 import NufftOperator

    rng = np.random.default_rng(3)
    om0, om1 = (rng.uniform(-np.pi, np.pi, (2, 2000, 2))).astype(np.float32)
    om0[:] = om0[0]
    op = NufftOperator((40, 36), om0, Jd=6, Kd=(80, 72))
    x = torch.randn((1, 40, 36), dtype=torch.complex64, device="cuda")
    y0 = op.forward(x).clone()
    to = (lambda o: torch.from_numpy(o).cuda()) if on_device else (lambda o: o)
    seen = 0
    try:
        for k in range(64):
            gpu_lib.gbn_debug_fail_alloc(k)
            try:
                op.set_omega(to(om1))
                break
            except GbnError:
                seen += 1
            gpu_lib.gbn_debug_fail_alloc(-1)
            assert torch.allclose(op.forward(x), y0, rtol=1e-4, atol=1e-4)
    finally:
        gpu_lib.gbn_debug_fail_alloc(-1)
    assert seen > 0


@pytest.mark.parametrize("rdt", [np.float32, np.float64])
def test_visit_coefficients_that_do_not_fit(gpu_lib, rdt):
    """A plan whose visit coefficients cannot be allocated works without them,
    to the same bits, and takes them up with weights, or when moved, with room."""
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    h = [kernel_table(N[d], J[d], K[d], 512, "real", rdt) for d in range(2)]
    _, many, ph = _points()

    def plan():
        return GpuPlan(N, K, J, 512, rdt, h, None, np.ones(N[0] * N[1], rdt), many, ph, max_coils=COILS)

    x, y = (t.to(torch.complex64 if rdt == np.float32 else torch.complex128) for t in _data())
    P = plan()
    want, held = _results(P, x, y), P.stats()["device_bytes"]
    lean = None
    try:
        for k in range(64):   # the last allocation of a construction is that of the visit coefficients
            gpu_lib.gbn_debug_fail_alloc(k)
            try:
                lean = plan()
                break
            except GbnError as e:
                assert e.code == GBN_ERR_NOMEM
    finally:
        gpu_lib.gbn_debug_fail_alloc(-1)
    got = _results(lean, x, y)
    assert lean.stats()["device_bytes"] < held
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    rng = np.random.default_rng(4)
    w = [rng.standard_normal((M, 6)) for _ in range(2)]
    P.set_weights(w)
    lean.set_weights(w)
    assert all(torch.equal(a, b) for a, b in zip(_results(lean, x, y), _results(P, x, y)))
    lean.set_points(many, ph)
    assert all(torch.equal(a, b) for a, b in zip(_results(lean, x, y), want))
    assert lean.stats()["device_bytes"] >= held
