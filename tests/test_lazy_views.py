"""Lazily conjugated and negated tensors (``t.conj()``, ``t.conj().imag`` and
their like are views that only carry a flag) mean the same as resolved ones,
in every layout and through autograd; a plan writes into no such view."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _f_order(shape, dtype=torch.complex64, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nd = len(shape)
    return torch.randn(tuple(reversed(shape)), dtype=dtype, device="cuda", generator=g).permute(*reversed(range(nd)))


def _lazy(t):
    """Views with the values of t: its conjugate's conjugate, its negative's."""
    conj = t.conj().resolve_conj().conj()
    neg = torch._neg_view(torch._neg_view(t).resolve_neg())
    assert conj.is_conj() and neg.is_neg()
    return [conj, neg, torch._neg_view(torch._neg_view(conj).resolve_neg())]


@pytest.mark.parametrize("Nd,reps", [((17,), 1), ((20, 13), 3), ((9, 8, 7), 2)])
@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("order", ["F", "C"])
def test_operator(gpu_lib, Nd, reps, precision, order):
    from mrrt.nufft_gb300 import NufftBase

    rng = np.random.default_rng(0)
    Kd = tuple(2 * n for n in Nd)
    A = NufftBase(Nd=Nd, omega=rng.uniform(-np.pi, np.pi, (70, len(Nd))), Jd=4, Kd=Kd, precision=precision,
                  on_gpu=True, max_coils=reps, order=order)
    dtype = torch.complex64 if precision == "single" else torch.complex128
    calls = [(A.fft, Nd), (A.adj, (A.M,))]
    if order == "F":
        calls += [(A.interp_table, Kd), (A.interp_table_adj, (A.M,))]
    for call, lead in calls:
        full = lead + ((reps,) if reps > 1 else ()) if order == "F" else ((reps,) if reps > 1 else ()) + lead
        for t in (_f_order(full, dtype), _f_order(full, dtype).contiguous()):
            want = call(t)
            for v in _lazy(t):
                assert torch.equal(call(v), want)


def test_series(gpu_lib):
    from mrrt.nufft_gb300.series import NufftSeries

    rng = np.random.default_rng(1)
    S = NufftSeries((20, 18), [rng.uniform(-np.pi, np.pi, (m, 2)) for m in (50, 81)], Jd=4, Kd=(40, 36), coils=3)
    x, y = torch.randn_like(S.empty_images()), torch.randn_like(S.empty_samples())
    img, maps = torch.randn_like(x[:, 0]), torch.randn_like(x[0])
    for a, b in zip(_lazy(x), _lazy(y)):
        assert torch.equal(S.forward(a), S.forward(x))
        assert torch.equal(S.adjoint(b), S.adjoint(y))
    for a, m, b in zip(_lazy(img), _lazy(maps), _lazy(y)):
        assert torch.equal(S.forward_sense(a, m), S.forward_sense(img, maps))
        assert torch.equal(S.adjoint_sense(b, m), S.adjoint_sense(y, maps))
    with pytest.raises(ValueError):
        S.forward(x, S.empty_samples().conj())
    with pytest.raises(ValueError):
        S.adjoint(y, torch._neg_view(S.empty_images()))


def test_gradients(gpu_lib):
    """Images, samples and upstream gradients that are lazy conjugates."""
    from mrrt.nufft_gb300 import NufftOperator

    rng = np.random.default_rng(2)
    om = rng.uniform(-np.pi, np.pi, (300, 2)).astype(np.float32)
    op = NufftOperator((18, 20), om, Jd=6, Kd=(36, 40), max_coils=2)
    x = torch.randn((2, 18, 20), dtype=torch.complex64, device="cuda")
    y = torch.randn((2, 300), dtype=torch.complex64, device="cuda")
    omt = torch.from_numpy(om).cuda()

    def grads(call, a, b, lazily):
        a, o = a.clone().requires_grad_(True), omt.clone().requires_grad_(True)
        out = call(a, o)
        # the gradient of sum Re(b conj(out)) reaches the operator as b, or, by way of
        # conj(out), as a lazy conjugate of conj(b)
        ((b.conj() * out).real if not lazily else (b * out.conj()).real).sum().backward()
        return a.grad, o.grad

    for call, a, b in ((op.forward, x, y), (op.adjoint, y, x)):
        want, got = grads(call, a, b, False), grads(call, a, b, True)
        for u, v in zip(want, got):
            assert torch.allclose(u, v, rtol=1e-5, atol=1e-4)
        for v in _lazy(a):
            assert torch.equal(call(v), call(a))
    # a real negated view as trajectory, and a lazily conjugated sample phase
    z = torch.complex(torch.zeros_like(omt), -omt)
    assert z.conj().imag.is_neg()
    assert torch.equal(op.forward(x, z.conj().imag), op.forward(x, omt))


def test_set_points_device(gpu_lib):
    from mrrt.nufft_gb300._kernels import kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    rng = np.random.default_rng(3)
    tm = torch.from_numpy((rng.uniform(0, 40, (200, 2))).astype(np.float32)).cuda()
    ph = torch.from_numpy(np.exp(1j * rng.uniform(0, 6, 200)).astype(np.complex64)).cuda()
    h = [kernel_table(20, 6, 40, 512, "real", np.float32)] * 2
    P = GpuPlan((20, 20), (40, 40), (6, 6), 512, np.float32, h, None, np.ones(400, np.float32), tm.cpu().numpy(), None)
    x = torch.randn((1, 20, 20), dtype=torch.complex64, device="cuda")
    y = torch.empty((1, 200), dtype=torch.complex64, device="cuda")
    P.set_points_device(tm, ph)
    want = P.forward(x, y, 1).clone()
    P.set_points_device(torch._neg_view(-tm), ph.conj().resolve_conj().conj())
    assert torch.equal(P.forward(x, y, 1), want)


def test_direct_sums_and_host_buffers(gpu_lib):
    from mrrt.nufft_gb300 import NufftBase, dtft, dtft_adj

    rng = np.random.default_rng(4)
    om = rng.uniform(-np.pi, np.pi, (60, 2))
    x, y = _f_order((12, 10), torch.complex128), _f_order((60,), torch.complex128)
    for a, b in zip(_lazy(x), _lazy(y)):
        assert torch.equal(dtft(a, om, (12, 10)), dtft(x, om, (12, 10)))
        assert torch.equal(dtft_adj(b, om, (12, 10)), dtft_adj(y, om, (12, 10)))
    P = NufftBase(Nd=(12, 10), omega=om, Jd=4, Kd=(24, 20)).plan
    x, y = torch.randn(120, dtype=torch.complex64), torch.randn(60, dtype=torch.complex64)
    for a, b in zip(_lazy(x), _lazy(y)):
        assert torch.equal(P.forward_host(a, torch.empty_like(y), 1), P.forward_host(x, torch.empty_like(y), 1))
        assert torch.equal(P.adjoint_host(b, torch.empty_like(x), 1), P.adjoint_host(y, torch.empty_like(x), 1))
    with pytest.raises(ValueError):
        P.forward_host(x, torch.empty_like(y).conj(), 1)
