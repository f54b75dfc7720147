"""``NufftBase`` on device tensors it takes as they lie, against the general
path: every layout gives the same values, shapes and strides."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nd,reps", [((17,), 1), ((17,), 4), ((20, 13), 1), ((20, 13), 3), ((9, 8, 7), 2)])
@pytest.mark.parametrize("precision", ["single", "double"])
def test_layouts_agree(gpu_lib, Nd, reps, precision):
    from mrrt.nufft_gb300 import NufftBase

    rng = np.random.default_rng(0)
    omega = rng.uniform(-np.pi, np.pi, (70, len(Nd)))
    A = NufftBase(Nd=Nd, omega=omega, Jd=4, Kd=tuple(2 * n for n in Nd), precision=precision, on_gpu=True,
                  max_coils=reps)
    dtype = torch.complex64 if precision == "single" else torch.complex128
    for call, lead in ((A.fft, Nd), (A.adj, (A.M,))):
        full = lead + ((reps,) if reps > 1 else ())
        c_order = torch.randn(full, dtype=dtype, device="cuda")
        f_order = c_order.permute(*reversed(range(c_order.dim()))).contiguous().permute(
            *reversed(range(c_order.dim())))
        want = call(c_order)
        inputs = [f_order, f_order.clone(memory_format=torch.preserve_format).requires_grad_(True),
                  f_order.conj().resolve_conj().conj(), c_order.cpu().numpy(),
                  f_order[..., None] if reps == 1 else f_order, f_order.to(torch.complex128)]
        for a in inputs:
            got = call(a)
            assert got.shape == want.shape and got.stride() == want.stride() and got.dtype == dtype
            assert not got.requires_grad
            if isinstance(a, torch.Tensor) and a.is_conj():
                continue   # what a lazy conjugate means here is the general path's
            assert torch.equal(got, want)
        with pytest.raises(ValueError):
            call(torch.randn((5,), dtype=dtype, device="cuda"))
    empty = NufftBase(Nd=Nd, omega=np.zeros((0, len(Nd))), Jd=4, Kd=tuple(2 * n for n in Nd), on_gpu=True)
    assert empty.fft(torch.zeros(Nd, dtype=torch.complex64, device="cuda")).shape == (0,)
