"""``gbn_grad_tm`` on the grid a forward call left, whichever came first, that
call (or the capture of its graph) or the derivative tables: the grid holds its
phases or the gradient kernel applies them.

The two agree to the rounding of the phases' angles, and so do plans on cuFFT's
passes, where the kernel always applies them: up to 250 rad here, half a unit in
the last place 8e-6 rad, three roundings a cell; relative L2 1e-4.  A forward
call after the tables leaves the same grid whatever came before it.
"""
import numpy as np
import pytest
import torch

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _plan(N, K, rdt, ortho, cufft_only=False):
    from mrrt.nufft_gb300._kernels import kernel_deriv_table, kernel_table
    from mrrt.nufft_gb300._plan import GpuPlan

    nd, J, M = len(N), 6, 900
    rng = np.random.default_rng(sum(K))
    tm = (rng.uniform(-1, 2, (M, nd)) * K).astype(rdt)
    ph = np.exp(1j * rng.uniform(0, 6, M))
    h = [kernel_table(N[d], J, K[d], 512, "real", rdt) for d in range(nd)]
    P = GpuPlan(N, K, (J,) * nd, 512, rdt, h, None, rng.uniform(0.5, 1.5, int(np.prod(N))), tm, ph, max_coils=3,
                pb_coef=[2 * np.pi / k * (n // 2) for n, k in zip(N, K)], pb_order=list(range(nd)), ortho=ortho,
                cufft_only=cufft_only)
    return P, [kernel_deriv_table(N[d], J, K[d], 512, rdt) for d in range(nd)]


@pytest.mark.parametrize("N,K", [((32, 36), (64, 72)), ((30, 32, 20), (60, 64, 60)), ((31, 33), (62, 66))])
@pytest.mark.parametrize("ortho", [False, True])
@pytest.mark.parametrize("rdt", [np.float32, np.float64])
def test_order_of_forward_and_tables(gpu_lib, N, K, ortho, rdt):
    C = 3
    P, tables = _plan(N, K, rdt, ortho)
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn((C,) + tuple(reversed(N)), dtype=P.ctype, device="cuda", generator=g)
    gy = torch.randn((C, P.M_total), dtype=P.ctype, device="cuda", generator=g)
    shift = [0.25 * (d + 1) for d in range(len(N))]

    def grad(Q):
        rt = torch.float32 if rdt == np.float32 else torch.float64
        out = torch.empty((Q.M_total, len(N)), dtype=rt, device="cuda")
        return Q.grad_tm(Q.forward_grid(C), gy, shift, out, C)

    first, y = grad_tables_first(P, tables, x, gy, C, grad)
    late, _ = _plan(N, K, rdt, ortho)
    ya = late.forward(x, torch.empty_like(gy), C)
    late.set_dtables(tables)
    assert rel_l2(grad(late).cpu().numpy(), first.cpu().numpy()) < 1e-4
    assert rel_l2(ya.cpu().numpy(), y.cpu().numpy()) < 1e-6
    late.forward(x, ya, C)
    assert torch.equal(ya, y) and torch.equal(grad(late), first)
    # a graph captured before the tables were set
    rec, _ = _plan(N, K, rdt, ortho)
    yc = rec.forward(x, torch.empty_like(gy), C)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rec.forward(x, yc, C)
    rec.set_dtables(tables)
    graph.replay()
    assert rel_l2(grad(rec).cpu().numpy(), first.cpu().numpy()) < 1e-4
    rec.forward(x, yc, C)
    assert torch.equal(grad(rec), first)
    graph.replay()
    assert rel_l2(grad(rec).cpu().numpy(), first.cpu().numpy()) < 1e-4
    other, _ = _plan(N, K, rdt, ortho, cufft_only=True)
    other, _ = grad_tables_first(other, tables, x, gy, C, grad)
    assert rel_l2(first.cpu().numpy(), other.cpu().numpy()) < 1e-4


def grad_tables_first(P, tables, x, gy, C, grad):
    P.set_dtables(tables)
    y = P.forward(x, torch.empty_like(gy), C)
    return grad(P), y
