"""gbn_interp_adjoint_noalloc where the coil-minor values of all coils do not
fit its fixed array: they are laid out a group of coils at a time, or the spread
copies them from the samples as they lie.  Its sums are those of
gbn_interp_adjoint, bit for bit, but for more than eight coils in single
precision copied as they lie, eight at a time (to rounding, the other no-alloc
tests' tolerance).  Few windows share a tile, so that the split tiles' partial
sums leave the array to the values."""
import numpy as np
import pytest
import torch

from tests.test_spread_sharing import plan_of
from tests.conftest import rel_l2
from tests.test_zz_no_alloc import NOALLOC_CAP, TOL, _call, _noalloc, _regular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [(40,), (40, 38), (20, 18, 16)])
@pytest.mark.parametrize("coils", [1, 4, 8, 17, 32])
@pytest.mark.parametrize("rdt", [np.float32, np.float64])
@pytest.mark.parametrize("table_only", [False, True])
def test_no_samples(gpu_lib, K, coils, rdt, table_only):
    P, _ = plan_of(K, 6, np.zeros((0, len(K))), rdt, "real", coils, table_only=table_only)
    y = torch.empty((coils, 0), dtype=P.ctype, device="cuda")
    x = torch.full((coils,) + tuple(k // 2 for k in reversed(K)), 7.0, dtype=P.ctype, device="cuda")
    P.adjoint(y, x, coils)
    grids = [torch.full((coils, P.Kprod), 7.0, dtype=P.ctype, device="cuda") for _ in range(2)]
    some = torch.zeros(1, dtype=P.ctype, device="cuda")   # an address: nothing is read
    for g, call in zip(grids, ("gbn_interp_adjoint", "gbn_interp_adjoint_noalloc")):
        assert _call(P, call, some, g, coils) == 0
    assert not bool(x.any()) and not bool(grids[0].any()) and not bool(grids[1].any())


def _row(coils, rdt):
    return (coils + 1) // 2 * 2 * 2 * np.dtype(rdt).itemsize


@pytest.mark.parametrize("K,J,coils,rdt,phasing,table_only", [
    ((1024, 1000), 6, 8, np.float32, "real", False), ((1024, 1000), 6, 13, np.float32, "real", False),
    ((1024, 1000), 4, 17, np.float32, "complex", False), ((1024, 1000), 6, 32, np.float32, "real", False),
    ((1024, 1000), 6, 9, np.float64, "real", False), ((1024, 1000), 5, 37, np.float64, "complex", False),
    ((200000,), 6, 16, np.float32, "real", False), ((90, 96, 96), 6, 8, np.float64, "real", False),
    ((96, 96, 101), 5, 7, np.float32, "real", False), ((160, 152, 160), 4, 3, np.float32, "real", False),
    ((1024, 1000), 6, 8, np.float32, "real", True), ((1024, 1000), 6, 32, np.float32, "complex", True),
    ((1024, 1000), 6, 8, np.float64, "real", True),
])
def test_values_beyond_the_array(gpu_lib, K, J, coils, rdt, phasing, table_only):
    # not even the values of one chunk of coil lanes fit
    M = NOALLOC_CAP // _row(min(coils, 32), rdt) + 5000
    tm = np.random.default_rng(coils).uniform(0, 1, (M, len(K))) * K
    P, _ = plan_of(K, J, tm, rdt, phasing, coils, table_only=table_only)
    g = torch.Generator(device="cuda").manual_seed(8)
    y = torch.randn((coils, M), dtype=P.ctype, device="cuda", generator=g)
    held = P.stats()["device_bytes"]
    a = _noalloc(P, y, coils)
    assert P.stats()["device_bytes"] == held
    r = _regular(P, y, coils)
    if coils > 8 and rdt == np.float32:
        assert rel_l2(a.cpu().numpy(), r.cpu().numpy()) < TOL
    else:
        assert torch.equal(a, r)


@pytest.mark.parametrize("coils,rdt,table_only", [(64, np.float32, False), (70, np.float32, True), (33, np.float64, False),
                                                  (50, np.float64, True)])
def test_groups_of_coils(gpu_lib, coils, rdt, table_only):
    # the values of the first 32 coils fit (with the coefficients of a plan that
    # stores none beside them, in double precision), those of all do not
    M = NOALLOC_CAP // (_row(32, rdt) + (2 * 6 * 8 if table_only and rdt == np.float64 else 0)) - 100
    assert M * _row(coils, rdt) > NOALLOC_CAP
    tm = np.random.default_rng(coils).uniform(0, 1, (M, 2)) * (1024, 1000)
    P, _ = plan_of((1024, 1000), 6, tm, rdt, "real", coils, table_only=table_only)
    g = torch.Generator(device="cuda").manual_seed(9)
    y = torch.randn((coils, M), dtype=P.ctype, device="cuda", generator=g)
    assert torch.equal(_noalloc(P, y, coils), _regular(P, y, coils))
