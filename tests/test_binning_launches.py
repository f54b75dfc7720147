"""Device binning at the edges of its launches: one sample, one tile of a scan
and one sample more, more scan tiles than a block sums for itself (2^21
elements) with the sorts of both lists in large tiles, and sorts of an odd
number of digits beside an even one.  The lists are those of the host planner,
so the transforms of both plans are the same bits."""
import numpy as np
import pytest
import torch

from tests.test_device_binning import STAT_KEYS, _plans, _transforms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nd, Kd, Jd, M", [
    ((100,), (200,), (7,), 1),
    ((3000,), (6000,), (4,), 2048),
    ((40, 36), (80, 72), (6, 5), 2049),
    ((64, 64), (128, 128), (4, 4), 2_200_000),
])
def test_lists_equal_host_lists(gpu_lib, Nd, Kd, Jd, M):
    rng = np.random.default_rng(M)
    om = [rng.uniform(-np.pi, np.pi, (M, len(Nd))) for _ in range(2)]
    tms = [o / (2 * np.pi / np.asarray(Kd, dtype=np.float64)) for o in om]
    host, dev = _plans(Nd, Kd, Jd, tms, 2)
    sh, sd = host.stats(), dev.stats()
    assert {k: sh[k] for k in STAT_KEYS} == {k: sd[k] for k in STAT_KEYS}
    yh, xh = _transforms(host, 2, 3)
    yd, xd = _transforms(dev, 2, 3)
    assert torch.equal(yh, yd)
    assert torch.equal(xh, xd)


@pytest.mark.parametrize("J", [4, 5, 6, 7])
def test_first_taps_at_edges(gpu_lib, J):
    """Coordinates a step of the format around integers, half integers and
    zero, and small enough to vanish beside J/2 in double: the single-precision
    first taps of the device are the host's, computed in double."""
    f = np.float32
    t = np.concatenate([np.arange(-90, 90) / 2.0, 2.0 ** np.arange(-60, 0), -(2.0 ** np.arange(-140, 0))]).astype(f)
    up, down = [t], [t]
    for _ in range(2):
        up.append(np.nextafter(up[-1], f(np.inf)))
        down.append(np.nextafter(down[-1], f(-np.inf)))
    t = np.concatenate(up + down[1:]).astype(np.float64)[:, None]
    host, dev = _plans((45,), (90,), (J,), [t[::-1].copy(), t], 1)
    sh, sd = host.stats(), dev.stats()
    assert {k: sh[k] for k in STAT_KEYS} == {k: sd[k] for k in STAT_KEYS}
    yh, xh = _transforms(host, 1, 3)
    yd, xd = _transforms(dev, 1, 3)
    assert torch.equal(yh, yd)
    assert torch.equal(xh, xd)
