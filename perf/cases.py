"""The transforms that are timed: forward and adjoint NUFFTs through the public entry points.

A case names a geometry (image size, oversampling, kernel width), a trajectory, a coil count and
the calls of one pass:

* ``kind = "operator"``: ``NufftBase.fft`` / ``NufftBase.adj`` on device tensors (``host``: on numpy
  arrays, which is how a program written for the CPU package calls it);
* ``kind = "series"``: ``NufftSeries.forward`` / ``adjoint`` of a dynamic series with uneven frames
  (``sense``: the coil-sensitivity forms);
* ``kind = "gradient"``: ``NufftOperator`` in two steps of a trajectory optimisation, each with its
  own trajectory: forward, loss, and gradients with respect to the image and the trajectory.

Sizes are those of ``bench.py`` and of the tests, or generic ones.  Images are complex N(0, 1) under
smooth coil maps, samples complex N(0, 1), trajectories radial, spiral or kooshball, turned by an
angle drawn from the seed.  ``exact`` evaluates the operator as it is defined -- the Kaiser-Bessel
tables, the sample coordinates and the grid phase in the operator's type, as its constructor fixes
them -- with every sum in 64 bits.
"""
import math

import numpy as np
import torch

from mrrt.nufft_gb300 import NufftBase, NufftOperator
from mrrt.nufft_gb300.series import NufftSeries
from mrrt.nufft_gb300.trajectories import kooshball_3d, radial_2d, spiral_2d

L = 1024   # table samples per grid cell, the default of every entry point


def listed():
    return [
        # smallest: one coil of a small image, the call of a simple script or a test; latency and
        # launches count
        dict(name="radial-128-1coil", kind="operator", Nd="128,128", Kd="256,256", J=6, coils=1, traj="radial",
             spokes=128, readout=256, calls="fft+adj", precision="single", host=False),
        # the ordinary multi-coil 2-D reconstruction, each direction by itself
        dict(name="radial-256-32coil-fft", kind="operator", Nd="256,256", Kd="512,512", J=6, coils=32,
             traj="radial", spokes=402, readout=512, calls="fft", precision="single", host=False),
        dict(name="radial-256-32coil-adj", kind="operator", Nd="256,256", Kd="512,512", J=6, coils=32,
             traj="radial", spokes=402, readout=512, calls="adj", precision="single", host=False),
        # the same from and to numpy arrays: a program that switched packages and nothing else
        dict(name="radial-256-32coil-host", kind="operator", Nd="256,256", Kd="512,512", J=6, coils=32,
             traj="radial", spokes=402, readout=512, calls="fft+adj", precision="single", host=True),
        # the constructor's defaults (J = 4, Kd = 1.5 Nd) on an odd, ragged size
        dict(name="default-200x181-12coil", kind="operator", Nd="200,181", Kd="300,271", J=4, coils=12,
             traj="radial", spokes=233, readout=400, calls="fft+adj", precision="single", host=False),
        # double precision, as used to check a reconstruction
        dict(name="radial-192-4coil-double", kind="operator", Nd="192,192", Kd="384,384", J=6, coils=4,
             traj="radial", spokes=201, readout=384, calls="fft+adj", precision="double", host=False),
        # 1-D: many short lines at once
        dict(name="lines-1d-48rep", kind="operator", Nd="1000", Kd="2000", J=6, coils=48, traj="line",
             spokes=1, readout=6000, calls="fft+adj", precision="single", host=False),
        # largest: a 3-D radial volume
        dict(name="koosh-128-8coil", kind="operator", Nd="128,128,128", Kd="256,256,256", J=6, coils=8,
             traj="koosh", spokes=12000, readout=256, calls="fft+adj", precision="single", host=False),
        # a small 3-D volume with odd sizes and an odd kernel
        dict(name="koosh-60x72x45-3coil", kind="operator", Nd="60,72,45", Kd="120,144,90", J=5, coils=3,
             traj="koosh", spokes=3001, readout=144, calls="fft+adj", precision="single", host=False),
        # a dynamic series with uneven frames, forward and adjoint
        dict(name="series-192-64x8", kind="series", Nd="192,192", Kd="384,384", J=6, coils=8, frames=64,
             least=13, most=89, readout=384, sense=False),
        # coil-combined (SENSE) forward and adjoint of a shorter series
        dict(name="sense-192-12x12", kind="series", Nd="192,192", Kd="384,384", J=6, coils=12, frames=12,
             least=13, most=89, readout=384, sense=True),
        # a differentiable step whose trajectory moves every time
        dict(name="spiral-grad-256", kind="gradient", Nd="256,256", Kd="512,512", J=6, coils=1,
             interleaves=16, samples=4096),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the same ranges: image edges 32-320 in 2-D and 24-96 in 3-D, oversampling 1.5
    and 2, J 4 to 6, 1 to 32 coils (8 in 3-D), from undersampled to fully sampled."""
    what = rng.choice(["2d", "2d", "2d", "3d", "3d", "series", "sense", "double", "1d", "gradient", "host"])
    over = rng.choice([2.0, 2.0, 1.5])
    J = rng.choice([6, 6, 6, 4, 5])

    def image(low, high, ndim):
        n = _log_int(rng, low, high)
        sizes = [n]
        for _ in range(ndim - 1):
            sizes.append(min(high, max(low, int(round(n * rng.choice([1.0, 1.0, rng.uniform(0.8, 1.25)]))))))
        return sizes

    def grid(sizes):
        return ",".join(str(int(over * n)) for n in sizes)

    def text(sizes):
        return ",".join(map(str, sizes))

    if what in ("2d", "host", "double"):
        Nd = image(32, 192 if what == "double" else 320, 2)
        n = max(Nd)
        return dict(kind="operator", Nd=text(Nd), Kd=grid(Nd), J=J,
                    coils=_log_int(rng, 1, 8 if what == "double" else 32), traj=rng.choice(["radial", "spiral"]),
                    spokes=max(8, int(n * rng.uniform(0.25, 1.6))), readout=2 * n,
                    calls="fft+adj" if what != "2d" else rng.choice(["fft", "adj", "fft+adj"]),
                    precision="double" if what == "double" else "single", host=what == "host")
    if what == "1d":
        n = _log_int(rng, 64, 4096)
        return dict(kind="operator", Nd=str(n), Kd=str(int(over * n)), J=J, coils=_log_int(rng, 1, 64), traj="line",
                    spokes=1, readout=int(n * rng.uniform(1, 8)), calls="fft+adj", precision="single", host=False)
    if what == "3d":
        Nd = image(24, 96, 3)
        n = max(Nd)
        return dict(kind="operator", Nd=text(Nd), Kd=grid(Nd), J=J, coils=_log_int(rng, 1, 8), traj="koosh",
                    spokes=max(32, int(n * n * rng.uniform(0.1, 0.6))), readout=2 * n,
                    calls=rng.choice(["fft", "adj", "fft+adj"]), precision="single", host=False)
    if what in ("series", "sense"):
        Nd = image(48, 224, 2)
        low = rng.randint(5, 21)
        return dict(kind="series", Nd=text(Nd), Kd=grid(Nd), J=J, coils=_log_int(rng, 2, 16),
                    frames=_log_int(rng, 2, 24), least=low, most=low + rng.randint(4, 60), readout=2 * max(Nd),
                    sense=what == "sense")
    Nd = image(48, 256, 2)
    return dict(kind="gradient", Nd=text(Nd), Kd=grid(Nd), J=J, coils=_log_int(rng, 1, 4),
                interleaves=rng.randint(2, 16), samples=_log_int(rng, 512, 4096))


def _ints(text):
    return tuple(int(v) for v in text.split(","))


def _rotate(om, seed):
    """The trajectory turned by an angle of the seed (in the first two axes)."""
    a = np.random.default_rng(seed).uniform(0, 2 * np.pi)
    out = om.copy()
    out[:, 0] = om[:, 0] * math.cos(a) - om[:, 1] * math.sin(a)
    out[:, 1] = om[:, 0] * math.sin(a) + om[:, 1] * math.cos(a)
    return out


def _trajectory(case, seed):
    """omega of an operator or gradient case, [M, ndim] radians."""
    if case["kind"] == "gradient":
        return _rotate(spiral_2d(case["interleaves"], case["samples"]), seed)
    if case["traj"] == "line":
        rng = np.random.default_rng(seed)
        return np.sort(rng.uniform(-np.pi, np.pi, case["readout"]))[:, None]
    if case["traj"] == "koosh":
        return _rotate(kooshball_3d(case["spokes"], case["readout"]), seed)
    if case["traj"] == "spiral":
        arms = max(1, case["spokes"] // 8)
        return _rotate(spiral_2d(arms, 8 * case["readout"]), seed)
    return _rotate(radial_2d(case["spokes"], case["readout"], golden=True), seed)


def _frames(case, seed):
    """omega of every frame: spoke counts fixed by the case, the golden-angle numbering begun anywhere."""
    frames, first = [], int(np.random.default_rng(seed).integers(0, 1000))
    for n in np.random.default_rng(4).integers(case["least"], case["most"] + 1, size=case["frames"]):
        frames.append(radial_2d(int(n), case["readout"], golden=True, first_spoke=first))
        first += int(n)
    return frames


def _normal(gen, shape, dtype):
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    parts = torch.randn(tuple(shape) + (2,), generator=gen, device="cuda", dtype=real)
    return torch.view_as_complex(parts)


def _maps(Nd, coils, dtype):
    """Smooth coil maps, [coils, *reversed(Nd)]: Gaussian blobs on a circle, each with its phase."""
    axes = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64) / n - 0.5 for n in reversed(Nd)],
                          indexing="ij")
    out = []
    for c in range(coils):
        a = 2 * math.pi * c / coils
        centre = [0.0] * (len(Nd) - 2) + [0.35 * math.sin(a), 0.35 * math.cos(a)][-len(Nd):]
        r2 = sum((x - x0) ** 2 for x, x0 in zip(axes, centre))
        out.append(torch.exp(-r2 / 0.18) * complex(math.cos(a), math.sin(a)))
    return torch.stack(out).to(dtype)


def _data(case, seed, M=None):
    """The device tensors of a case, in the plan's memory order (coil-major, first axis fastest)."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    Nd = _ints(case["Nd"])
    dtype = torch.complex128 if case.get("precision") == "double" else torch.complex64
    rev, C = tuple(reversed(Nd)), case["coils"]
    if case["kind"] == "operator":
        x = _normal(gen, rev, dtype)[None] * _maps(Nd, C, dtype) if len(Nd) > 1 else _normal(gen, (C,) + rev, dtype)
        return x, _normal(gen, (C, M), dtype)
    if case["kind"] == "series":
        F = case["frames"]
        if case["sense"]:
            return _normal(gen, (F,) + rev, dtype), _maps(Nd, C, dtype), _normal(gen, (C * M,), dtype)
        x = _normal(gen, (F, 1) + rev, dtype) * _maps(Nd, C, dtype)[None]
        return x, _normal(gen, (C * M,), dtype)
    # gradient: image [coils, *Nd] (C order) and measured samples of both steps
    scale = math.sqrt(math.prod(Nd))
    return _normal(gen, (C,) + Nd, dtype), _normal(gen, (2, C, M), dtype) * scale


def prepare(case, seed):
    Nd, Kd = _ints(case["Nd"]), _ints(case["Kd"])
    Jd = (case["J"],) * len(Nd)
    if case["kind"] == "operator":
        A = NufftBase(Nd=Nd, omega=_trajectory(case, seed), Jd=Jd, Kd=Kd, precision=case["precision"],
                      on_gpu=not case["host"], max_coils=case["coils"])
        x, k = _data(case, seed, A.M)
        # the package's convention: Nd + (coils,) and (M, coils) in Fortran order
        x, k = x.permute(*reversed(range(x.dim()))), k.t()
        if case["coils"] == 1:
            x, k = x[..., 0], k[..., 0]
        if case["host"]:
            x, k = np.asfortranarray(x.cpu().numpy()), np.asfortranarray(k.cpu().numpy())
        return dict(case=case, A=A, x=x, k=k)
    if case["kind"] == "series":
        S = NufftSeries(Nd, _frames(case, seed), Jd=Jd, Kd=Kd, coils=case["coils"])
        return dict(case=case, S=S, data=_data(case, seed, S.M_total))
    om = _trajectory(case, seed)
    op = NufftOperator(Nd, om, Jd=Jd, Kd=Kd, max_coils=case["coils"])
    x, y = _data(case, seed, op.M)
    omegas = [torch.from_numpy(o.astype(np.float32)).cuda() for o in _moved(om)]
    return dict(case=case, op=op, x=x, y=y, omegas=omegas)


def _moved(om):
    """The trajectories of two successive steps."""
    return [om * 0.999, om * 0.998 + 0.001]


def run(state):
    case = state["case"]
    if case["kind"] == "operator":
        A, out = state["A"], []
        if "fft" in case["calls"]:
            out.append(A.fft(state["x"]))
        if "adj" in case["calls"]:
            out.append(A.adj(state["k"]))
        return out
    if case["kind"] == "series":
        S = state["S"]
        if case["sense"]:
            image, maps, k = state["data"]
            return [S.forward_sense(image, maps), S.adjoint_sense(k, maps)]
        x, k = state["data"]
        return [S.forward(x), S.adjoint(k)]
    out = []
    for om, y in zip(state["omegas"], state["y"]):
        x = state["x"].detach().requires_grad_(True)
        om = om.detach().requires_grad_(True)
        residual = state["op"].forward(x, om) - y
        loss = (residual.real ** 2 + residual.imag ** 2).sum()
        gx, gom = torch.autograd.grad(loss, (x, om))
        out.append([loss.detach(), gx, gom])
    return out


def _samples(case):
    """Sample count of a case."""
    if case["kind"] == "gradient":
        return case["interleaves"] * case["samples"]
    if case["kind"] == "series":
        return sum(len(om) for om in _frames(case, 0))
    if case["traj"] == "spiral":
        return max(1, case["spokes"] // 8) * 8 * case["readout"]
    return case["spokes"] * case["readout"]


def work(case):
    """Images, samples and coordinates read and written once; the oversampled FFT (5 K log2 K) and the
    J^d multiply-adds of each sample and coil, per direction."""
    Nd, Kd = _ints(case["Nd"]), _ints(case["Kd"])
    M, C, d = _samples(case), case["coils"], len(Nd)
    size = 16 if case.get("precision") == "double" else 8
    N, K, F = math.prod(Nd), math.prod(Kd), case.get("frames", 1)
    taps = case["J"] ** d
    one = dict(bytes=size * C * (F * N + M) + size // 2 * d * M,
               flops=C * (F * 5 * K * math.log2(K) + 4 * taps * M))
    times = 2
    if case["kind"] == "operator":
        times = 2 if case["calls"] == "fft+adj" else 1
    if case.get("sense"):
        one["bytes"] = size * (F * N + C * N + C * M) + size // 2 * d * M
    if case["kind"] == "gradient":
        # per step: the forward, the image gradient and the trajectory gradient
        one = dict(bytes=2 * one["bytes"] + size * C * M + size * d * M, flops=3 * one["flops"])
    return dict(bytes=times * one["bytes"], flops=times * one["flops"])


# ---- the operator in 64 bits ------------------------------------------------------------------------


class _Exact:
    """The table NUFFT of one trajectory: constants in the operator's type, sums in 64 bits."""

    def __init__(self, case, omega):
        self.Nd, self.Kd, self.J = _ints(case["Nd"]), _ints(case["Kd"]), case["J"]
        self.real = np.float64 if case.get("precision") == "double" else np.float32
        self.d = len(self.Nd)
        self.mid = [n // 2 for n in self.Nd]
        omega = np.asarray(omega)
        om = omega.astype(self.real)
        tm = np.stack([(om[:, a] / (2 * np.pi / self.Kd[a])).astype(self.real) for a in range(self.d)], 1)
        self.phase = torch.from_numpy(np.exp(-1j * (omega.astype(np.float64) @ np.asarray(self.mid, np.float64)))).cuda()
        sn = np.array([1.0])
        self.cells, self.coef, self.slope = [], [], []
        points = np.arange(-self.J * L / 2.0, self.J * L / 2.0 + 1) / L
        for a in range(self.d):
            N, K = self.Nd[a], self.Kd[a]
            alpha = math.pi * math.sqrt(self.J ** 2 / (K / N) ** 2 * (K / N - 0.5) ** 2 - 0.8)
            i0a = float(np.i0(alpha))
            z = np.lib.scimath.sqrt((np.pi * self.J * (np.arange(N) - self.mid[a]) / K) ** 2 - alpha ** 2)
            sn = np.outer(sn.ravel(), 1 / np.real(self.J * np.sin(z) / z / i0a))
            s = np.sqrt(np.maximum(0, 1 - (2 * points / self.J) ** 2))
            inside = 2 * np.abs(points) < self.J
            h = np.where(inside, np.i0(alpha * s) / i0a, 0.0)
            i1 = torch.special.i1(torch.from_numpy(alpha * s)).numpy()
            ratio = np.where(s > 1e-12, i1 / np.maximum(s, 1e-300), alpha / 2)
            dh = np.where(inside, -(4 * alpha * points / self.J ** 2) * ratio / i0a, 0.0)
            t = tm[:, a].astype(np.float64)
            first = 1 + np.floor(t - self.J / 2)
            taps = first[:, None] + np.arange(self.J)
            at = (t[:, None] - taps) * L
            low = np.floor(at)
            n, f = low.astype(np.int64) + self.J * L // 2, at - low
            for table, to in ((h, self.coef), (dh, self.slope)):
                tab = np.concatenate([[0, 0], table.astype(self.real).astype(np.float64), [0, 0]])
                n2 = np.clip(n + 2, 0, len(tab) - 2)
                to.append(torch.from_numpy((1 - f) * tab[n2] + f * tab[n2 + 1]).cuda())
            self.cells.append(torch.from_numpy(np.mod(taps.astype(np.int64), K)).cuda())
        # [*reversed(Nd)], as the images lie in memory
        sn = sn.reshape(self.Nd).astype(self.real).astype(np.float64)
        self.sn = torch.from_numpy(np.ascontiguousarray(sn.transpose())).cuda()
        total = np.zeros((1,), self.real)
        for a in range(self.d):
            c = self.real(2 * np.pi / self.Kd[a] * self.mid[a])
            total = total[..., None] + (c * np.arange(self.Kd[a], dtype=self.real)).astype(self.real)
        total = total.reshape(self.Kd).astype(np.float64)
        self.before = torch.from_numpy(np.ascontiguousarray(np.exp(1j * total).transpose())).cuda()

    def _taps(self):
        """(cell, weight, weights of the derivative along each axis) for each of the J^d taps."""
        J, d = self.J, self.d
        for q in range(J ** d):
            j = [q // J ** a % J for a in range(d)]
            cell, w = 0, 1
            for a in reversed(range(d)):
                cell = cell * self.Kd[a] + self.cells[a][:, j[a]]
                w = w * self.coef[a][:, j[a]]

            def slopes(j=j):
                return [math.prod([(self.slope if b == a else self.coef)[b][:, j[b]] for b in range(d)])
                        for a in range(d)]
            yield cell, w, slopes

    def _grid(self, x):
        """[coils, *reversed(Nd)] -> [prod(Kd), coils]"""
        axes = tuple(range(1, self.d + 1))
        g = torch.fft.fftn(x.to(torch.complex128) * self.sn, s=tuple(reversed(self.Kd)), dim=axes) * self.before
        return g.reshape(x.shape[0], -1).t().contiguous()

    def forward(self, x):
        g = self._grid(x)
        y = torch.zeros((len(self.phase), x.shape[0]), dtype=torch.complex128, device="cuda")
        for cell, w, _ in self._taps():
            y += w[:, None] * g[cell]
        return (y * self.phase[:, None]).t().contiguous()

    def adjoint(self, y):
        C = y.shape[0]
        v = torch.view_as_real((y.to(torch.complex128) * self.phase.conj()).t().contiguous()).reshape(-1, 2 * C)
        g = torch.zeros((math.prod(self.Kd), 2 * C), dtype=torch.float64, device="cuda")
        for cell, w, _ in self._taps():
            g.index_add_(0, cell, v * w[:, None])
        g = torch.view_as_complex(g.reshape(-1, C, 2)).t().reshape((C,) + tuple(reversed(self.Kd)))
        g = torch.fft.ifftn(g * self.before.conj(), dim=tuple(range(1, self.d + 1))) * math.prod(self.Kd)
        return (g[(slice(None),) + tuple(slice(0, n) for n in reversed(self.Nd))] * self.sn).contiguous()

    def slope_products(self, x, y, gy):
        """[M, ndim]: sum over coils of Re(conj(gy) dy / d omega), y = forward(x)."""
        g = self._grid(x)
        cols = [torch.zeros((len(self.phase), x.shape[0]), dtype=torch.complex128, device="cuda") for _ in self.Nd]
        for cell, _, slopes in self._taps():
            v = g[cell]
            for col, w in zip(cols, slopes()):
                col += w[:, None] * v
        out = []
        for a, col in enumerate(cols):
            dy = (col * self.phase[:, None]).t() * (self.Kd[a] / (2 * np.pi)) - 1j * self.mid[a] * y
            out.append((gy.conj() * dy).real.sum(0))
        return torch.stack(out, 1)


def exact(case, seed):
    if case["kind"] == "operator":
        om = _trajectory(case, seed)
        A = _Exact(case, om)
        x, k = _data(case, seed, len(om))
        out = []
        if "fft" in case["calls"]:
            y = A.forward(x).t()
            out.append(y[..., 0] if case["coils"] == 1 else y)
        if "adj" in case["calls"]:
            xa = A.adjoint(k)
            xa = xa.permute(*reversed(range(xa.dim())))
            out.append(xa[..., 0] if case["coils"] == 1 else xa)
        return out
    if case["kind"] == "series":
        frames = _frames(case, seed)
        ends = np.cumsum([len(om) for om in frames])
        data, C = _data(case, seed, int(ends[-1])), case["coils"]
        ys, xs = [], []
        for f, om in enumerate(frames):
            A = _Exact(case, om)
            k = data[-1][C * int(ends[f] - len(om)):C * int(ends[f])].reshape(C, len(om))
            if case["sense"]:
                maps = data[1].to(torch.complex128)
                ys.append(A.forward(maps * data[0][f]).reshape(-1))
                xs.append((maps.conj() * A.adjoint(k)).sum(0))
            else:
                ys.append(A.forward(data[0][f]).reshape(-1))
                xs.append(A.adjoint(k))
        return [torch.cat(ys), torch.stack(xs)]
    om = _trajectory(case, seed)
    x, y = _data(case, seed, len(om))
    turned = x.permute(0, *reversed(range(1, x.dim())))
    out = []
    for o, measured in zip(_moved(om), y):
        A = _Exact(case, o.astype(np.float32))
        predicted = A.forward(turned)
        r = predicted - measured.to(torch.complex128)
        gx = 2 * A.adjoint(r)
        out.append([(r.real ** 2 + r.imag ** 2).sum(), gx.permute(0, *reversed(range(1, gx.dim()))),
                    A.slope_products(turned, predicted, 2 * r)])
    return out
