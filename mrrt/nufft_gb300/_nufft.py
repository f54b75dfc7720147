"""``NufftBase``: drop-in for the reference operator, running on the GB300.

Same constructor signature, ``.fft()`` / ``.adj()`` methods and attributes
as the reference (mrrt/nufft/_nufft.py:122-621).  Plan-time math (kernel
shape, deapodisation ``sn``, tables ``h``, normalised coordinates ``tm`` and
``phase_after``) is computed on the host exactly as the reference computes it
(same formulas, same numpy dtypes, so the float32 rounding of the phases
follows the reference); the transforms run in libgbnufft's CUDA kernels.
There is no CPU execution path.

Input and output conventions follow the reference (mrrt/nufft/_nufft.py:
1275-1397, 1459-1578): images are ``Nd + (reps,)`` in Fortran order
(``order='F'``) or ``(reps,) + Nd`` (``order='C'``); sample arrays are
``(M, reps)`` / ``(reps, M)``; a single repetition is squeezed; real input is
promoted to the operator's complex dtype and the output dtype always equals
the operator precision.  ``on_gpu=False`` returns numpy arrays (host buffers,
copies inside the call); ``on_gpu=True`` returns torch CUDA tensors.  Inputs
may be numpy arrays or torch tensors in either case.
"""
import math
import warnings

import numpy as np
import torch

from ._kaiser_bessel import kaiser_bessel_ft
from ._kernels import BeattyKernel, kernel_deriv_table, kernel_table
from . import _lib
from ._plan import GpuPlan, raw_stream, require_cuda

__all__ = ["NufftBase"]

supported_real_types = [np.float32, np.float64]


def _as_tuple(seq, type=int, n=None):
    if np.isscalar(seq):
        if n is None:
            raise ValueError("for scalar, seq, n must be specified")
        return (type(seq),) * n
    if n is not None and len(seq) != n:
        raise ValueError("array did not have the expected size of {}".format(n))
    return tuple(type(s) for s in seq)


def _to_numpy(a):
    if isinstance(a, torch.Tensor):
        return a.detach().cpu().numpy()
    return np.asarray(a)


def deapodisation(Nd, Kd, Jd, n_mid, alpha, rdt):
    """Scaling factors ``sn`` (mrrt/nufft/_nufft.py:726-748): the float64 outer
    product of 1 / KB-transform per axis, cast to the operator's real dtype,
    Fortran order."""
    sn = np.array([1.0])
    for d in range(len(Nd)):
        nc = np.arange(-n_mid[d], -n_mid[d] + Nd[d])
        tmp = 1 / kaiser_bessel_ft(nc / Kd[d], Jd[d], alpha[d], 0, 1)
        sn = np.outer(sn.ravel(), tmp.conj())
    return np.asfortranarray(sn.reshape(tuple(Nd)).astype(rdt))


def sample_phase_of(omega, n_shift, n_mid, phasing, rdt, cdt):
    """Per-sample phase (mrrt/nufft/_nufft.py:717-724, 898-903): phase_after =
    exp(i omega . (n_shift - n_mid)) for real phasing (omega in its given
    dtype, the shift vector in the operator's real dtype); for complex phasing
    exp(i omega . n_shift) when the shift is non-zero, else None."""
    if phasing == "real":
        shift_vec = [(s - m) for s, m in zip(n_shift, n_mid)]
        return np.exp(1j * np.dot(omega, np.asarray(shift_vec, dtype=rdt))).astype(cdt, copy=False)
    if any(s != 0 for s in n_shift):
        return np.exp(1j * np.dot(omega.astype(rdt), np.asarray(n_shift))).astype(cdt)
    return None


def normalised_coordinates(omega, Kd, rdt):
    """tm = omega / (2 pi / K_d) in the operator's real dtype
    (mrrt/nufft/_nufft.py:1012-1016)."""
    omega = np.asarray(omega, dtype=rdt)
    tm = np.zeros_like(omega)
    for d in range(omega.shape[1]):
        gam = 2 * np.pi / Kd[d]
        tm[:, d] = omega[:, d] / gam
    return tm


def sparse_weights(omega, Nd, Jd, Kd, kernel, phasing, rdt):
    """Per-axis factors of the reference's sparse interpolation matrix
    (``_init_sparsemat``, mrrt/nufft/_nufft.py:750-877, with ``_nufft_offset``
    and ``_nufft_coef``, mrrt/nufft/_utils.py:20-86): for sample m and tap j
    of axis d, ``u = kernel_d(dk_m - (j + 1))`` with
    ``dk = om / gam - floor(om / gam - J / 2)`` (om in the operator's real
    dtype), times ``exp(i gam (N - 1) / 2 * arg)`` for complex phasing.  The
    matrix entry is the conjugate of the product over axes, so the factors
    are returned conjugated.  Returns ``(w_re, w_im)``: lists of
    ``[M, J_d]`` arrays (``w_im`` None for real phasing)."""
    w_re, w_im = [], []
    for d in range(len(Nd)):
        J, K, N = Jd[d], Kd[d], Nd[d]
        om = omega[:, d]
        gam = 2 * np.pi / K
        koff = np.floor(om / gam - J / 2.0)
        dk = om / gam - koff
        arg = -np.arange(1, J + 1)[:, None] + dk[None, :]      # [J, M]
        c = kernel.kernels[d](arg)
        if phasing == "complex":
            u = np.conj(np.exp(1j * gam * (N - 1) / 2.0 * arg) * c)
            w_re.append(np.ascontiguousarray(u.real.T, dtype=rdt))
            w_im.append(np.ascontiguousarray(u.imag.T, dtype=rdt))
        else:
            w_re.append(np.ascontiguousarray(np.asarray(c).real.T, dtype=rdt))
    return w_re, (w_im if phasing == "complex" else None)


class NufftBase(object):
    """Non-uniform FFT operator (table-based interpolation) on the GPU.

    Parameters are those of the reference ``NufftBase``; see the module
    docstring for the data conventions.  ``mode`` is ``'table'`` or
    ``'sparse'`` (the reference's exact Kaiser-Bessel interpolation weights,
    applied by the same kernels).

    Extra keywords (not in the reference): ``max_coils`` -- the repetition
    count the tile plan is sized for (default 1).  Any batch size works; a
    batch wider than the tiles were sized for runs in more coil chunks.
    ``tile`` / ``stile`` -- gather / spread tile edges per axis (default: the
    planner's choice; ``autotune.tune_operator`` measures the best).
    """

    def __init__(self, Nd, omega, Jd=4, Kd=None, precision="single", mode="table", Ld=1024,
                 ortho=False, n_shift=None, phasing="real", adjoint_scalefactor=1.0,
                 preplan_cufft=True, order="F", verbose=False, on_gpu=False, max_coils=1,
                 tile=None, stile=None):
        require_cuda()
        # the constructor's arguments, kept so that a pickled operator is
        # rebuilt (replanned on the GPU) on load; the reference's operator is
        # picklable (mrrt/nufft/_nufft.py:405-407)
        self._init_args = dict(
            Nd=Nd, omega=np.array(_to_numpy(omega), copy=True), Jd=Jd, Kd=Kd, precision=precision,
            mode=mode, Ld=Ld, ortho=ortho, n_shift=n_shift, phasing=phasing,
            adjoint_scalefactor=adjoint_scalefactor, preplan_cufft=preplan_cufft, order=order,
            verbose=verbose, on_gpu=on_gpu, max_coils=max_coils, tile=tile, stile=stile)
        self.verbose = verbose
        self.order = order
        if order not in ("F", "C"):
            raise ValueError("order must be 'F' or 'C'")
        self.on_gpu = on_gpu
        # the reference's attribute: the interpolation matrix format in
        # sparse mode (mrrt/nufft/_nufft.py:319-323), None in table mode
        self.__sparse_format = "CSC" if mode == "sparse" else None
        if np.isscalar(Nd):
            Nd = (Nd,)
        self.__Nd = _as_tuple(Nd, type=int)
        self.ndim = len(self.__Nd)
        if self.ndim > 3:
            raise NotImplementedError("dimensions > 3 not implemented")
        if phasing not in ("real", "complex"):
            raise ValueError("Invalid phasing: {}. phasing must be 'real' or 'complex'".format(phasing))
        self.__phasing = phasing
        self.__Jd = _as_tuple(Jd, type=int, n=self.ndim)
        if Kd is None:
            Kd = tuple(int(1.5 * n) for n in self.__Nd)
        self.__Kd = _as_tuple(Kd, type=int, n=self.ndim)
        self.ortho = ortho
        self.scale_ortho = math.sqrt(math.prod(self.__Kd)) if ortho else 1
        if mode not in ("table", "sparse"):
            raise ValueError("Invalid NUFFT mode: {}".format(mode))
        self.__mode = mode
        self.adjoint_scalefactor = adjoint_scalefactor
        self.preplan_cufft = preplan_cufft
        self._p = None
        self.__Ld = int(Ld)
        if self.__Ld % 2 == 1 and any(j % 2 == 1 for j in self.__Jd):
            warnings.warn("accuracy may be compromised when L and J are both odd")

        # omega validation (mrrt/nufft/_nufft.py:552-573)
        omega = _to_numpy(omega)
        if omega.ndim == 1:
            omega = omega[:, np.newaxis]
        if omega.shape[1] != self.ndim:
            raise ValueError("number of cols must match NUFFT dimension")
        if omega.dtype not in supported_real_types:
            raise ValueError("omega must be one of the following types: {}".format(supported_real_types))
        if precision == "auto":
            precision = "single" if omega.dtype == np.float32 else "double"
        if precision == "single":
            self._cplx_dtype, self._real_dtype = np.dtype(np.complex64), np.dtype(np.float32)
        elif precision == "double":
            self._cplx_dtype, self._real_dtype = np.dtype(np.complex128), np.dtype(np.float64)
        else:
            raise ValueError("precision must be 'single', 'double' or 'auto'")
        self.__precision = precision

        if n_shift is None:
            self.__n_shift = (0.0,) * self.ndim
        else:
            self.__n_shift = _as_tuple(n_shift, type=float, n=self.ndim)
        if phasing == "real":
            self.n_mid = tuple(n // 2 for n in self.__Nd)
        else:
            self.n_mid = tuple((n - 1) / 2.0 for n in self.__Nd)

        self.kernel = BeattyKernel(shape=self.__Jd, grid_shape=self.__Nd, os_grid_shape=self.__Kd)
        rdt, cdt = self._real_dtype, self._cplx_dtype
        self.sn = deapodisation(self.__Nd, self.__Kd, self.__Jd, self.n_mid, self.kernel.alpha, rdt)
        if phasing == "real":
            self.phase_after = sample_phase_of(omega, self.__n_shift, self.n_mid, "real", rdt, cdt)
            self.phase_shift = None
            sample_phase = self.phase_after
        else:
            self.phase_after = None
            self.phase_shift = sample_phase_of(omega, self.__n_shift, self.n_mid, "complex", rdt, cdt)
            sample_phase = self.phase_shift
        self.__omega = np.asfortranarray(omega.astype(rdt))
        self.M = self.__omega.shape[0]
        self.tm = normalised_coordinates(self.__omega, self.__Kd, rdt)
        tdt = cdt if phasing == "complex" else rdt
        self.h = [kernel_table(self.__Nd[d], self.__Jd[d], self.__Kd[d], self.__Ld, phasing, tdt)
                  for d in range(self.ndim)]
        self.nargin1 = math.prod(self.__Nd)
        self.nargout1 = self.M
        self._phase_before = None
        # phase_before(k) = exp(i sum_d c_d k_d), c_d = 2 pi n_mid_d / K_d
        pb_coef = [2 * np.pi / self.__Kd[d] * self.n_mid[d] for d in range(self.ndim)]
        self._plan = GpuPlan(
            self.__Nd, self.__Kd, self.__Jd, self.__Ld, rdt,
            [np.real(h) for h in self.h],
            [np.imag(h) for h in self.h] if phasing == "complex" else None,
            self.sn.ravel(order="F"), np.ascontiguousarray(self.tm), sample_phase,
            ortho=ortho, adjoint_scale=adjoint_scalefactor, pb_coef=pb_coef,
            pb_order=list(range(self.ndim)), phasing=phasing, max_coils=max_coils,
            tile=tile, stile=stile)
        # per direction: input axes, their Fortran-order strides, values per
        # repetition, the same of the output
        strides = [math.prod(self.__Nd[:d]) for d in range(self.ndim)]
        image, samples = (self.__Nd, tuple(strides), self.nargin1), ((self.M,), (1,), self.M)
        self._direct = {True: image + samples, False: samples + image}
        self._p = None
        if mode == "sparse":
            self._weights = sparse_weights(self.__omega, self.__Nd, self.__Jd, self.__Kd, self.kernel,
                                           phasing, rdt)
            self._plan.set_weights(*self._weights)

    # ------------------------------------------------------------------ props
    @property
    def on_gpu(self):
        """bool: results are returned as torch CUDA tensors (True) or numpy
        arrays (False); the transforms always run on the GPU."""
        return self.__on_gpu

    @on_gpu.setter
    def on_gpu(self, on_gpu):
        if on_gpu in [True, False]:
            self.__on_gpu = bool(on_gpu)
        else:
            raise ValueError("on_gpu must be True or False")

    @property
    def sparse_format(self):
        """str: internal sparse matrix format (``'CSC'`` when ``mode=='sparse'``)."""
        return self.__sparse_format

    @property
    def Nd(self):
        return self.__Nd

    @property
    def Kd(self):
        return self.__Kd

    @property
    def Jd(self):
        return self.__Jd

    @property
    def Ld(self):
        return self.__Ld

    @property
    def mode(self):
        return self.__mode

    @property
    def phasing(self):
        return self.__phasing

    @property
    def precision(self):
        return self.__precision

    @property
    def n_shift(self):
        return self.__n_shift

    @property
    def omega(self):
        return self.__omega

    @property
    def xp(self):
        return torch if self.on_gpu else np

    @property
    def plan(self):
        """The underlying :class:`GpuPlan` (memory-axis order = reference axis order)."""
        return self._plan

    @property
    def p(self):
        """Sparse mode: the interpolation matrix [M, prod(Kd)] as a scipy CSC
        matrix on the host (the reference's ``self.p``), built on first
        access from the uploaded weights; None in table mode.  The GPU path
        never uses it."""
        if self.__mode != "sparse":
            return None
        if self._p is None:
            import scipy.sparse

            w_re, w_im = self._weights
            M = self.M
            rows = np.arange(M)
            kk = np.zeros((M, 1), dtype=np.int64)
            uu = np.ones((M, 1), dtype=self._cplx_dtype if w_im is not None else self._real_dtype)
            stride = 1
            for d in range(self.ndim):
                J, K = self.__Jd[d], self.__Kd[d]
                gam = 2 * np.pi / K
                koff = np.floor(self.__omega[:, d] / gam - J / 2.0).astype(np.int64)
                kd = np.mod(koff[:, None] + np.arange(1, J + 1)[None, :], K) * stride
                wd = w_re[d] if w_im is None else w_re[d] + 1j * w_im[d]
                kk = (kk[:, :, None] + kd[:, None, :]).reshape(M, -1, order="F")
                uu = (uu[:, :, None] * wd[:, None, :]).reshape(M, -1, order="F")
                stride *= K
            if self.__phasing == "complex" and self.phase_shift is not None:
                # the reference folds the n_shift phase into the rows
                # (_nufft.py:836-844); the GPU applies it as the sample phase
                uu = uu * self.phase_shift[:, None]
            mm = np.repeat(rows[:, None], kk.shape[1], axis=1)
            self._p = scipy.sparse.coo_matrix((uu.ravel(), (mm.ravel(), kk.ravel())),
                                              shape=(M, int(np.prod(self.__Kd)))).tocsc()
        return self._p

    @property
    def phase_before(self):
        """Kd-grid phase exp(i sum_d 2 pi n_mid_d k_d / K_d) as the reference
        builds it (mrrt/nufft/_nufft.py:703-715); computed on first access."""
        if self.__phasing != "real":
            return None
        if self._phase_before is None:
            rdt = self._real_dtype
            ph = (2 * np.pi / self.__Kd[0] * self.n_mid[0]) * np.arange(self.__Kd[0], dtype=rdt)
            for d in range(1, self.ndim):
                tmp = (2 * np.pi / self.__Kd[d] * self.n_mid[d]) * np.arange(self.__Kd[d], dtype=rdt)
                ph = ph.reshape(ph.shape + (1,)) + tmp.reshape((1,) * d + (tmp.size,))
            self._phase_before = np.exp(1j * ph).astype(self._cplx_dtype, copy=False)
        return self._phase_before

    def kernel_deriv_tables(self):
        """Derivative tables dh/dt per axis (phasing 'real'), for the trajectory gradient."""
        return [kernel_deriv_table(self.__Nd[d], self.__Jd[d], self.__Kd[d], self.__Ld, self._real_dtype)
                for d in range(self.ndim)]

    # ------------------------------------------------------------- transforms
    def _device_in(self, a, narg, leading_shape):
        """Return (tensor [reps, *reversed(leading_shape)] contiguous on the
        plan device, reps).  ``a`` follows the Fortran-order convention
        leading_shape + (reps,)."""
        dev = self._plan.device
        ct = self._plan.ctype
        if isinstance(a, torch.Tensor):
            t = a.detach()
            if not t.is_complex():
                t = t.to(torch.float64 if self._real_dtype == np.float64 else torch.float32)
            t = t.to(device=dev, dtype=ct).resolve_conj().resolve_neg()
        else:
            arr = np.asarray(a)
            if arr.dtype != self._cplx_dtype:
                arr = arr.astype(self._cplx_dtype)
            t = None
        total = (t.numel() if t is not None else arr.size)
        if narg == 0:
            # empty sample set: repetitions come from the trailing axis, if any
            shp = tuple(t.shape) if t is not None else arr.shape
            if total != 0:
                raise ValueError("Input signal has the wrong size.")
            reps = int(shp[-1]) if len(shp) == 2 else 1
        elif total % narg != 0:
            raise ValueError("Input signal has the wrong size.")
        else:
            reps = total // narg
        if reps < 1:
            raise ValueError("Input signal has the wrong size.")
        full = tuple(leading_shape) + (reps,)
        if t is not None:
            t = t.reshape(full) if t.dim() != len(full) or tuple(t.shape) != full else t
            t = t.permute(*reversed(range(len(full)))).contiguous()
        else:
            arr = np.asfortranarray(arr.reshape(full, order="F") if arr.shape != full else arr)
            # one host-to-device copy straight from the caller's memory (no
            # pinned staging copy: host memory is directly reachable by the
            # copy engines at full speed on Grace-Blackwell, and arrays this
            # operator returned are pinned already)
            host = torch.from_numpy(arr.ravel(order="F"))
            # asynchronous only when the call ends with a stream synchronisation
            # (host outputs), so the caller may reuse its array on return
            t = host.to(dev, non_blocking=not self.on_gpu).reshape(tuple(reversed(full)))
        return t, reps

    def _device_out(self, t, reps, leading_shape):
        """Convert a device tensor [reps, *reversed(leading_shape)] to the
        Fortran-order result leading_shape + (reps,) (squeezed for reps == 1)."""
        nd = len(leading_shape) + 1
        if self.on_gpu:
            out = t.permute(*reversed(range(nd)))
        else:
            # pinned result buffer from torch's caching host allocator: no
            # first-touch page faults on a fresh allocation, full-speed copy;
            # the returned array keeps the buffer alive
            host = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
            host.copy_(t, non_blocking=True)
            torch.cuda.current_stream(t.device).synchronize()
            out = host.numpy().transpose(tuple(reversed(range(nd))))
        if reps == 1:
            out = out[..., 0]
        return out

    def _swap_reps(self, x, narg):
        size = x.numel() if isinstance(x, torch.Tensor) else np.size(x)
        if size != narg:
            nd = x.dim() if isinstance(x, torch.Tensor) else np.ndim(x)
            perm = tuple(range(1, nd)) + (0,)
            x = x.permute(*perm) if isinstance(x, torch.Tensor) else np.transpose(x, perm)
        return x

    def _unswap_reps(self, x, narg):
        size = x.numel() if isinstance(x, torch.Tensor) else np.size(x)
        if size != narg:
            nd = x.dim() if isinstance(x, torch.Tensor) else np.ndim(x)
            perm = (nd - 1,) + tuple(range(nd - 1))
            x = x.permute(*perm) if isinstance(x, torch.Tensor) else np.transpose(x, perm)
        return x

    # -------------------------------------- host arrays: pipelined by coil chunk
    def _host_transform(self, a, forward):
        """Host numpy in, host numpy out, through the library's host-buffer
        entry points: one call copies in, transforms and copies out (large
        batches as a copy / transform pipeline of coil chunks).  The result
        lands in pinned memory from torch's caching host allocator, so the
        copy out runs at the link's rate.  Returns None for inputs this path
        does not take (device tensors, on_gpu operators, graph capture, sizes
        that do not divide); the caller's one-piece path then applies and
        raises the reference's errors."""
        if self.on_gpu or not isinstance(a, np.ndarray) or torch.cuda.is_current_stream_capturing():
            return None
        narg = self.nargin1 if forward else self.M
        lead = self.__Nd if forward else (self.M,)
        out_lead = (self.M,) if forward else self.__Nd
        if narg == 0 or a.size == 0 or a.size % narg:
            return None
        reps = a.size // narg
        arr = a if a.dtype == self._cplx_dtype else a.astype(self._cplx_dtype)
        full = tuple(lead) + (reps,)
        arr = np.asfortranarray(arr.reshape(full, order="F") if arr.shape != full else arr)
        host_in = torch.from_numpy(arr.reshape(-1, order="F"))
        host_out = torch.empty((reps,) + tuple(reversed(out_lead)), dtype=self._plan.ctype, pin_memory=True)
        if forward:
            self._plan.forward_host(host_in, host_out, reps)
        else:
            self._plan.adjoint_host(host_in, host_out, reps)
        nd = len(out_lead) + 1
        out = host_out.numpy().transpose(tuple(reversed(range(nd))))
        return out[..., 0] if reps == 1 else out

    def _device_direct(self, a, forward):
        """A device tensor already in the plan's precision and memory order,
        Fortran-order ``lead + (reps,)`` or ``lead`` -- what ``fft`` and
        ``adj`` of an ``on_gpu`` operator return, say: the library is called on
        it as it lies, without the general path's conversions and views (which
        took 30 of the 50 us of a small call).  Returns None for anything
        else."""
        plan = self._plan
        if type(a) is not torch.Tensor or a.dtype is not plan.ctype or a.device != plan.device or \
                not self.__on_gpu or self.order != "F" or a.is_conj() or a.is_neg():
            return None
        lead, strides, n, out_lead, out_strides, m = self._direct[forward]
        nd = len(lead)
        shape = a.shape
        if n == 0 or shape[:nd] != lead:
            return None
        if len(shape) == nd:
            reps = 1
            if a.stride() != strides:
                return None
        elif len(shape) == nd + 1:
            reps = shape[nd]
            if reps < 1 or a.stride() != strides + (n,):
                return None
        else:
            return None
        if reps > 1:
            out_lead, out_strides = out_lead + (reps,), out_strides + (m,)
        out = torch.empty_strided(out_lead, out_strides, dtype=plan.ctype, device=plan.device)
        call = plan.lib.gbn_forward if forward else plan.lib.gbn_adjoint
        rc = call(plan.handle, a.data_ptr(), out.data_ptr(), reps, raw_stream(plan.device.index))
        if rc:
            _lib.check_with(plan.lib, rc)
        return out

    def fft(self, x):
        """Forward NUFFT (uniform image -> non-uniform samples)."""
        out = self._device_direct(x, True)
        if out is not None:
            return out
        if self.order == "C":
            x = self._swap_reps(x, self.nargin1)
        out = self._host_transform(x, True)
        if out is not None:
            return self._unswap_reps(out, self.nargout1) if self.order == "C" else out
        xt, reps = self._device_in(x, self.nargin1, self.__Nd)
        y = torch.empty((reps, self.M), dtype=self._plan.ctype, device=self._plan.device)
        self._plan.forward(xt, y, reps)
        out = self._device_out(y, reps, (self.M,))
        if self.order == "C":
            out = self._unswap_reps(out, self.nargout1)
        return out

    def adj(self, k):
        """Adjoint NUFFT (non-uniform samples -> uniform image)."""
        out = self._device_direct(k, False)
        if out is not None:
            return out
        if self.order == "C":
            k = self._swap_reps(k, self.nargout1)
        out = self._host_transform(k, False)
        if out is not None:
            return self._unswap_reps(out, self.nargin1) if self.order == "C" else out
        yt, reps = self._device_in(k, self.M, (self.M,))
        x = torch.empty((reps,) + tuple(reversed(self.__Nd)), dtype=self._plan.ctype,
                        device=self._plan.device)
        self._plan.adjoint(yt, x, reps)
        out = self._device_out(x, reps, self.__Nd)
        if self.order == "C":
            out = self._unswap_reps(out, self.nargin1)
        return out

    # ------------------------------------------- table interpolation alone
    def interp_table(self, xk):
        """Table interpolation only (the reference's ``_nufft_table_interp``
        without its phase_shift, mrrt/nufft/_nufft.py:998-1097): oversampled
        grid ``[prod(Kd), reps]`` (Fortran order) -> samples ``[M, reps]``."""
        gt, reps = self._device_in(xk, math.prod(self.__Kd), self.__Kd)
        y = torch.empty((reps, self.M), dtype=self._plan.ctype, device=self._plan.device)
        self._plan.interp_forward(gt, y, reps)
        return self._device_out(y, reps, (self.M,))

    def interp_table_adj(self, xm):
        """Adjoint table interpolation only (``_nufft_table_adj`` without its
        phase, mrrt/nufft/_nufft.py:1101-1191): samples ``[M, reps]`` ->
        oversampled grid ``[*Kd, reps]`` (Fortran order)."""
        yt, reps = self._device_in(xm, self.M, (self.M,))
        g = torch.empty((reps,) + tuple(reversed(self.__Kd)), dtype=self._plan.ctype,
                        device=self._plan.device)
        self._plan.interp_adjoint(yt, g, reps)
        return self._device_out(g, reps, self.__Kd)

    def __getstate__(self):
        """Pickle the constructor's arguments (not the GPU state); loading
        rebuilds the plan on the current CUDA device."""
        state = dict(self._init_args)
        state["on_gpu"] = self.on_gpu
        return state

    def __setstate__(self, state):
        self.__init__(**state)
