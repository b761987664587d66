"""Differentiable forms of the operator chain for torch.autograd.

Each operator is a ``torch.autograd.Function`` whose backward pass is the
hand-written adjoint kernel (PyTorch's convention for a complex-linear map is
that the backward of ``y = A x`` is ``A^H grad_y``; for a real input ``p`` of
a complex output it is ``Re <grad_y, dy/dp>``):

* ``radon(obj, tomo)``: ``R obj`` (tomo.py:56-86); backward ``R^T``
  (``ht_tomo_RT``, tomo.py:88-116);
* ``shift(psi, pos, mag, sh)``: ``S(coeff(psi); pos, mag)`` (shift.py:128-132);
  backward for ``psi``: ``coeff(S^T g)``, for ``pos``: the position
  derivative ``Re <g, dS/dpos>`` -- both from ``ht_shift_dSadj``
  (shift.py:185-204) -- the prefilter being self-adjoint;
* ``propagate(psi, j, prop)``: ``D_j psi`` (propagation.py:70-89); backward
  ``D_j^T`` (``ht_prop_DT``, propagation.py:91-112).

``DataFidelity`` composes them (with the probe product, whose gradient sum
over angles is taken in complex128) into the BH data term
(rec_mpi.py:517-813): ``F = 1/N sum (|D_k(prb_k exp(i S_k(coeff(R obj))))| - d)^2``
over (angle, distance) images, optionally in angle chunks whose forward is
recomputed in the backward pass, so that only one chunk's intermediates are held
at a time.  Where the fused cascade takes the inputs (``_use_fused``) a chunk is
one function, ``ht_rec_forward`` and ``ht_rec_gradient`` in its backward pass
(256^2 x 90 angles x 4 distances, value and gradients: 4.7 ms against 11.0
operator by operator); else the operators are composed, with
``torch.utils.checkpoint``.

The backward passes are library calls, which autograd does not see into: the
operators and the data term are differentiable once, and a derivative of their
gradients is refused.
"""
import contextlib
import ctypes

import numpy as np
import torch
from torch.autograd.function import once_differentiable
from torch.utils.checkpoint import checkpoint

from . import _lib
from .propagation import Propagation
from .shift import Shift
from .tomo import Tomo


class _Radon(torch.autograd.Function):
    @staticmethod
    def forward(ctx, obj, tomo):
        ctx.tomo = tomo
        return tomo.R(obj.contiguous())

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        return ctx.tomo.RT(g.contiguous()), None


class _Shift(torch.autograd.Function):
    @staticmethod
    def forward(ctx, psi, pos, mag, sh):
        c = sh.coeff(psi.contiguous())
        ctx.sh = sh
        ctx.save_for_backward(c, pos, mag)
        return sh.S(c, pos, mag)

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        c, pos, mag = ctx.saved_tensors
        sh = ctx.sh
        gc, gpos = sh.dcurlySadjc(c, pos, mag, g.contiguous())
        gpsi = sh.coeff(gc) if ctx.needs_input_grad[0] else None
        return gpsi, (gpos.to(pos.dtype) if ctx.needs_input_grad[1] else None), None, None


class _Propagate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, psi, j, prop):
        ctx.prop, ctx.j = prop, j
        return prop.D(psi.contiguous(), j)

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        return ctx.prop.DT(g.contiguous(), ctx.j), None, None


class _ProbeMul(torch.autograd.Function):
    """prb [nz, n] times x12 [B, nz, n]; the probe gradient, a sum over the B
    angles, is accumulated in complex128 (as the fused cascade's is)."""

    @staticmethod
    def forward(ctx, prb, x12):
        ctx.save_for_backward(prb, x12)
        return prb.unsqueeze(0) * x12

    @staticmethod
    def backward(ctx, g):
        prb, x12 = ctx.saved_tensors
        gprb = gx = None
        if ctx.needs_input_grad[0]:
            gprb = torch.sum((g * x12.conj()).to(torch.complex128), dim=0).to(prb.dtype)
        if ctx.needs_input_grad[1]:
            gx = g * prb.conj().unsqueeze(0)
        return gprb, gx


class _Cascade:
    """The fused cascade of one angle chunk, over the operators that the data term
    has at the time of the call: F and the gradients come from handles that live
    for a call, in workspaces of torch's allocator."""

    def __init__(self, term, ntheta, tomo):
        self.sh, self.prop, self.tomo = term.sh, term.prop, tomo
        self.data_size = term.data_size
        self.sizes = (term.n, term.nz, term.nobj, term.nzobj, ntheta, term.ndist,
                      int(term.sh.obj_dtype == "complex64"))
        self.bytes = term._workspace_bytes

    def coeff(self, x):
        return self.sh.coeff(x if self.tomo is None else self.tomo.R(x.contiguous()))

    @contextlib.contextmanager
    def handle(self, forward_only=False):
        with torch.cuda.device(self.sh.device):
            key = self.sizes + (int(forward_only),)
            size = self.bytes.get(key)
            if size is None:
                out = ctypes.c_size_t()
                _lib.call("ht_rec_workspace_bytes", *self.sizes, self.prop._h, key[-1], ctypes.byref(out))
                size = self.bytes[key] = out.value
            work, h = torch.empty(size, dtype=torch.uint8, device=self.sh.device), ctypes.c_void_p()
            _lib.call("ht_rec_create_in", *self.sizes, self.prop._h, key[-1], _lib.ptr(work), size,
                      float(self.data_size), 1, ctypes.byref(h))   # 1: torch.abs has gradient 0 at 0
            try:
                yield h
            finally:
                _lib.lib().ht_rec_destroy(h)


class _ChunkMisfit(torch.autograd.Function):
    """1/N sum (|D_k(prb_k exp(i S_k(coeff(x))))| - d)^2 of one angle chunk by the
    fused cascade (ht_rec_forward; ht_rec_gradient in the backward pass, which
    repeats the forward from the saved inputs, so that no image stack is held
    between the two).  x is the chunk's projections, or the object where the
    cascade has a Radon transform."""

    @staticmethod
    def forward(ctx, x, prb, pos, mag, data, cascade):
        ctx.cascade = cascade
        ctx.save_for_backward(x, prb, pos, mag, data)
        c = cascade.coeff(x)
        f = torch.empty((), dtype=torch.float64, device=x.device)
        with cascade.handle(forward_only=True) as h:
            _lib.call("ht_rec_forward", h, _lib.ptr(c), _lib.ptr(pos), _lib.ptr(mag), _lib.ptr(prb), _lib.ptr(data),
                      None, _lib.ptr(f), _lib.stream_ptr())
        return (f / cascade.data_size).to(torch.float32)

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        x, prb, pos, mag, data = (t.contiguous() for t in ctx.saved_tensors)   # as a hook may not leave them
        cascade = ctx.cascade
        c = cascade.coeff(x)
        gc, gpos, gprb = torch.empty_like(c), torch.empty_like(pos), torch.empty_like(prb)
        with cascade.handle() as h:
            _lib.call("ht_rec_gradient", h, _lib.ptr(c), _lib.ptr(pos), _lib.ptr(mag), _lib.ptr(prb),
                      _lib.ptr(data), _lib.ptr(gc), _lib.ptr(gpos), _lib.ptr(gprb), None, 1.0, 1.0, 0,
                      _lib.stream_ptr())
        del c
        gx = None
        if ctx.needs_input_grad[0]:
            gx = cascade.sh.coeff(gc.mul_(g))   # scaled where the array is smallest
            del gc
            gx = gx if cascade.tomo is None else cascade.tomo.RT(gx)
        return (gx, gprb * g if ctx.needs_input_grad[1] else None, gpos * g if ctx.needs_input_grad[2] else None,
                None, None, None)


def radon(obj, tomo):
    """R obj for obj [nz, n, n] complex64 -> [ntheta, nz, n]."""
    return _Radon.apply(obj, tomo)


def shift(psi, pos, mag, sh):
    """S(coeff(psi)) for psi [B, nzpsi, npsi], pos [B, 2] (y, x), mag [B]."""
    return _Shift.apply(psi, pos, mag, sh)


def propagate(psi, j, prop):
    """D_j psi for psi [B, nz, n]."""
    return _Propagate.apply(psi, j, prop)


class DataFidelity(torch.nn.Module):
    """The BH data term as a differentiable function of (obj or proj, prb, pos).

    Sizes as for Rec: object [nzobj, nobj, nobj], detector [nz, n], angles
    ``theta``, ``ndist`` distances (metres), probe [ndist, nz, n], positions
    [ntheta, ndist, 2] (y, x) and magnifications [ntheta, ndist].  With
    ``chunk`` the angles are processed ``chunk`` at a time and each chunk's
    forward is recomputed during the backward pass.  Its Radon transforms own one
    workspace each, so one DataFidelity serves one stream at a time."""

    FUSED_ROWS = (32, 64, 128, 256, 384, 512, 768, 1024, 2048)   # detector row lengths of the fused cascade

    def __init__(self, sh, prop, theta, mask_r, nobj, nzobj, chunk=None):
        super().__init__()
        theta = np.asarray(theta.cpu() if isinstance(theta, torch.Tensor) else theta, dtype="float32")
        self.n, self.nz, self.ndist = prop.n, prop.nz, prop.ndist
        self.nobj, self.nzobj = nobj, nzobj
        self.ntheta = len(theta)
        self.data_size = self.ntheta * self.ndist * self.nz * self.n
        self.chunk = chunk or self.ntheta
        self.bounds = [(a, min(a + self.chunk, self.ntheta)) for a in range(0, self.ntheta, self.chunk)]
        self.tomos = [Tomo(nobj, nzobj, theta[a:b], mask_r, norm_ntheta=self.ntheta) for a, b in self.bounds]
        self.sh, self.prop = sh, prop
        self._workspace_bytes = {}   # of the fused cascade, by its sizes

    @classmethod
    def create(cls, n, nz, nobj, nzobj, theta, ndist, wavelength, voxelsize, distance, mask_r=None, chunk=None,
               obj_dtype="complex64"):
        """Operators built from the geometry."""
        ntheta = len(theta)
        return cls(Shift(n, nobj, nz, nzobj, obj_dtype),
                   Propagation(n, nz, chunk or ntheta, ndist, wavelength, voxelsize, distance),
                   theta, mask_r, nobj, nzobj, chunk)

    @classmethod
    def from_rec(cls, rec, chunk=None):
        """The data term of a Rec (its shift and propagation operators, angles
        and object mask)."""
        return cls(rec.cl_shift, rec.cl_prop, rec.cl_tomo.theta, rec.mask, rec.nobj, rec.nzobj, chunk)

    # ------------------------------------------------ the fused cascade
    def _use_fused(self, x, prb, pos, mag, data, proj):
        """The fused cascade takes detectors of its row lengths under objects of
        up to twice their width (its rows' shared memory), contiguous arrays
        of the operators' types on their device, a normalisation of at least the
        number of samples, and gives no gradient for the data or the
        magnifications.  It stands for the operators as they were made: a
        propagator set to the padded grid (``_use_cufftdx``) and operators of other
        sizes or types put in the place of the first ones go operator by operator,
        like the rest."""
        sh, prop = self.sh, self.prop
        if type(sh) is not Shift or type(prop) is not Propagation:
            return False
        odt = torch.complex64 if sh.obj_dtype == "complex64" else torch.float32
        shape = (self.ntheta, self.nzobj, self.nobj) if proj else (self.nzobj, self.nobj, self.nobj)
        nd, f32 = (self.ndist, self.nz, self.n), torch.float32
        want = ((x, odt, shape), (prb, torch.complex64, nd), (pos, f32, (self.ntheta, self.ndist, 2)),
                (mag, f32, (self.ntheta, self.ndist)), (data, f32, (self.ntheta,) + nd))
        return (self.n in self.FUSED_ROWS and self.nobj <= 2 * self.n and not data.requires_grad
                and prop._use_cufftdx and (prop.ndist, prop.nz, prop.n) == nd and prop.device == sh.device
                and (sh.n, sh.nz, sh.npsi, sh.nzpsi) == (self.n, self.nz, self.nobj, self.nzobj)
                and all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.dtype == dt and tuple(t.shape) == sz
                        and t.device == sh.device and t.is_contiguous() and not t.is_conj() and not t.is_neg()
                        for t, dt, sz in want)
                and self.data_size >= self.ntheta * self.ndist * self.nz * self.n)

    def _term(self, proj, prb, pos, mag, data):
        out = proj.new_zeros((), dtype=torch.float32).real
        for k in range(self.ndist):
            x22 = shift(proj, pos[:, k].contiguous(), mag[:, k].contiguous(), self.sh)
            x12 = torch.exp(1j * x22)
            x0 = propagate(_ProbeMul.apply(prb[k], x12), k, self.prop)
            out = out + torch.sum((torch.abs(x0) - data[:, k]) ** 2)
        return out

    def _chunk_obj(self, i, obj, prb, pos, mag, data):
        return self._term(radon(obj, self.tomos[i]), prb, pos, mag, data)

    def forward(self, x, prb, pos, mag, data, proj=False):
        """F at (x, prb, pos): x is the object, or with proj=True the
        projections [ntheta, nzobj, nobj] (the BH variable proj)."""
        total = None
        if self._use_fused(x, prb, pos, mag, data, proj):
            for i, (a, b) in enumerate(self.bounds):
                f = _ChunkMisfit.apply(x[a:b] if proj else x, prb, pos[a:b], mag[a:b], data[a:b],
                                       _Cascade(self, b - a, None if proj else self.tomos[i]))
                total = f if total is None else total + f
            return total
        for i, (a, b) in enumerate(self.bounds):
            args = (prb, pos[a:b], mag[a:b], data[a:b])
            if proj:
                f = self._term
                args = (x[a:b],) + args
            else:
                f = self._chunk_obj
                args = (i, x) + args
            t = checkpoint(f, *args, use_reentrant=False) if len(self.bounds) > 1 else f(*args)
            total = t if total is None else total + t
        return total / self.data_size
