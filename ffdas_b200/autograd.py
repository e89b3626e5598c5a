"""torch.autograd.Function for delay-and-sum with hand-written backward kernels.

Forward calls ffdas_das / ffdas_das_sparse; backward calls ffdas_das_backward,
which recomputes each interpolation tap (no stored indices) and returns the
gradients with respect to channel data (two-tap adjoint scatter), weights,
delays (through the interpolant's slope) and voxel / channel positions.
Real channel data (float32, float16, bfloat16) without phase rotation, and
complex IQ data (complex64, complex32) with any wavenum; element directivity
(srcdir) masks taps as in the forward, and the mask has no gradient (it is
piecewise constant in the positions).  The gradient of x is returned in x's
dtype and layout.
"""
from __future__ import annotations

from array import array

import torch

from . import _lib
from ._lib import DataType
from .das import _FFDAS_DTYPE, _astype, _bits, _check_spatial, _raw_stream, _run, _to_torch, _x_layout
from .library import get_library_handle


def _backward_supported(x: torch.Tensor, wavenum: float) -> bool:
    if x.is_complex():
        return x.dtype in (torch.complex64, torch.complex32)
    return wavenum == 0.0 and x.dtype in (torch.float32, torch.float16, torch.bfloat16, torch.int16)


class DASFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, srcpos, dstpos, offsets, weights, sparse_indices, opts: dict):
        ctx.opts = opts
        xt = x.detach()
        # Where the forward builds interpolation-pair rows and the backward can run,
        # they are kept in a buffer and the backward skips building them again.
        keep = _backward_supported(xt, opts["wavenum"])
        out = _run(xt, srcpos.detach(), dstpos.detach(), offsets.detach(), weights.detach(), sparse_indices,
                   srcdir=opts["srcdir"], wavenum=opts["wavenum"], algorithm=0, use_fp16=opts["use_fp16"],
                   use_bf16=opts["use_bf16"], channels_trailing=opts["channels_trailing"], out=None,
                   keep_pairs=keep)
        out, ctx.pairs = out if keep else (out, None)
        ctx.save_for_backward(x, srcpos, dstpos, offsets, weights,
                              sparse_indices if sparse_indices is not None else torch.empty(0))
        ctx.has_sparse = sparse_indices is not None
        return out

    @staticmethod
    def backward(ctx, gout):
        x, srcpos, dstpos, offsets, weights, idx = ctx.saved_tensors
        opts = ctx.opts
        if not _backward_supported(x, opts["wavenum"]):
            raise NotImplementedError("das backward supports real data without phase rotation (wavenum 0) "
                                      "and complex64 / complex32 data")
        need = ctx.needs_input_grad
        dev = x.device
        cplx = x.is_complex()
        gout = gout.contiguous().to(torch.complex64 if cplx else torch.float32)
        xt = x.detach()
        lead = xt.shape if xt.ndim == 4 else (1, *xt.shape)
        if opts["channels_trailing"]:
            B, S, C, N = lead
        else:
            B, C, S, N = lead
        gx = torch.zeros((B, C, S, N), dtype=torch.complex64 if cplx else torch.float32, device=dev) if need[0] else None
        goff = torch.empty(offsets.shape, dtype=torch.float32, device=dev) if need[3] else None
        gw = torch.empty(weights.shape, dtype=torch.float32, device=dev) if need[4] else None
        gdst = torch.empty(dstpos.shape, dtype=torch.float32, device=dev) if need[2] else None
        gsrc = torch.empty(srcpos.shape, dtype=torch.float32, device=dev) if need[1] else None

        f32 = lambda t: _astype(t.detach(), torch.float32, dev, "input")  # noqa: E731
        srcpos_t, dstpos_t, offsets_t, weights_t = f32(srcpos), f32(dstpos), f32(offsets), f32(weights)
        srcdir_t = f32(_to_torch(opts["srcdir"])) if opts["srcdir"] is not None else None
        idx_t = _astype(idx, torch.int32, dev, "sparse_indices") if ctx.has_sparse else None
        handle = get_library_handle(dev)
        ptr = lambda t: 0 if t is None else t.data_ptr()  # noqa: E731
        # one native call; the forward's pair rows are read instead of rebuilt when they match
        gd = gout.shape
        q = array("q", [handle.h.value, _raw_stream(dev.index), ptr(srcpos_t), ptr(srcdir_t), _bits(opts["wavenum"]),
                        ptr(xt), _FFDAS_DTYPE[xt.dtype], *_x_layout(xt, opts["channels_trailing"]), ptr(dstpos_t),
                        ptr(offsets_t), ptr(weights_t), idx_t.shape[0] if idx_t is not None else 0, ptr(idx_t),
                        ptr(gout), DataType.C_32F if cplx else DataType.R_32F, ptr(gx), ptr(goff), ptr(gw), ptr(gdst),
                        ptr(gsrc), ptr(ctx.pairs), ctx.pairs.numel() if ctx.pairs is not None else 0, len(gd), *gd,
                        *gout.stride()])
        _lib.check(_lib.load().ffdas_das_backward_call(q.buffer_info()[0], len(q)))
        ctx.pairs = None
        if gx is not None:
            if opts["channels_trailing"]:
                gx = gx.transpose(1, 2)
            if xt.ndim == 3:
                gx = gx[0]
            gx = gx.to(xt.dtype)
        cast = lambda g, ref: None if g is None else g.to(ref.dtype)  # noqa: E731
        return gx, cast(gsrc, srcpos), cast(gdst, dstpos), cast(goff, offsets), cast(gw, weights), None, None


def das_autograd(x, srcpos, dstpos, offsets, weights, sparse_indices=None, *, srcdir=None, wavenum=0.0,
                 use_fp16=False, use_bf16=False, channels_trailing=False):
    """Differentiable das / das_sparse (see ffdas_b200.das)."""
    _check_spatial(dstpos, offsets, weights, sparse_indices)
    tens = [_to_torch(t) for t in (x, srcpos, dstpos, offsets, weights)]
    idx = _to_torch(sparse_indices) if sparse_indices is not None else None
    opts = dict(srcdir=srcdir, wavenum=float(wavenum), use_fp16=use_fp16, use_bf16=use_bf16,
                channels_trailing=channels_trailing)
    return DASFunction.apply(*tens, idx, opts)
