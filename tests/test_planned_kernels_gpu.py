"""GPU tests of the kernels a call without a schedule takes: the staged kernels
on a planned tile shape, IQ batch tiles, sorted list entries and the tensor-core
batches, at sizes where they can go wrong (ragged tiles, windows wider than a
slot, record ends, channel remainders), against the FP64 oracle and the float64
torch reference.

Tolerances: an image is a sum of taps whose delays are rounded to FP32, a
relative error of about 2^-23 N * 0.25 cycles * 2 pi per tap on this white data
(3e-5 at N = 600 measured for every kernel), so 1e-4 holds each case.  A delay
rounded across a sample boundary takes the neighbouring slope: with |d tau| up
to 6e-5 a share 2 |d tau| of the taps does, each off by about 1.6 of its own size,
so delay and position gradients are held to sqrt(1.2e-4) * 1.6 = 1.8e-2, to 2.5e-2.
"""
import ctypes

import numpy as np
import pytest
import torch

import ffdas_b200
from ffdas_b200 import _lib
from oracle import oracle
from torch_ref import das_ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = 1e-4
GTOL = 2.5e-2


def _problem(B, C, S, N, nz, nx, pitch=(1.0, 1.0), dtype=torch.float32, seed=0, n=None, z0=20.0):
    """Linear array, (nz, nx) pixels `pitch` wavelengths apart, delays within the record and past both its ends."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn((B, C, S, N), generator=g, dtype=torch.complex64 if dtype.is_complex else torch.float32)
    src = torch.zeros((C, 3))
    src[:, 0] = torch.arange(C) - (C - 1) / 2
    z = z0 + pitch[0] * torch.arange(nz, dtype=torch.float32)
    xx = pitch[1] * (torch.arange(nx, dtype=torch.float32) - (nx - 1) / 2)
    zz, xg = torch.meshgrid(z, xx, indexing="ij")
    dst = torch.stack([xg, 0.1 * xg, zz], -1).contiguous()
    E = S if n is None else n
    offs = (zz[None] + 0.3 * torch.arange(E)[:, None, None] * xg / max(nx, 1) - z0 - 3.0).contiguous()
    w = (torch.rand((E, nz, nx), generator=g) + 0.2)
    return x.to(dtype), src, dst, offs, w


def _dev(*ts):
    return [t.to(DEV) for t in ts]


def _info():
    return ffdas_b200.get_library_handle(torch.device(DEV)).last_kernel_info()


def _oracle(x, src, dst, offs, w, **kw):
    xn = x.to(torch.complex64 if x.is_complex() else torch.float32).numpy()
    kw = {k: (v.numpy() if torch.is_tensor(v) else v) for k, v in kw.items()}
    return oracle.das_f64(xn, src.numpy(), dst.numpy(), offs.numpy(), w.numpy(), **kw)


def _cone(C):
    d = torch.zeros((C, 4))
    d[:, 2], d[:, 3] = 1.0, 0.81
    return d


@pytest.mark.parametrize("pitch", [(0.2, 0.2), (1.7, 0.5), (5.0, 0.4), (0.3, 6.0)], ids=str)
@pytest.mark.parametrize("B,S", [(1, 1), (1, 5), (3, 4)])
@pytest.mark.parametrize("cone", [False, True])
def test_planned_tiles(pitch, B, S, cone):
    # 131 x 67 pixels and 41 channels divide no tile or stage; fine, ordinary and
    # coarse pitches along either axis take different shapes and widths
    x, src, dst, offs, w = _problem(B, 41, S, 600, 131, 67, pitch, seed=S)
    rep = 30 if S > 1 else 120               # enough channels to pass the direct kernel's range
    big = torch.cat([x] * rep, dim=1), src.repeat(rep, 1)
    srcdir = _cone(41 * rep) if cone else None
    got = ffdas_b200.das(*_dev(big[0], big[1], dst, offs, w), srcdir=srcdir.to(DEV) if cone else None)
    assert _info()["variant"] == 2
    ref = rep * _oracle(x, src, dst, offs, w, srcdir=_cone(41) if cone else None)
    assert oracle.rel_l2(got.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("B", [1, 3])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_calls_without_tensor_maps(B, beta):
    # batches then run the 256-voxel kernel one item at a time, which reads no
    # plan: once, in one width, channel slices and all
    # (40 channels, repeated for one item to pass the direct kernel's range: an array of
    # a thousand would lengthen its delays, and their rounding, beyond TOL's N = 600)
    rep = 25 if B == 1 else 4
    x, src, dst, offs, w = _problem(B, 40, 4, 600, 131, 67, (1.7, 0.5))
    ref = rep * _oracle(x, src, dst, offs, w)
    x, src = x.repeat(1, rep, 1, 1), src.repeat(rep, 1)
    old = torch.randn(ref.shape, generator=torch.Generator().manual_seed(2))
    args = _dev(x, src, dst, offs, w)
    L, h, out = _lib.load(), ffdas_b200.get_library_handle(torch.device(DEV)), old.to(DEV)
    b = ctypes.c_float(beta)
    L.ffdas_debug_no_tensor_maps(1)
    try:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        xd = _lib.TensorDesc(list(x.shape), None, _lib.DataType.R_32F)
        od = _lib.TensorDesc(list(out.shape), None, _lib.DataType.R_32F)
        p = [t.data_ptr() for t in args]
        _lib.check(L.ffdas_das(h.h, p[1], None, 0.0, xd.desc, p[0], p[2], p[3], p[4],
                               ctypes.cast(ctypes.byref(b), ctypes.c_void_p), od.desc, out.data_ptr(), 0, 0))
        info = _info()
    finally:
        L.ffdas_debug_no_tensor_maps(0)
    assert info["variant"] == 2 and info["copy_engine"] == 2 and info["batch_tile"] == 1
    assert oracle.rel_l2(out.cpu().numpy(), ref + beta * old.numpy()) < TOL


@pytest.mark.parametrize("dtype,B", [(torch.float32, 1), (torch.float32, 3), (torch.complex64, 2)], ids=str)
def test_adjoint_of_a_voxel_without_a_position_stays_in_its_rows(dtype, B):
    # a NaN position has the distance sqrt(1e-7) of the clamp and no part in its tile's
    # window: a tap in the record, but 60 samples before the window, at the record's end
    C, S, N = 9, 4, 300
    x, src, dst, offs, w = _problem(B, C, S, N, 64, 40, (0.05, 0.05), dtype=dtype, z0=60.0)
    offs = offs - offs.mean() + (N - 80.0)
    clean = offs.clone()
    dst[30, 20] = float("nan")
    args = [t.contiguous() for t in _dev(x, src, dst, offs, w)]
    cplx = dtype.is_complex
    gout = torch.ones((B, 64, 40), device=DEV, dtype=dtype)
    room = torch.zeros(B * C * S * N + 4096, device=DEV, dtype=dtype)      # the gradient, and what follows it
    L, h = _lib.load(), ffdas_b200.get_library_handle(torch.device(DEV))
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    dt = _lib.DataType.C_32F if cplx else _lib.DataType.R_32F
    xd, gd = _lib.TensorDesc(list(x.shape), None, dt), _lib.TensorDesc(list(gout.shape), None, dt)
    p = [t.data_ptr() for t in args]
    _lib.check(L.ffdas_das_backward(h.h, p[1], None, 0.0, xd.desc, p[0], p[2], p[3], p[4], 0, None, gd.desc, gout.data_ptr(),
                                    room.data_ptr(), None, None, None, None))
    assert _info()["variant"] == (8 if cplx else 4)
    assert (room[B * C * S * N:] == 0).all()
    gx = room[: B * C * S * N].reshape(x.shape)
    # every other voxel's taps, as without it
    w2 = w.clone()
    w2[:, 30, 20] = 0.0
    dst[30, 20] = dst[30, 21]
    xr = x.to(torch.complex128 if cplx else torch.float64).requires_grad_(True)
    das_ref(xr, *(t.double() for t in (src, dst, clean, w2))).sum().real.backward()
    few = (gx.cpu() - xr.grad).abs()
    assert few[..., N - 60:].norm() < TOL * xr.grad.norm()


def _with_config(config, f, *args, **kw):
    h = ffdas_b200.get_library_handle(torch.device(DEV))
    h.set_config(config)
    try:
        return f(*args, **kw)
    finally:
        h.set_config(None)


@pytest.mark.parametrize("dtype,B,S,C", [(torch.float32, 1, 5, 1200), (torch.float32, 3, 4, 200), (torch.complex64, 1, 4, 33),
                                         (torch.complex64, 3, 5, 20), (torch.float16, 96, 3, 33)], ids=str)
@pytest.mark.parametrize("far", [2.0 ** 22, 2.0 ** 28])
def test_far_delays_that_cancel_far_distances(dtype, B, S, C, far):
    # distances round to 0.5 and to 32 samples: every kernel takes the same taps as
    # the gather kernels, which test each one by itself (TOL: the same FP32 taps
    # summed in another order, weights of 22 bits in the products)
    x, src, dst, offs, w = _problem(B, C, S, 500, 131, 67, dtype=dtype)
    dst[..., 2] += far
    offs = offs - far + 100.0
    cplx = dtype.is_complex
    args = _dev(x, src, dst, offs, w)
    got = ffdas_b200.das(*args)
    assert _info()["variant"] == (10 if dtype == torch.float16 else 2)
    ref = _with_config({"variant": 1}, ffdas_b200.das, *args)
    assert _info()["variant"] == 1 and ref.abs().max() > 0
    assert oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < TOL
    if dtype == torch.float16:
        return
    gy = torch.randn(got.shape, generator=torch.Generator().manual_seed(1), dtype=got.dtype).to(DEV)
    grads = []
    for config in (None, {"variant": 3}):
        leaf = [t.clone().requires_grad_(True) for t in args]
        _with_config(config, lambda: ffdas_b200.das(*leaf).backward(gy))
        assert _info()["variant"] == (8 if cplx else 3 if config else 4)
        grads.append([t.grad.cpu().numpy() for t in leaf])
    for a, b in zip(*grads):
        assert oracle.rel_l2(a, b) < TOL


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex32])
@pytest.mark.parametrize("B,S,C,N", [(1, 1, 24, 500), (1, 4, 17, 40), (2, 5, 33, 501), (3, 3, 9, 502), (4, 2, 30, 96), (5, 8, 40, 500)])
@pytest.mark.parametrize("pitch", [(0.7, 0.5), (6.0, 0.5)], ids=str)
def test_iq_batch_tiles(dtype, B, S, C, N, pitch):
    # rows read in place and copied (odd lengths), shorter than a window, one to four items a tile
    x, src, dst, offs, w = _problem(B, C, S, N, 50, 37, pitch, dtype=torch.complex64, seed=B + S)
    x = x.to(dtype)
    wn = -1.3
    got = ffdas_b200.das(*_dev(x, src, dst, offs, w), srcdir=_cone(C).to(DEV), wavenum=wn)
    assert _info()["variant"] == 2 and got.dtype == torch.complex64
    ref = _oracle(x, src, dst, offs, w, srcdir=_cone(C), wavenum=wn)
    assert oracle.rel_l2(got.cpu().numpy(), ref) < TOL * (1 + abs(wn))


def test_iq_excluded_channel_with_a_position_that_is_not_finite():
    # outside every cone, as in the oracle: no tap of it, and no NaN from its phase
    x, src, dst, offs, w = _problem(2, 12, 4, 300, 50, 37, dtype=torch.complex64)
    src[5, 0], src[7, 2], dst[20, 10, 1] = float("nan"), float("inf"), float("nan")
    leaf = [t.to(DEV).requires_grad_(i in (0, 3, 4)) for i, t in enumerate((x, src, dst, offs, w))]
    got = ffdas_b200.das(*leaf, srcdir=_cone(12).to(DEV), wavenum=0.3)
    assert _info()["variant"] == 2
    ref = _oracle(x, src, dst, offs, w, srcdir=_cone(12), wavenum=0.3)
    assert np.isfinite(ref).all() and oracle.rel_l2(got.detach().cpu().numpy(), ref) < TOL
    got.backward(torch.ones_like(got))
    assert all(torch.isfinite(leaf[i].grad).all() for i in (0, 3, 4))


def test_iq_strided_data():
    # channels trailing, a row pitch of its own, and starts that are not 16-byte aligned
    x, src, dst, offs, w = _problem(3, 20, 4, 300, 50, 37, dtype=torch.complex64)
    args = _dev(src, dst, offs, w)
    ref = ffdas_b200.das(x.to(DEV), *args, wavenum=0.3)
    wide = torch.zeros((3, 20, 4, 330), device=DEV, dtype=torch.complex64)
    for first in (0, 8, 3):
        wide[..., first:first + 300] = x.to(DEV)
        got = ffdas_b200.das(wide[..., first:first + 300], *args, wavenum=0.3)   # sums in another order at most
        assert torch.linalg.norm(got - ref) < 1e-6 * torch.linalg.norm(ref)
    xt = x.transpose(1, 2).contiguous().to(DEV)
    got = ffdas_b200.das(xt, *args, wavenum=0.3, channels_trailing=True)
    assert torch.linalg.norm(got - ref) < 1e-6 * torch.linalg.norm(ref)


@pytest.mark.parametrize("B,S,C,N,pitch", [(1, 1, 9, 300, (0.7, 0.5)), (2, 5, 20, 301, (0.7, 0.5)), (3, 4, 40, 300, (0.6, 4.0)),
                                           (2, 3, 12, 299, (9.0, 0.5)), (4, 1, 70, 48, (0.3, 0.3)), (6, 6, 13, 128, (0.7, 0.5))], ids=str)
def test_iq_adjoint(B, S, C, N, pitch):
    x, src, dst, offs, w = _problem(B, C, S, N, 24, 19, pitch, dtype=torch.complex64, seed=3)
    wn = 0.4
    gpu = [t.to(DEV).requires_grad_(True) for t in (x, src, dst, offs, w)]
    ref = [t.to(torch.complex128 if t.is_complex() else torch.float64).requires_grad_(True)
           for t in (x, src, dst, offs, w)]
    g = torch.Generator().manual_seed(1)
    gy = torch.randn((B, 24, 19), generator=g, dtype=torch.complex64)
    ffdas_b200.das(*gpu, wavenum=wn).backward(gy.to(DEV))
    assert _info()["variant"] == 8
    das_ref(*ref, wavenum=wn).backward(gy.to(torch.complex128))
    for name, a, b in zip(("x", "srcpos", "dstpos", "offsets", "weights"), gpu, ref):
        tol = TOL if name in ("x", "weights") else GTOL
        assert oracle.rel_l2(a.grad.cpu().numpy(), b.grad.numpy()) < tol, name


def _lists(S, n, V, seed, dup=False):
    g = torch.Generator().manual_seed(seed)
    idx = torch.argsort(torch.rand((S, *V), generator=g), dim=0)[:n].int()
    if dup:
        idx[-1] = idx[0]
    idx[0, 0, 0] = S + 3                     # an event outside x adds nothing
    idx[1 % n, 1, 1] = -1
    w = torch.rand((n, *V), generator=g) + 0.1
    w[torch.rand((n, *V), generator=g) < 0.3] = 0.0
    return idx.contiguous(), w


def _gather_kernel(*args, **kw):
    h = ffdas_b200.get_library_handle(torch.device(DEV))
    h.set_config({"variant": 1})
    try:
        return ffdas_b200.das_sparse(*args, **kw)
    finally:
        h.set_config(None)


def _against_gather(x, src, dst, offs, w, idx, srcdir=None):
    """Both kernels on the whole grid, the oracle on every 13th and 7th pixel: (got, oracle's pixels)."""
    args = _dev(x, src, dst, offs, w, idx)
    kw = {} if srcdir is None else {"srcdir": srcdir.to(DEV)}
    got = ffdas_b200.das_sparse(*args, **kw)
    assert _info()["variant"] == 9
    ref = _gather_kernel(*args, **kw)
    assert _info()["variant"] == 1
    cut = (slice(None), slice(None, None, 13), slice(None, None, 7))
    few = _oracle(x, src, dst[cut[1:]].contiguous(), offs[cut].contiguous(), w[cut].contiguous(),
                  sparse_indices=idx[cut].contiguous(), srcdir=srcdir)
    return got.cpu().numpy(), ref.cpu().numpy(), few


# (2^27 list places and more; items and channels off the box sizes, lists of
# every event and of a few, rows that are copied and rows read in place)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.int16])
@pytest.mark.parametrize("B,C,S,n,N,pitch", [(4, 1000, 4, 4, 512, (1.0, 0.5)), (3, 1101, 6, 5, 509, (4.0, 0.5)), (2, 400, 20, 20, 512, (0.3, 0.3)),
                                             (1, 490, 64, 32, 384, (1.5, 0.5)), (5, 1100, 3, 3, 128, (0.5, 0.5)),
                                             (1, 327, 180, 48, 128, (0.7, 0.4))], ids=str)
def test_sorted_entries(dtype, B, C, S, n, N, pitch):
    x, src, dst, offs, _ = _problem(B, C, S, N, 131, 67, pitch, seed=n, n=n)
    x = (x * 300).round().to(dtype) if dtype == torch.int16 else x.to(dtype)
    idx, w = _lists(S, n, (131, 67), seed=S, dup=True)
    got, ref, few = _against_gather(x, src, dst, offs, w, idx, _cone(C) if n % 2 else None)
    assert oracle.rel_l2(got, ref) < TOL
    assert oracle.rel_l2(got[:, ::13, ::7], few) < TOL


def test_sorted_entries_strided_data():
    # channels trailing, a row pitch of its own, and an offset that is not 16-byte aligned
    x, src, dst, offs, _ = _problem(2, 500, 16, 300, 131, 67, n=16)
    idx, w = _lists(16, 16, (131, 67), seed=3)
    args = _dev(src, dst, offs, w, idx)
    ref = ffdas_b200.das_sparse(x.to(DEV), *args)
    assert _info()["variant"] == 9
    wide = torch.zeros((2, 500, 16, 330), device=DEV)
    for first in (0, 8, 3):
        wide[..., first:first + 300] = x.to(DEV)
        got = ffdas_b200.das_sparse(wide[..., first:first + 300], *args)   # sums in another order at most
        assert torch.linalg.norm(got - ref) < 1e-6 * torch.linalg.norm(ref)
    xt = x.transpose(1, 2).contiguous().to(DEV)
    got = ffdas_b200.das_sparse(xt, *args, channels_trailing=True)
    assert torch.linalg.norm(got - ref) < 1e-6 * torch.linalg.norm(ref)


def test_sorted_entries_without_memory_fall_back_to_pair_rows():
    # FP32 rows that are read in place take no room for a copy; a workspace that does
    # not fit leaves the call to the kernels on pair rows, as before
    x, src, dst, offs, _ = _problem(4, 1000, 4, 512, 131, 67, n=4)
    idx, w = _lists(4, 4, (131, 67), seed=2)
    args = _dev(x, src, dst, offs, w, idx)
    ref = ffdas_b200.das_sparse(*args)
    assert _info()["variant"] == 9
    _lib.load().ffdas_debug_fail_alloc_after(1)
    try:
        got = ffdas_b200.das_sparse(*args)
        assert _info()["variant"] != 9
    finally:
        _lib.load().ffdas_debug_fail_alloc_after(0)
    assert oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < TOL


def test_sorted_entries_non_finite_delay_stays_in_its_voxel():
    x, src, dst, offs, _ = _problem(4, 1000, 4, 512, 131, 67, n=4)
    idx, w = _lists(4, 4, (131, 67), seed=2)
    w[2, 10, 10], idx[2, 10, 10] = 1.0, 1
    offs[2, 10, 10] = float("nan")
    dst[40, 20, 0] = float("inf")
    got, ref, _ = _against_gather(x, src, dst, offs, w, idx)
    ok = np.ones((131, 67), bool)
    ok[10, 10] = ok[40, 20] = False
    assert np.isnan(got[:, 10, 10]).all() and (np.isfinite(got[:, 40, 20]) == np.isfinite(ref[:, 40, 20])).all()
    assert oracle.rel_l2(got[:, ok], ref[:, ok]) < TOL


@pytest.mark.parametrize("B,C,S,N,pitch", [(32, 9, 1, 256, (1.0, 0.5)), (33, 40, 3, 250, (1.5, 0.5)), (64, 17, 4, 504, (6.0, 0.5)),
                                           (270, 8, 2, 160, (0.5, 0.5))], ids=str)
def test_tensor_core_batches(B, C, S, N, pitch):
    # item counts off the multiples of 16 and past one product's 256 columns,
    # rows that are not 16-byte aligned, windows wider than one box, weights
    # spread over six decades (hi + lo parts under one scale per voxel)
    x, src, dst, offs, w = _problem(B, C, S, N, 37, 29, pitch, dtype=torch.float16, seed=B)
    w = w * 10.0 ** (-6.0 * torch.rand(w.shape, generator=torch.Generator().manual_seed(7)))
    for srcdir in (None, _cone(C)):
        got = ffdas_b200.das(*_dev(x, src, dst, offs, w), srcdir=None if srcdir is None else srcdir.to(DEV))
        assert _info()["variant"] == 10
        ref = _oracle(x, src, dst, offs, w, srcdir=srcdir)
        assert oracle.rel_l2(got.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("V,C,S,late", [((128, 296), 260, 3, 0), ((40, 31), 260, 3, 0), ((128, 296), 260, 3, 40),
                                        ((128, 296), 196, 1, 4)], ids=str)
def test_tensor_core_batches_many_drains(V, C, S, late):
    # up to 780 (channel, event) pairs per CTA, with (1240 voxels) and without (37888: a tile an SM)
    # channel slices; `late`: the last channels lie outside the record, and no window
    # follows the last drain
    B = 32 if S == 1 else 96   # (fewer items of three events may take the batch tiles)
    x, src, dst, offs, w = _problem(B, C, S, 256, *V, (0.5, 0.5), dtype=torch.float16, seed=late)
    if late:
        src[C - late:, 2] = 1e6
    args = _dev(x, src, dst, offs, w)
    got = ffdas_b200.das(*args)
    info = _info()
    assert info["variant"] == 10 and (info["kernels"] == 3) == (V != (40, 31))   # plan, products, fix-up: no slices
    ref = _with_config({"variant": 1}, ffdas_b200.das, *args)
    assert oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < TOL
    cut = (slice(None), slice(None, None, 29), slice(None, None, 17))
    few = _oracle(x, src, dst[cut[1:]].contiguous(), offs[cut].contiguous(), w[cut].contiguous())
    assert oracle.rel_l2(got[:, ::29, ::17].cpu().numpy(), few) < TOL
    if late:
        # a NaN position among them has no window either, and the distance sqrt(1e-7)
        # of the clamp: its taps reach every voxel through the fix-up
        src[C - 1, 0] = float("nan")
        args = _dev(x, src, dst, offs + 30.0, w)
        got = ffdas_b200.das(*args)
        ref = _with_config({"variant": 1}, ffdas_b200.das, *args)
        assert oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < TOL


@pytest.mark.parametrize("C,S,N", [(48, 1, 512), (192, 9, 512), (100, 5, 1000)])
def test_tensor_core_batches_are_no_less_exact_than_the_pair_kernels(C, S, N):
    # 22-bit weights and truncated sums against FP32 weights and sums, on the same
    # data, both against the oracle
    x, src, dst, offs, w = _problem(96, C, S, N, 37, 59, (0.2 * N / 37, 0.5), dtype=torch.float16, seed=C)
    args, ref = _dev(x, src, dst, offs, w), _oracle(x, src, dst, offs, w)
    got = ffdas_b200.das(*args)
    assert _info()["variant"] == 10
    pairs = _with_config({"variant": 1}, ffdas_b200.das, *args)
    assert oracle.rel_l2(got.cpu().numpy(), ref) <= oracle.rel_l2(pairs.cpu().numpy(), ref)


@pytest.mark.parametrize("B,C,S,N,pitch", [(32, 40, 4, 256, (0.4, 0.5)), (33, 40, 4, 250, (12.0, 9.0)), (40, 150, 3, 504, (0.5, 0.4)),
                                           (40, 150, 3, 501, (15.0, 15.0)), (64, 20, 5, 256, (3.0, 2.0))], ids=str)
def test_batches_on_the_products_or_the_batch_tiles(B, C, S, N, pitch):
    # few items: fine pitches leave the image to the batch tiles, coarse ones, whose
    # windows overflow, to the products; both launched, with channel slices and without
    x, src, dst, offs, w = _problem(B, C, S, N, 131, 67, pitch, dtype=torch.float16, seed=B + S)
    args = _dev(x, src, dst, offs, w)
    out = torch.full((B, 131, 67), float("nan"), device=DEV)
    for srcdir in (None, _cone(C).to(DEV)):
        ffdas_b200.das(*args, srcdir=srcdir, out=out)
        assert _info()["variant"] == 10
        ref = _with_config({"variant": 1}, ffdas_b200.das, *args, srcdir=srcdir)
        # (each is off 64 bits by less than TOL)
        assert oracle.rel_l2(out.cpu().numpy(), ref.cpu().numpy()) < 2 * TOL
        few = _oracle(x, src, dst[::13, ::7].contiguous(), offs[:, ::13, ::7].contiguous(), w[:, ::13, ::7].contiguous(),
                      srcdir=None if srcdir is None else _cone(C))
        assert oracle.rel_l2(out[:, ::13, ::7].cpu().numpy(), few) < TOL
    if B == 64:   # (on the products in any case)
        return
    _lib.load().ffdas_debug_fail_alloc_after(1)   # no room for pair rows: the products need none
    try:
        got = ffdas_b200.das(*args, srcdir=srcdir)
    finally:
        _lib.load().ffdas_debug_fail_alloc_after(0)
    assert _info()["kernels"] <= 5 and oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < 2 * TOL


def test_tensor_core_batches_channels_trailing_view_and_non_finite_values():
    # a (B, S, C, N) view; an infinite and a NaN sample, a NaN delay and an
    # infinite weight reach the values whose taps meet them and no others
    x, src, dst, offs, w = _problem(40, 12, 3, 256, 40, 31, (1.0, 0.5), dtype=torch.float16, seed=5)
    clean = _oracle(x, src, dst, offs, w)
    x[3, 4, 1, 100], x[7, 2, 0, 60] = float("inf"), float("nan")
    offs[1, 5, 5], w[2, 30, 8] = float("nan"), float("inf")
    ref = _oracle(x, src, dst, offs, w)
    ref[:, 5, 5] = np.nan   # a NaN delay makes its voxel NaN; the oracle leaves the tap out
    xt = x.transpose(1, 2).contiguous().to(DEV)
    got = ffdas_b200.das(xt, *_dev(src, dst, offs, w), channels_trailing=True).cpu().numpy()
    assert _info()["variant"] == 10
    assert (np.isfinite(got) == np.isfinite(ref)).mean() > 0.9999   # a delay may round across a spoiled sample
    both = np.isfinite(got) & np.isfinite(ref)
    assert both.mean() > 0.9 and not both.all()
    assert oracle.rel_l2(got[both], clean[both]) < TOL


@pytest.mark.parametrize("kind,variant,kept", [("staged", 2, True), ("batch", 2, True), ("lists", 1, True), ("direct", 5, False),
                                               ("iq", 2, False), ("entries", 9, False)])
def test_pair_buffer_only_where_the_backward_reads_it(kind, variant, kept):
    B, C, S, n, dtype = dict(staged=(1, 1200, 4, 4, torch.float32), batch=(33, 20, 3, 3, torch.float16),
                             lists=(1, 40, 8, 4, torch.float32), direct=(1, 40, 3, 3, torch.float32),
                             iq=(2, 20, 3, 3, torch.complex64), entries=(4, 1000, 4, 4, torch.float32))[kind]
    x, src, dst, offs, w = _problem(B, C, S, 512, 131, 67, dtype=dtype, n=n)
    x, src, dst, offs, w = [t.to(DEV).requires_grad_(i == 3) for i, t in enumerate((x, src, dst, offs, w))]
    if kind in ("lists", "entries"):
        out = ffdas_b200.das_sparse(x, src, dst, offs, w, _lists(S, n, (131, 67), seed=1)[0].to(DEV))
    else:
        out = ffdas_b200.das(x, src, dst, offs, w)
    assert _info()["variant"] == variant
    assert (out.grad_fn.pairs is not None) == kept
    out.backward(torch.ones_like(out))
    assert torch.isfinite(offs.grad).all() and offs.grad.abs().max() > 0


_CAPTURED = dict(staged=(1, 1200, 4, torch.float32, 2), batch=(3, 200, 3, torch.float32, 2), products=(96, 12, 3, torch.float16, 10),
                 either=(33, 40, 3, torch.float16, 10),
                 iq=(3, 20, 4, torch.complex64, 2), iq_copied=(1, 20, 1, torch.complex64, 2), entries=(4, 1000, 4, torch.float32, 9))


@pytest.mark.parametrize("kind", _CAPTURED)
def test_captured_call_follows_its_inputs(kind):
    # a graph of one unscheduled call: the plan, its overlapped ingest, both widths,
    # the sort, the clearing of sliced images -- all made again at each replay, for
    # new data and for delays of another spread
    B, C, S, dtype, variant = _CAPTURED[kind]
    N = 501 if kind == "iq_copied" else 512
    x, src, dst, offs, w = _problem(B, C, S, N, 131, 67, (0.4, 0.5), dtype=dtype)
    args = _dev(x, src, dst, offs, w)
    if kind == "entries":
        idx = _lists(S, S, (131, 67), seed=1)[0].to(DEV)
        call = lambda out=None: ffdas_b200.das_sparse(*args, idx, out=out)  # noqa: E731
    else:
        call = lambda out=None: ffdas_b200.das(*args, out=out)  # noqa: E731
    out = call()
    assert _info()["variant"] == variant
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call(out)
    for spread in (1.0, 1.9):
        args[0].copy_(args[0].roll(7, dims=-1))
        args[3].copy_(offs.to(DEV) * spread)
        ref = call()
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        # the same taps; sums that meet in atomics come in another order
        assert oracle.rel_l2(out.cpu().numpy(), ref.cpu().numpy()) < 1e-6


@pytest.mark.parametrize("per_item", [False, True])
def test_channel_scale_and_beta_on_the_iq_and_entry_kernels(per_item):
    L, h = _lib.load(), ffdas_b200.get_library_handle(torch.device(DEV))
    for kind in ("iq", "entries"):
        B, C, S, dtype = (2, 24, 4, torch.complex64) if kind == "iq" else (4, 1000, 4, torch.float32)
        x, src, dst, offs, w = _problem(B, C, S, 300, 131, 67, dtype=dtype)
        idx = _lists(S, S, (131, 67), seed=1)[0] if kind == "entries" else None
        g = torch.rand((B, C) if per_item else (C,), generator=torch.Generator().manual_seed(3)) + 0.5
        args = _dev(x, src, dst, offs, w)
        call = (lambda *a, **k: ffdas_b200.das_sparse(*a, idx.to(DEV), **k)) if kind == "entries" else ffdas_b200.das
        got = call(*args, channel_scale=g.to(DEV))
        assert _info()["variant"] == (2 if kind == "iq" else 9)
        xs = x * g.reshape(-1, C, 1, 1)
        ref = _with_config({"variant": 1}, call, xs.to(DEV), *args[1:])
        assert oracle.rel_l2(got.cpu().numpy(), ref.cpu().numpy()) < TOL
        # beta through the C entry: out = beta * out + image, with and without channel slices
        old = torch.randn(got.shape, generator=torch.Generator().manual_seed(4), dtype=got.dtype)
        out, plain = old.to(DEV), call(*args)
        beta = (ctypes.c_float * 2)(0.5, 0.25 if kind == "iq" else 0.0)
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        dt = _lib.DataType.C_32F if kind == "iq" else _lib.DataType.R_32F
        xd, od = _lib.TensorDesc(list(x.shape), None, dt), _lib.TensorDesc(list(out.shape), None, dt)
        p, b = [t.data_ptr() for t in args], ctypes.cast(beta, ctypes.c_void_p)
        if kind == "iq":
            _lib.check(L.ffdas_das(h.h, p[1], None, 0.0, xd.desc, p[0], p[2], p[3], p[4], b, od.desc, out.data_ptr(), 0, 0))
        else:
            i = idx.to(DEV)
            _lib.check(L.ffdas_das_sparse(h.h, p[1], None, 0.0, xd.desc, p[0], p[2], p[3], p[4], S, i.data_ptr(), b, od.desc,
                                          out.data_ptr(), 0, 0))
        assert _info()["variant"] == (2 if kind == "iq" else 9)
        want = plain.cpu() + (complex(0.5, 0.25) if kind == "iq" else 0.5) * old
        assert oracle.rel_l2(out.cpu().numpy(), want.numpy()) < 1e-6


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex32])
@pytest.mark.parametrize("need", ["x", "weights", "offsets", "srcpos", "dstpos", "dstpos,offsets", "x,weights"])
def test_iq_adjoint_subsets(dtype, need):
    # each gradient by itself (the kernel scatters, sums and clears only what is asked
    # for) against all of them at once; complex32 data at odd sizes
    x, src, dst, offs, w = _problem(3, 21, 5, 301, 24, 19, (1.1, 0.6), dtype=torch.complex64, seed=9)
    x = x.to(dtype)
    names = ("x", "srcpos", "dstpos", "offsets", "weights")
    gy = torch.randn((3, 24, 19), generator=torch.Generator().manual_seed(1), dtype=torch.complex64).to(DEV)
    some, every = ([t.to(DEV).requires_grad_(n in which) for n, t in zip(names, (x, src, dst, offs, w))]
                   for which in (need.split(","), names))
    for leaf in (some, every):
        ffdas_b200.das(*leaf, wavenum=0.4).backward(gy)
        assert _info()["variant"] == 8
    for n, a, b in zip(names, some, every):
        if n in need.split(","):
            # fixed-point sums are exact in any order; the rest differ by the order of FP32 sums
            assert oracle.rel_l2(a.grad.cfloat().cpu().numpy(), b.grad.cfloat().cpu().numpy()) < 1e-5
    if dtype == torch.complex32:   # the same numbers in single precision
        ref = [t.detach().cfloat() if t.is_complex() else t.detach() for t in every]
        ref = [t.clone().requires_grad_(True) for t in ref]
        ffdas_b200.das(*ref, wavenum=0.4).backward(gy)
        for n, a, b in zip(names, every, ref):   # (x's gradient comes back in 11 bits)
            assert oracle.rel_l2(a.grad.cfloat().cpu().numpy(), b.grad.cfloat().cpu().numpy()) < (1e-3 if n == "x" else TOL)


@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("S", [33, 97])
def test_select_sizes(k, S):
    # around the group sizes 4, 8, 16, 32 and the staged event limit, one voxel past a block
    g = torch.Generator().manual_seed(k * 100 + S)
    w = torch.randint(0, 9, (S, 129), generator=g).float()      # many ties
    o = torch.rand((S, 129), generator=g)
    idx, sw, so = ffdas_b200.sparse_select(w.to(DEV), k, offsets=o.to(DEV))
    order = torch.sort(w, dim=0, descending=True, stable=True)[1][:k]
    assert torch.equal(idx.cpu().long(), order)
    assert torch.equal(sw.cpu(), w.gather(0, order)) and torch.equal(so.cpu(), o.gather(0, order))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int16])
@pytest.mark.parametrize("S", [1, 2, 3, 5, 7, 8, 9])
def test_rows_where_every_window_is_too_wide(dtype, S):
    # pixels 24 samples apart along both axes: each channel's windows all overflow, or
    # some of an event chunk do (the tile's corner), with chunks that are not full
    C = 40
    x, src, dst, offs, w = _problem(1, C, S, 700, 40, 110, (24.0, 24.0), seed=S, dtype=torch.float32)
    x = (x * 300).round().to(dtype) if dtype == torch.int16 else x.to(dtype)
    rep = 1 + (1 << 25) // (C * S * 4400)   # past the direct kernel
    ref = rep * _oracle(x.float(), src, dst, offs, w)
    got = ffdas_b200.das(*_dev(x.repeat(1, rep, 1, 1), src.repeat(rep, 1), dst, offs, w))
    assert _info()["variant"] == 2
    assert oracle.rel_l2(got.cpu().numpy(), ref) < TOL
