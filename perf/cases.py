"""Timed cases of the delay-and-sum library, through its public Python calls.

`listed()` holds one case for each thing a program does with this library:
beamform one small frame, one compounded frame, a volume, an ensemble of
frames, IQ data and focused transmits with per-pixel lists; differentiate each
of the dense, list and IQ forms; choose the lists; filter the clutter out of an
ensemble.  `draw` gives further cases of the same kinds with sizes spread over
the ranges between (and around) them.  Channel data is band-limited noise
centred on a quarter of the sampling rate (speckle); geometry is a linear or a
square array with plane, diverging or focused transmits.  Positions are in
sampling wavelengths, delays in samples.
"""
from __future__ import annotations

import math

import torch

import ffdas_b200 as ffdas

_DTYPES = {
    "f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "i16": torch.int16,
    "f64": torch.float64, "c64": torch.complex64,
}


# ------------------------------------------------------------------- cases ---
def listed():
    return [
        # a preview or a region of interest: the smallest call, host time and one launch
        dict(name="frame_small", kind="das", array="linear", dtype="f32", B=1, C=32, S=1, N=512, nz=64, nx=32,
             z0=38.0, z1=240.0, xhalf=16.0, grad=False),
        # one compounded 2-D frame straight from the digitiser (raw int16), with element
        # directivity and sizes that divide nothing
        dict(name="frame_compound", kind="das", array="linear", dtype="i16", B=1, C=127, S=11, N=1535, nz=401, nx=255,
             z0=50.0, z1=700.0, xhalf=64.0, directivity=True, grad=False),
        # 3-D volume of a 32 x 32 matrix array, 16 diverging waves: the largest single call
        dict(name="volume", kind="das", array="matrix", dtype="f32", B=1, C=1024, S=16, N=4096, nz=128, ny=128,
             nx=128, z0=100.0, z1=3900.0, xhalf=40.0, grad=False),
        # 200-frame ensemble of half-precision channel data (flow imaging)
        dict(name="ensemble", kind="das", array="linear", dtype="f16", B=200, C=128, S=11, N=1536, nz=400, nx=256,
             z0=50.0, z1=700.0, xhalf=64.0, grad=False),
        # demodulated (IQ) data of a few frames with the phase rotation
        dict(name="iq_frames", kind="das", array="linear", dtype="c64", B=4, C=128, S=8, N=2048, nz=256, nx=256,
             z0=60.0, z1=940.0, xhalf=64.0, wavenum=-1.5707963, grad=False),
        # focused transmits, each pixel summing its own 1..32 of 64 (lists padded with weight 0)
        dict(name="sparse_focus", kind="sparse", lists="uneven", dtype="f32", C=128, S=64, k=32, N=1536, nz=400,
             nx=256, z0=50.0, z1=700.0, xhalf=64.0, grad=False),
        # one autofocus step on four frames: image and the gradients of data, delays,
        # weights and both position sets
        dict(name="train_autofocus", kind="das", array="linear", dtype="f32", B=4, C=128, S=8, N=2048, nz=256, nx=256,
             z0=6.0, z1=70.0, xhalf=48.0, grad=True),
        # the same through per-pixel lists of focused transmits
        dict(name="train_sparse", kind="sparse", lists="uneven", dtype="f32", C=128, S=64, k=32, N=1536, nz=400,
             nx=256, z0=50.0, z1=700.0, xhalf=64.0, grad=True),
        # the same on IQ data
        dict(name="train_iq", kind="das", array="linear", dtype="c64", B=2, C=128, S=8, N=2048, nz=192, nx=256,
             z0=60.0, z1=940.0, xhalf=64.0, wavenum=0.05, grad=True),
        # choosing the lists: per pixel the 32 strongest of 64 transmits, with their delays
        dict(name="select_lists", kind="select", S=64, k=32, nz=400, nx=256),
        # clutter filter of a 200-frame ensemble of images, five tissue components removed
        dict(name="clutter_frames", kind="rank", dtype="f32", m=200, n=102400, start=5),
        # the same for 64 complex volumes of 64^3 voxels
        dict(name="clutter_volumes", kind="rank", dtype="c64", m=64, n=262144, start=5),
    ]


def _spread(rng, lo, hi):
    """A whole number in lo..hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "volume", "ensemble", "iq", "sparse", "train", "train_sparse", "train_iq",
                       "select", "rank", "rank"])
    if kind == "rank":
        dtype = rng.choice(["f32", "f32", "c64", "f64"])
        return dict(kind="rank", dtype=dtype, m=_spread(rng, 16, 200 if dtype == "f32" else 64),
                    n=_spread(rng, 10000, 100000 if dtype == "f64" else 260000), start=rng.randint(1, 5))
    if kind == "select":
        S = _spread(rng, 8, 128)
        return dict(kind="select", S=S, k=_spread(rng, 2, min(S, 32)), nz=_spread(rng, 100, 400),
                    nx=_spread(rng, 64, 256))
    N = _spread(rng, 512, 2560)
    z = dict(z0=round(0.03 * N, 2), z1=round(rng.uniform(0.2, 0.46) * N, 2))
    if kind == "volume":
        side = rng.randint(12, 32)
        nv = rng.randint(40, 96)
        return dict(kind="das", array="matrix", dtype=rng.choice(["f32", "f32", "i16", "bf16"]), B=1, C=side * side,
                    S=rng.randint(2, 9), N=N, nz=rng.randint(40, 96), ny=nv, nx=nv, xhalf=side * 1.25, grad=False, **z)
    C = _spread(rng, 48, 192)
    grid = dict(nz=_spread(rng, 100, 400), nx=_spread(rng, 64, 256), xhalf=C / 2.0)
    if kind in ("sparse", "train_sparse"):
        S = _spread(rng, 16, 64)
        return dict(kind="sparse", lists=rng.choice(["uneven", "nearest"]), dtype="f32", C=C, S=S,
                    k=rng.randint(4, min(S, 32)), N=N, grad=kind == "train_sparse", **grid, **z)
    if kind == "ensemble":
        return dict(kind="das", array="linear", dtype=rng.choice(["f16", "f16", "bf16", "f32", "i16"]),
                    B=_spread(rng, 16, 128), C=C, S=rng.randint(1, 9), N=N, grad=False, **grid, **z)
    if kind in ("iq", "train_iq"):
        return dict(kind="das", array="linear", dtype="c64", B=rng.randint(1, 2 if kind == "train_iq" else 8), C=C,
                    S=rng.randint(1, 11), N=N, wavenum=rng.choice([-1.5707963, 0.05]), grad=kind == "train_iq",
                    directivity=rng.random() < 0.25, **grid, **z)
    if kind == "train":
        return dict(kind="das", array="linear", dtype="f32", B=rng.randint(1, 6), C=C, S=rng.randint(1, 11), N=N,
                    grad=True, **grid, **z)
    return dict(kind="das", array="linear", dtype=rng.choice(["f32", "i16", "f16"]), B=1, C=C, S=_spread(rng, 1, 16), N=N,
                directivity=rng.random() < 0.25, grad=False, **grid, **z)


# ------------------------------------------------------------------ inputs ---
def _gen(seed, dev):
    return torch.Generator(device=dev).manual_seed(seed)


def _speckle(shape, dtype, gen, dev):
    """Noise band-limited around a quarter of the sampling rate (low-pass for IQ data), unit RMS."""
    *lead, n = shape
    if dtype.is_complex:
        y = torch.randn(*lead, n + 2, generator=gen, device=dev, dtype=torch.complex64)
        return ((y[..., 2:] + 2 * y[..., 1:-1] + y[..., :-2]) / math.sqrt(6.0)).contiguous()
    out = torch.empty(shape, dtype=dtype, device=dev)
    for b in range(lead[0]):     # item by item: an ensemble's float32 noise would not fit beside it
        y = torch.randn(*lead[1:], n + 4, generator=gen, device=dev)
        y = (y[..., 4:] - 2 * y[..., 2:-2] + y[..., :-4]) / math.sqrt(6.0)
        out[b] = (y * 500.0).round() if dtype == torch.int16 else y
    return out


def _geometry(case, dev):
    """Channel positions (C, 3), voxel positions (..., 3) and the spatial shape."""
    C, xh = case["C"], case["xhalf"]
    z = torch.linspace(case["z0"], case["z1"], case["nz"], device=dev)
    x = torch.linspace(-xh, xh, case["nx"], device=dev)
    if case.get("array") == "matrix":
        side = math.isqrt(C)
        e = torch.arange(side, device=dev, dtype=torch.float32) - (side - 1) / 2
        ey, ex = torch.meshgrid(e, e, indexing="ij")
        src = torch.stack([ex.reshape(-1), ey.reshape(-1), torch.zeros(C, device=dev)], -1)
        y = torch.linspace(-xh, xh, case["ny"], device=dev)
        zz, yy, xx = torch.meshgrid(z, y, x, indexing="ij")
        return src, torch.stack([xx, yy, zz], -1).contiguous()
    src = torch.zeros(C, 3, device=dev)
    src[:, 0] = torch.arange(C, device=dev, dtype=torch.float32) - (C - 1) / 2
    zz, xx = torch.meshgrid(z, x, indexing="ij")
    return src, torch.stack([xx, torch.zeros_like(xx), zz], -1).contiguous()


def _plane_or_diverging(case, dst, dev):
    """Delays (S, ...) of plane waves (linear array) or diverging waves (matrix array)."""
    S = case["S"]
    if case["array"] == "matrix":
        g = torch.linspace(-12.0, 12.0, max(1, math.isqrt(S - 1) + 1) if S > 1 else 1, device=dev)
        sy, sx = torch.meshgrid(g, g, indexing="ij")
        vs = torch.stack([sx.reshape(-1), sy.reshape(-1), torch.full((g.numel() ** 2,), -50.0, device=dev)], -1)[:S]
        return torch.stack([(dst - v).norm(dim=-1) - 50.0 for v in vs])
    th = torch.deg2rad(torch.linspace(-10.0, 10.0, S, device=dev) if S > 1 else torch.zeros(1, device=dev))
    return torch.stack([dst[..., 0] * torch.sin(t) + dst[..., 2] * torch.cos(t) for t in th])


def _focused(case, dst, gen, dev):
    """Lists (k, ...) of focused transmits: indices, delays and weights."""
    S, k = case["S"], case["k"]
    zf = case["z1"] * 8.0 / 7.0
    fx = torch.linspace(-0.94 * case["xhalf"], 0.94 * case["xhalf"], S, device=dev)
    dist = torch.hypot(dst[..., 0][None] - fx[:, None, None], dst[..., 2][None] - zf)
    full = zf + torch.where(dst[..., 2] < zf, -1.0, 1.0)[None] * dist          # (S, nz, nx)
    shape = dst.shape[:-1]
    if case["lists"] == "nearest":     # the k transmits nearest in x, Hann-weighted over them
        order = (dst[..., 0][None] - fx[:, None, None]).abs().argsort(dim=0, stable=True)[:k]
        h = torch.sin(math.pi * (torch.arange(k, device=dev) + k + 0.5) / (2 * k)) ** 2
        return order.int().contiguous(), full.gather(0, order).contiguous(), h[:, None, None].expand(k, *shape).contiguous()
    length = torch.randint(1, k + 1, shape, generator=gen, device=dev)
    start = (torch.rand(shape, generator=gen, device=dev) * (S - length + 1)).long()
    i = torch.arange(k, device=dev)[:, None, None]
    valid = i < length[None]
    idx = torch.where(valid, start[None] + i, start[None])
    return idx.int().contiguous(), full.gather(0, idx).contiguous(), valid.float().contiguous()


def _das_inputs(case, seed, dev):
    gen = _gen(seed, dev)
    dtype = _DTYPES[case["dtype"]]
    src, dst = _geometry(case, dev)
    B, S = case.get("B", 1), case["S"]
    d = dict(x=_speckle((B, case["C"], S, case["N"]), dtype, gen, dev), srcpos=src, dstpos=dst)
    if case["kind"] == "sparse":
        d["idx"], d["offsets"], d["weights"] = _focused(case, dst, gen, dev)
    else:
        d["offsets"] = _plane_or_diverging(case, dst, dev).contiguous()
        h = 0.5 + 0.5 * torch.sin(math.pi * (torch.arange(S, device=dev, dtype=torch.float32) + 0.5) / S) ** 2
        d["weights"] = h.reshape(-1, *[1] * (dst.ndim - 1)).expand_as(d["offsets"]).contiguous()
    if case.get("directivity"):      # elements look along +z, 40 degree acceptance half-angle
        d["srcdir"] = torch.tensor([0.0, 0.0, 1.0, math.cos(math.radians(40.0))], device=dev).repeat(case["C"], 1)
    if case["grad"]:
        g = torch.randn((B, *dst.shape[:-1]), generator=gen, device=dev,
                        dtype=torch.complex64 if dtype.is_complex else torch.float32)
        d["gout"] = g
    return d


def _ensemble(case, seed, dev):
    """(m, n) slow-time data: five low-rank tissue components, each 4x weaker than the last, and weak blood."""
    gen = _gen(seed, dev)
    dt = _DTYPES[case["dtype"]]
    m, n, tissue = case["m"], case["n"], min(5, case["m"])
    wide = torch.complex128 if dt.is_complex else torch.float64
    u = torch.linalg.qr(torch.randn(m, tissue, generator=gen, device=dev, dtype=wide))[0]
    v = torch.randn(tissue, n, generator=gen, device=dev, dtype=dt)
    s = 10.0 * 4.0 ** -torch.arange(tissue, device=dev, dtype=torch.float64)
    return ((u * s).to(dt) @ v + 1e-2 * torch.randn(m, n, generator=gen, device=dev, dtype=dt)).contiguous()


def prepare(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "rank":
        return dict(case=case, x=_ensemble(case, seed, dev))
    if case["kind"] == "select":     # apodization that falls with the lateral distance to the focus, and the delays
        gen = _gen(seed, dev)
        S, nz, nx = case["S"], case["nz"], case["nx"]
        fx = torch.linspace(-60.0, 60.0, S, device=dev)[:, None, None]
        px = torch.linspace(-64.0, 64.0, nx, device=dev)[None, None, :]
        w = torch.exp(-((px - fx) / 40.0) ** 2) * (0.5 + torch.rand(S, nz, nx, generator=gen, device=dev))
        return dict(case=case, weights=w.contiguous(), offsets=700.0 * torch.rand(S, nz, nx, generator=gen, device=dev))
    d = _das_inputs(case, seed, dev)
    d["case"] = case
    if case["grad"]:
        for k in ("x", "srcpos", "dstpos", "offsets", "weights"):
            d[k].requires_grad_(True)
    return d


# --------------------------------------------------------------------- run ---
def run(state):
    case = state["case"]
    if case["kind"] == "rank":
        return ffdas.truncate_rank(state["x"], case["start"])
    if case["kind"] == "select":
        return ffdas.sparse_select(state["weights"], case["k"], offsets=state["offsets"])
    args = [state[k] for k in ("x", "srcpos", "dstpos", "offsets", "weights")]
    if case["kind"] == "sparse":
        out = ffdas.das_sparse(*args, state["idx"])
    else:
        out = ffdas.das(*args, srcdir=state.get("srcdir"), wavenum=case.get("wavenum", 0.0))
    if not case["grad"]:
        return out
    return [out.detach(), *torch.autograd.grad(out, args, state["gout"])]


# -------------------------------------------------------------------- work ---
def _size(dtype):
    return {"f32": 4, "f16": 2, "bf16": 2, "i16": 2, "f64": 8, "c64": 8}[dtype]


def work(case):
    if case["kind"] == "rank":
        # the Gram matrix (upper half) and the projection onto `start` vectors
        m, n, f = case["m"], case["n"], 4 if case["dtype"] == "c64" else 1
        return {"bytes": 2 * m * n * _size(case["dtype"]), "flops": f * (m * m * n + 4 * m * n * case["start"])}
    if case["kind"] == "select":
        V = case["nz"] * case["nx"]
        return {"bytes": 8 * case["S"] * V + 12 * case["k"] * V, "flops": case["S"] * V}
    B, C, S, N = case.get("B", 1), case["C"], case["S"], case["N"]
    V = case["nz"] * case["nx"] * case.get("ny", 1)
    E = case["k"] if case["kind"] == "sparse" else S
    # an uneven list has (k + 1) / 2 entries on average
    units = B * C * V * ((E + 1) / 2 if case.get("lists") == "uneven" else E)
    cplx = case["dtype"] == "c64"
    x, img = B * C * S * N * _size(case["dtype"]), B * V * (8 if cplx else 4)
    geom = 4 * (V * E * (3 if case["kind"] == "sparse" else 2) + 3 * V + 3 * C)
    # forward: tap (3 flops a component) and accumulation (2, or 8 complex); adjoint: two scattered
    # products, the tap, and the slope in the delay and position sums
    flops = units * (14 if cplx else 5)
    total = x + img + geom
    if case["grad"]:
        flops += units * (40 if cplx else 14)
        total += 2 * x + img + 4 * (2 * V * E + 3 * V + 3 * C)
    return {"bytes": int(total), "flops": int(flops)}


# --------------------------------------------------------------- tolerance ---
def tolerance(case):
    """About four times the distance measured between the results and `exact`."""
    if case["kind"] == "select":
        return "exact"
    if case["kind"] == "rank":
        # rounding of the Gram matrix tilts the weakest removed component into the rest: the
        # distance grows 4x with each further component (1.2e-3 at five, 5e-7 to 5e-6 at one)
        return {"rel": (1e-10 if case["dtype"] == "f64" else 2e-5 * 4.0 ** (case["start"] - 1))}
    if case["grad"]:
        # a delay rounded across a sample boundary takes the neighbouring slope: the delay and
        # position gradients are 3e-3 to 9e-3 from float64
        return {"rel": 3.5e-2}
    # float32 delays of up to N samples: 1.5e-5 at 512 samples, 4.6e-5 at 1536, 1.3e-4 at 4096,
    # and the phase of IQ data turns by wavenum times the delay's rounding (2.1e-4 at 2048)
    return {"rel": 1.3e-7 * case["N"] * (1 + 1.5 * abs(case.get("wavenum", 0.0)))}


# ------------------------------------------------------------------- exact ---
def exact(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "select":
        d = prepare(case, seed)
        order = d["weights"].double().sort(dim=0, descending=True, stable=True)[1][: case["k"]]
        return order.int(), d["weights"].gather(0, order), d["offsets"].gather(0, order)
    if case["kind"] == "rank":
        x = _ensemble(case, seed, dev)
        a = x.to(torch.complex128 if x.is_complex() else torch.float64)
        u = torch.linalg.eigh(a @ a.mH)[1].flip(1)[:, : case["start"]]
        return a - u @ (u.mH @ a)
    return _exact_das(case, _das_inputs(case, seed, dev))


def _exact_das(case, d):
    """Delay-and-sum and its gradients in float64, channel by channel."""
    x, src, dst = d["x"], d["srcpos"].double(), d["dstpos"].double().reshape(-1, 3)
    B, C, S, N = x.shape
    V, E = dst.shape[0], d["offsets"].shape[0]
    ofs, w = d["offsets"].double().reshape(E, V), d["weights"].double().reshape(E, V)
    ev = d["idx"].long().reshape(E, V) if "idx" in d else torch.arange(S, device=x.device)[:, None].expand(E, V)
    cplx, wn = x.is_complex(), case.get("wavenum", 0.0)
    wide = torch.complex128 if cplx else torch.float64
    out = torch.zeros(B, V, dtype=wide, device=x.device)
    grad = case["grad"]
    if grad:
        g = d["gout"].to(wide).reshape(B, V)
        gx = torch.zeros(B, C, S * N, dtype=wide, device=x.device)
        gsrc, gdst, gofs, gw = (torch.zeros_like(t) for t in (src, dst, ofs, w))
    step = max(1, (48 << 20) // (E * B))
    for c in range(C):
        rows = x[:, c].reshape(B, S * N).to(wide)
        for v0 in range(0, V, step):
            at = slice(v0, min(V, v0 + step))
            diff = dst[at] - src[c]
            r = diff.norm(dim=-1).clamp_min(math.sqrt(1e-7))
            tau = ofs[:, at] + r
            k = tau.floor()
            t = tau - k
            ok = (k >= 0) & (k < N - 1)
            if "srcdir" in d:
                n = d["srcdir"][c].double()
                ok &= ((diff @ n[:3]) / r > n[3])[None]
            lin = ev[:, at] * N + torch.where(ok, k, 0.0).long()
            x0, x1 = rows[:, lin], rows[:, lin + 1]          # (B, E, V)
            slope = (x1 - x0) * ok
            tap = x0 * ok + t * slope
            rot = torch.polar(torch.ones_like(tau), wn * tau) if cplx else None
            a = w[:, at] * rot if cplx else w[:, at]
            out[:, at] += (a * tap).sum(dim=1)
            if not grad:
                continue
            gv = g[:, at].conj()[:, None] if cplx else g[:, at][:, None]
            if cplx:
                gw[:, at] += (gv * rot * tap).real.sum(dim=0)
                q = (gv * a * (1j * wn * tap + slope)).real.sum(dim=0)
            else:
                gw[:, at] += (gv * tap).sum(dim=0)
                q = (gv * a * slope).sum(dim=0)
            gofs[:, at] += q
            p = (q.sum(dim=0) / r)[:, None] * diff
            gdst[at] += p
            gsrc[c] -= p.sum(dim=0)
            s = (a.conj() if cplx else a) * g[:, at][:, None] * ok     # (B, E, V)
            flat = lin.reshape(-1)
            gx[:, c].index_add_(1, flat, (s * (1 - t)).reshape(B, -1))
            gx[:, c].index_add_(1, flat + 1, (s * t).reshape(B, -1))
    shape = d["dstpos"].shape[:-1]
    out = out.reshape(B, *shape)
    if not grad:
        return out
    return [out, gx.reshape(x.shape), gsrc, gdst.reshape(*shape, 3), gofs.reshape(E, *shape), gw.reshape(E, *shape)]
