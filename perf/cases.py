"""Performance cases of the X-engine: the work its users have it do.

Five kinds of call, each through the public entry points of
`daqiri-mixer_b200/mixer.py` (the ctypes binding of include/mixer.h):

  step         one burst of wire-format packets through corner_turn and
               xcorr_tri into a caller-owned cube: int64 accumulation (mode
               "acc64"), int32 accumulation followed by the exact flush
               ("flush"), or an int32 store ("store32")
  corner_turn  the corner-turn alone, for callers that keep the int8 planes
  dump_cycle   an array context integrating one dump: reset, correlate the
               dump's packets in chunks of max_heaps, FP32 dump cube and image
  monitor      output of an integrated cube: FP32 dump record, exact gridding,
               FFT image with per-channel extrema
  receive      the live receiver: packets in pinned host memory, int64
               accumulation, delta image back in pinned host memory
  batch        uneven arrays in one persistent launch of a kept plan

Packets hold complex int8 samples: three point sources plus Gaussian noise, or
uniform integers in [-127, 127] (sigma 0).  All of it is made with torch from
the seed; the 64-bit values in exact() use torch alone.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "daqiri-mixer_b200"))
import mixer  # noqa: E402

HDR = 64                # packet header bytes
DEV = "cuda"
MODES = {"store32": mixer.VIS_STORE_I32, "flush": mixer.VIS_ACC_I32, "acc64": mixer.VIS_ACC_I64}


def step(name, nant, nch, tpkt, nheaps, side, mode="acc64", sigma=8.0):
    return dict(name=name, kind="step", nant=nant, nch=nch, tpkt=tpkt, nheaps=nheaps, side=side,
                mode=mode, sigma=sigma)


def listed():
    return [
        # The smallest call: one short sub-integration (K 256) of a 64-element array with few
        # channels, where launches and latency count.
        step("step_64x16_k256", 64, 16, 32, 8, 8, sigma=12.0),
        # One V-update of the reference's receiver: 256 elements, 128 channels, HBATCH 32 heaps.
        step("vupdate_256x128_k1024", 256, 128, 32, 32, 16, sigma=16.0),
        # A ragged array (element count no multiple of the GEMM's 128) in the reference's two-step
        # integration: int32 accumulation, then the exact int64 flush.
        step("flush_200x128_k1536", 200, 128, 32, 48, 16, mode="flush", sigma=12.0),
        # One sub-integration of the 1024-element array, integrated on its own.
        step("step_1024x256_k1024", 1024, 256, 16, 64, 32),
        # The benchmark's streaming step: 32 sub-integrations of the 1024-element array at once.
        step("stream_1024x256_k32768", 1024, 256, 16, 2048, 32),
        # One sub-integration of the 4096-element array, full-range int8.
        step("step_4096x64_k2048", 4096, 64, 64, 32, 64, sigma=0.0),
        # A burst cut short by a lost packet: odd heap count, odd element count, planes kept.
        dict(name="corner_turn_300x128_h45", kind="corner_turn", nant=300, nch=128, tpkt=32,
             nheaps=45, side=20, sigma=12.0),
        # One dump of the reference's own array: 64 sub-integrations of K 256 through the context
        # with its default chunk of 32 heaps, then dump and image.
        dict(name="dump_cycle_256x128", kind="dump_cycle", nant=256, nch=128, tpkt=32, nheaps=512,
             max_heaps=32, side=16, grid=32, sigma=16.0),
        # Output products of the 1024-element array: 2.1 GB dump record and 64 x 64 images.
        dict(name="monitor_1024x256_g64", kind="monitor", nant=1024, nch=256, side=32, grid=64),
        # The live receiver, host memory to host memory, one V-update at a time.
        dict(name="receive_256x128_k1024", kind="receive", nant=256, nch=128, tpkt=32, nheaps=32,
             side=16, grid=32, sigma=16.0),
        # Many small uneven arrays in one launch.
        dict(name="batch_48_small", kind="batch", arrays=48, nmax=256, cmax=64, kmax=4096, subs=1,
             draw=20261203),
        # Uneven arrays of every size, two sub-integrations each.
        dict(name="batch_12_mixed", kind="batch", arrays=12, nmax=1024, cmax=512, kmax=4096, subs=2,
             draw=20261203),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(nant):
    return max(1, math.isqrt(nant))


def _grid(nant, side):
    g = 32
    while g < 2 * max(side, -(-nant // side)) and g < 128:
        g *= 2
    return g


def draw(rng):
    """One more case of the same kinds: sizes over the logarithm of their range, odd ones too."""
    kind = rng.choice(["step", "step", "step", "corner_turn", "dump_cycle", "monitor", "receive",
                       "batch"])
    if kind == "batch":
        small = rng.random() < 0.5
        return dict(kind=kind, arrays=rng.randint(4, 48 if small else 12), nmax=256 if small else 1024,
                    cmax=64 if small else 512, kmax=rng.choice([1024, 2048, 4096]),
                    subs=rng.choice([1, 2]), draw=rng.randrange(1 << 30))
    tpkt = rng.choice([16, 32, 48, 64])
    nant = _log(rng, 24, 1500)
    if rng.random() < 0.3:
        nant = max(32, nant // 32 * 32)
    nch = max(4, 4096 // tpkt // rng.choice([1, 1, 2, 4]))
    nheaps = max(1, _log(rng, 128, 16384) // tpkt)
    sigma = rng.choice([0.0, 8.0, 12.0, 16.0])
    # at most 4 GB of packets and 4 GB of cube
    while nant * nant * nch * 8 > 4e9:
        nch //= 2
    nheaps = max(1, min(nheaps, int(4e9 / (nant * 2 * nch * tpkt))))
    side = _side(nant)
    base = dict(kind=kind, nant=nant, nch=nch, side=side)
    if kind == "monitor":
        return dict(base, grid=_grid(nant, side))
    base.update(tpkt=tpkt, nheaps=nheaps, sigma=sigma)
    if kind == "step":
        base["mode"] = rng.choice(["acc64", "acc64", "flush", "store32"])
    if kind == "dump_cycle":
        base.update(max_heaps=min(nheaps, rng.choice([8, 32, 64])), grid=_grid(nant, side))
    if kind == "receive":
        base.update(nheaps=max(1, min(nheaps, int(4e8 / (nant * 2 * nch * tpkt)))),
                    grid=_grid(nant, side))
    return base


# ---- inputs -----------------------------------------------------------------

def _stride(case):
    return HDR + 2 * case["nch"] * case["tpkt"]


def _sky(case, seed):
    """[nch][nant] complex amplitudes of three sources, unit-spaced array side elements wide."""
    g = torch.Generator().manual_seed(seed)
    lm = (torch.rand(3, 2, generator=g, dtype=torch.float64) * 2 - 1) * 0.4
    a = torch.arange(case["nant"], dtype=torch.float64)
    x, y = a % case["side"], torch.div(a, case["side"], rounding_mode="floor")
    f = 1 + torch.arange(case["nch"], dtype=torch.float64) / case["nch"]
    sky = torch.zeros(case["nch"], case["nant"], dtype=torch.complex128)
    for s, amp in enumerate((4.0, 2.0, 1.0)):
        ph = -2 * math.pi * f[:, None] * (x * lm[s, 0] + y * lm[s, 1])[None, :]
        sky += amp * torch.polar(torch.ones_like(ph), ph)
    return sky.to(DEV)


def _packets(case, seed):
    """uint8 [nheaps][nant][stride]: packet p = h * nant + a carries big-endian seq p at byte 48,
    then planar re [nch][tpkt] | im [nch][tpkt]."""
    nh, na, nch, tp = case["nheaps"], case["nant"], case["nch"], case["tpkt"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    pk = torch.zeros(nh, na, _stride(case), dtype=torch.uint8, device=DEV)
    seq = torch.arange(nh * na, dtype=torch.int64, device=DEV).view(nh, na)
    for b in range(4):
        pk[:, :, 48 + b] = ((seq >> (24 - 8 * b)) & 255).to(torch.uint8)
    if case["sigma"] > 0:
        sky = _sky(case, seed).T                                 # [nant][nch]
        mean = torch.stack((sky.real, sky.imag), 1).float()      # [nant][2][nch]
        mean = mean.view(1, na, 2, nch, 1)
    per = max(1, (1 << 27) // (na * 2 * nch * tp))
    for h in range(0, nh, per):
        n = min(per, nh - h)
        if case["sigma"] > 0:
            v = torch.randn(n, na, 2, nch, tp, device=DEV, generator=g).mul_(case["sigma"]).add_(mean)
            v = v.round_().clamp_(-127, 127).to(torch.int8)
        else:
            v = torch.randint(-127, 128, (n, na, 2, nch, tp), device=DEV, generator=g,
                              dtype=torch.int8)
        pk[h:h + n, :, HDR:] = v.view(n, na, -1).view(torch.uint8)
    return pk


def _cube(case, seed):
    """An integrated cube, tile-packed int64: Hermitian, large auto-correlations, zero padding."""
    na, nch = case["nant"], case["nch"]
    nb = -(-na // 128)
    g = torch.Generator(device=DEV).manual_seed(seed)
    vis = torch.empty(nch, nb * (nb + 1) // 2, 2, 128, 128, dtype=torch.int64, device=DEV)
    for i in range(nb):
        for j in range(i + 1):
            v = (torch.randn(nch, 2, 128, 128, device=DEV, generator=g) * 3e6).round_().to(torch.int64)
            if i == j:
                v[:, 0] = v[:, 0] + v[:, 0].transpose(1, 2)
                v[:, 1] = v[:, 1] - v[:, 1].transpose(1, 2)
                v[:, 0].diagonal(dim1=1, dim2=2).abs_().add_(4 << 30)
            v[..., max(0, na - 128 * i):] = 0                    # rows m past the last element
            v[:, :, max(0, na - 128 * j):] = 0                   # columns n
            vis[:, i * (i + 1) // 2 + j] = v
    return vis


def _batch_shapes(case):
    import random
    r = random.Random(case["draw"])
    return [(r.choice(range(64, case["nmax"] + 1, 32)), r.choice(range(16, case["cmax"] + 1, 16)),
             r.choice(range(256, case["kmax"] + 1, 256))) for _ in range(case["arrays"])]


def _batch_planes(case, seed, p, shape):
    n, c, k = shape
    g = torch.Generator(device=DEV).manual_seed(seed * 1000 + p)
    pl = torch.empty(2, c, n, k * case["subs"], dtype=torch.int8, device=DEV)
    per = max(1, (1 << 27) // (n * k * case["subs"]))
    for q in range(2):
        for c0 in range(0, c, per):
            v = pl[q, c0:c0 + per]
            v.copy_(torch.randn(v.shape, device=DEV, generator=g).mul_(12).round_().clamp_(-127, 127))
    return pl


def _vis(nant, nch, dtype=torch.int64):
    return torch.zeros(mixer.vis_elems(nant, nch), dtype=dtype, device=DEV)


def _planes(case):
    kt = -(-case["nheaps"] * case["tpkt"] // 128) * 128
    return torch.zeros(2, case["nch"], case["nant"], kt, dtype=torch.int8, device=DEV)


def _image_out(case, **kw):
    g, c = case["grid"], case["nch"]
    return (torch.zeros(c, g, g, **kw), torch.zeros(c, **kw), torch.zeros(c, **kw))


def _context(case, max_heaps):
    return mixer.ArrayContext(nant=case["nant"], nch=case["nch"], tpkt=case["tpkt"],
                              ksub=case["tpkt"], side_x=case["side"], grid=case["grid"],
                              pkt_stride=_stride(case), hdr_bytes=HDR, max_heaps=max_heaps)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("step", "corner_turn"):
        s["pk"] = _packets(case, seed)
        s["planes"] = _planes(case)
        s["seq_errors"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        s["err"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        if kind == "step":
            mode = case["mode"]
            s["vis"] = _vis(case["nant"], case["nch"], torch.int64 if mode == "acc64" else torch.int32)
            if mode == "flush":
                s["vis64"] = _vis(case["nant"], case["nch"])
    elif kind == "dump_cycle":
        s["pk"] = _packets(case, seed)
        s["ctx"] = _context(case, case["max_heaps"])
        s["dump"] = torch.zeros(case["nch"], 2, case["nant"], case["nant"], device=DEV)
        s["image"] = _image_out(case, device=DEV)
    elif kind == "receive":
        s["pk"] = _packets(case, seed).cpu().pin_memory()
        s["ctx"] = _context(case, case["nheaps"])
        s["image"] = _image_out(case, pin_memory=True)
    elif kind == "monitor":
        g, c = case["grid"], case["nch"]
        s["vis"] = _cube(case, seed)
        s["dump"] = torch.zeros(c, 2, case["nant"], case["nant"], device=DEV)
        s["grid"] = torch.zeros(c, g, g, 2, dtype=torch.int64, device=DEV)
        s["image"] = _image_out(case, device=DEV)
    else:
        s["vis"], probs = [], []
        for p, (n, c, k) in enumerate(_batch_shapes(case)):
            pl = _batch_planes(case, seed, p, (n, c, k))
            s["vis"].append(_vis(n, c))
            probs.append(dict(planes=pl, nant=n, nch=c, kt=k * case["subs"], mode=mixer.VIS_ACC_I64,
                              vis=s["vis"][-1]))
        s["batch"] = mixer.Batch(probs)
    return s


# ---- one pass ---------------------------------------------------------------

def _corner_turn(s):
    c = s["case"]
    mixer.corner_turn(s["pk"], _stride(c), HDR, c["nant"], c["nch"], c["tpkt"], c["nheaps"], 0,
                      s["planes"], s["planes"].shape[3], 0, s["seq_errors"], s["err"])


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "corner_turn":
        _corner_turn(s)
        return s["planes"], s["seq_errors"]
    if kind == "step":
        _corner_turn(s)
        mode = c["mode"]
        mixer.xcorr_tri(s["planes"], c["nant"], c["nch"], s["planes"].shape[3], 0,
                        c["nheaps"] * c["tpkt"], MODES[mode], s["vis"], s["err"])
        if mode != "flush":
            return s["vis"], s["seq_errors"], s["err"]
        mixer.vis_flush(s["vis"], s["vis64"], s["vis"].numel())
        return s["vis64"], s["vis"], s["seq_errors"], s["err"]
    if kind == "dump_cycle":
        ctx, (img, vmax, vmin) = s["ctx"], s["image"]
        ctx.reset()
        ctx.correlate(s["pk"], c["nheaps"], 0)
        ctx.dump(s["dump"])
        ctx.image(img, vmax, vmin)
        return s["dump"], img, vmax, vmin
    if kind == "receive":
        ctx, (img, vmax, vmin) = s["ctx"], s["image"]
        ctx.correlate(s["pk"], c["nheaps"], 0, on_device=False)
        ctx.image(img, vmax, vmin, delta=True, on_device=False)
        return img, vmax, vmin
    if kind == "monitor":
        img, vmax, vmin = s["image"]
        mixer.vis_dump_f32(s["vis"], c["nant"], c["nch"], s["dump"])
        mixer.grid(s["vis"], c["nant"], c["nch"], c["side"], c["grid"], s["grid"])
        mixer.image_fft(s["grid"], c["nch"], c["grid"], img, vmax, vmin)
        return s["dump"], s["grid"], img, vmax, vmin
    s["batch"].run()
    return s["vis"]


# ---- what a pass cannot do without ------------------------------------------

def _cube_bytes(nant, nch, each=8):
    return mixer.vis_elems(nant, nch) * each


def _tri_ops(nant, nch, k):
    return 8.0 * nant * (nant + 1) / 2 * nch * k


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for n, c, k in _batch_shapes(case):
            b += 2.0 * c * n * k * case["subs"] + 2.0 * _cube_bytes(n, c)
            f += _tri_ops(n, c, k * case["subs"])
        return {"bytes": b, "flops": f}
    n, c = case["nant"], case["nch"]
    image = 4.0 * c * case.get("grid", 0) ** 2 + 8.0 * c
    fft = 10.0 * c * case.get("grid", 0) ** 2 * math.log2(max(2, case.get("grid", 0)))
    if kind == "monitor":
        return {"bytes": _cube_bytes(n, c) + 8.0 * c * n * n + 16.0 * c * case["grid"] ** 2 + image,
                "flops": 4.0 * c * n * n + fft}
    packets = float(case["nheaps"]) * n * _stride(case)
    k = case["nheaps"] * case["tpkt"]
    if kind == "corner_turn":
        return {"bytes": packets + 2.0 * c * n * k, "flops": 0.0}
    ops = _tri_ops(n, c, k)
    if kind == "dump_cycle":
        return {"bytes": packets + 8.0 * c * n * n + image, "flops": ops + fft}
    if kind == "receive":
        return {"bytes": packets + 2.0 * _cube_bytes(n, c) + image, "flops": ops + fft}
    cube = {"acc64": 2.0 * _cube_bytes(n, c), "store32": _cube_bytes(n, c, 4),
            "flush": 2.0 * _cube_bytes(n, c)}[case["mode"]]
    return {"bytes": packets + cube, "flops": ops}


# ---- the same in 64 bits ----------------------------------------------------

def _samples(case, pk, c):
    """re, im float64 [nant][K] of channel c."""
    n, tp = case["nant"], case["tpkt"]
    v = pk[:, :, HDR:].view(torch.int8).view(case["nheaps"], n, 2, case["nch"], tp)[:, :, :, c]
    v = v.permute(2, 1, 0, 3).reshape(2, n, -1).double()     # [plane][nant][heap * tpkt]
    return v[0], v[1]


def _correlate(re, im):
    """X X^H: exact in float64 (every partial sum is an integer below 2^53)."""
    return re @ re.T + im @ im.T, im @ re.T - re @ im.T


def _pack(vr, vi, out):
    """Tile-packed lower triangle of one channel: out [ntiles][2][128 columns][128 rows]."""
    nb = -(-vr.shape[0] // 128)
    for p, v in enumerate((vr, vi)):
        full = torch.zeros(nb * 128, nb * 128, dtype=v.dtype, device=v.device)
        full[:v.shape[0], :v.shape[1]] = v
        t = 0
        for i in range(nb):
            for j in range(i + 1):
                out[t, p] = full[128 * i:128 * i + 128, 128 * j:128 * j + 128].T
                t += 1


def _unpack(vis, nant):
    """Full square [nch][2][nant][nant] float64 of a tile-packed cube."""
    nch, nb = vis.shape[0], -(-nant // 128)
    full = torch.zeros(nch, 2, nb * 128, nb * 128, dtype=torch.float64, device=vis.device)
    for i in range(nb):
        for j in range(i + 1):
            v = vis[:, i * (i + 1) // 2 + j].double().transpose(2, 3)
            full[:, :, 128 * i:128 * i + 128, 128 * j:128 * j + 128] = v
            if i != j:
                full[:, 0, 128 * j:128 * j + 128, 128 * i:128 * i + 128] = v[:, 0].transpose(1, 2)
                full[:, 1, 128 * j:128 * j + 128, 128 * i:128 * i + 128] = -v[:, 1].transpose(1, 2)
    return full[:, :, :nant, :nant]


def _grid_image(case, vr, vi, grid, img):
    """Grids one channel's full square (integers in float64: exact) and images it."""
    n, g, sx = case["nant"], case["grid"], case["side"]
    a = torch.arange(n, device=vr.device)
    x, y = a % sx, torch.div(a, sx, rounding_mode="floor")
    cell = ((y[:, None] - y[None, :]) % g * g + (x[:, None] - x[None, :]) % g).reshape(-1)
    for p, v in enumerate((vr, vi)):
        s = torch.zeros(g * g, dtype=torch.float64, device=vr.device)
        grid[..., p] = s.index_add_(0, cell, v.reshape(-1)).view(g, g)
    f = torch.fft.fft2(torch.complex(grid[..., 0].contiguous(), grid[..., 1].contiguous()))
    img.copy_(torch.fft.fftshift(f).real)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        if sum(8.0 * n * n * c * k * case["subs"] for n, c, k in shapes) > 4e13:
            return None
        out = []
        for p, (n, c, k) in enumerate(shapes):
            pl = _batch_planes(case, seed, p, (n, c, k))
            nb = -(-n // 128)
            v = torch.zeros(c, nb * (nb + 1) // 2, 2, 128, 128, dtype=torch.float64, device=DEV)
            for ch in range(c):
                _pack(*_correlate(pl[0, ch].double(), pl[1, ch].double()), v[ch])
            out.append(v.reshape(-1).to(torch.int64))
        return out
    n, c = case["nant"], case["nch"]
    nb = -(-n // 128)
    zero = torch.zeros(1, dtype=torch.int32, device=DEV)
    if kind == "monitor":
        full = _unpack(_cube(case, seed), n)
        grid = torch.zeros(c, case["grid"], case["grid"], 2, dtype=torch.float64, device=DEV)
        img = torch.zeros(c, case["grid"], case["grid"], dtype=torch.float64, device=DEV)
        for ch in range(c):
            _grid_image(case, full[ch, 0], full[ch, 1], grid[ch], img[ch])
        return full, grid.to(torch.int64), img, img.amax((1, 2)), img.amin((1, 2))
    k = case["nheaps"] * case["tpkt"]
    if kind != "corner_turn" and 8.0 * n * n * c * k > 4e13:
        return None
    pk = _packets(case, seed)
    if kind == "corner_turn":
        planes = _planes(case)
        for ch in range(c):
            re, im = _samples(case, pk, ch)
            planes[0, ch, :, :k], planes[1, ch, :, :k] = re.to(torch.int8), im.to(torch.int8)
        return planes, zero
    if kind == "step":
        v = torch.zeros(c, nb * (nb + 1) // 2, 2, 128, 128, device=DEV,
                        dtype=torch.int32 if case["mode"] == "store32" else torch.int64)
        for ch in range(c):
            _pack(*_correlate(*_samples(case, pk, ch)), v[ch])
        v = v.reshape(-1)
        if case["mode"] == "flush":
            return v, torch.zeros(v.numel(), dtype=torch.int32, device=DEV), zero, zero
        return v, zero, zero
    g = case["grid"]
    grid = torch.zeros(g, g, 2, dtype=torch.float64, device=DEV)
    img = torch.zeros(c, g, g, dtype=torch.float64, device=DEV)
    dump = torch.zeros(c, 2, n, n, dtype=torch.float64, device=DEV) if kind == "dump_cycle" else None
    for ch in range(c):
        vr, vi = _correlate(*_samples(case, pk, ch))
        _grid_image(case, vr, vi, grid, img[ch])
        if dump is not None:
            dump[ch, 0], dump[ch, 1] = vr, vi
    vmax, vmin = img.amax((1, 2)), img.amin((1, 2))
    return (dump, img, vmax, vmin) if dump is not None else (img, vmax, vmin)
