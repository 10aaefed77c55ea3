"""The work a user of lizard_gb300 has it do, as cases that can be timed: the decoder batch, the receiver on one frame
and on batches, the multi-stream tick, the transform alone, the registration from the anchors, its refinement by the
adjoint, the sender and the camera develop. Each case is a dict of plain values; prepare() makes its inputs on the GPU
from a seed alone, run() is one pass through the public entry points.

Captured frames are painted here (torch, in double where it matters): seeded blocks through the format's code, bit
map and whitening onto the QPSK spectrum, its inverse transform clipped to a page with the border's cells and the
anchors, seen by a pinhole camera with radial distortion, blurred in linear light, with sensor noise, in 8 bits."""
import ctypes
import functools
import math

import numpy as np
import torch

import lizard_gb300 as lz

# The rate mix of a frame's blocks (the format's profile) and the multi-stream tick's formats (n, sub-channels, ring
# span), smallest picture first.
MIX = ((6, 0.39), (4, 0.26), (3, 0.15), (2, 0.20))
TICK_FORMATS = ((384, 64, 128), (768, 320, 128), (1152, 720, 256), (1536, 1024, 256), (1536, 1024, 512))
# Sub-channels that fill each picture size as the largest fills its own.
SUBCH = {384: 80, 512: 128, 768: 320, 1024: 560, 1152: 720, 1280: 880, 1536: 1024}
RGBA8, RAW10, RAW12, P010 = "rgba8", "raw10", "raw12", "p010"
RAW_CODE = {P010: 0x36, RAW10: 0x25, RAW12: 0x26}


def listed():
    return [
        # the decoder on a handful of codewords: one small frame's blocks handed over by a program with its own demodulator
        dict(name="ldpc_37", kind="ldpc", count=37, rate=0, lo_db=1.0, hi_db=4.0, memory="device"),
        # the decoder's batch: every code in the profile's mix over the whole waterfall, soft values resident on the device
        dict(name="ldpc_65536", kind="ldpc", count=65536, rate=0, lo_db=1.0, hi_db=4.0, memory="device"),
        # a phone's preview frame: the smallest picture, one frame a call, where latency counts
        dict(name="rx_384_1", kind="rx", n=384, subch=64, span=128, w=1280, h=720, frames=1, k1=0.0, blur=0.0, noise=2.0,
             read="decode", graph=False),
        # one 4K frame of the largest picture: a receiver that decodes each frame as it comes
        dict(name="rx_1536_1", kind="rx", n=1536, subch=1024, span=128, w=3840, h=2160, frames=1, k1=0.0, blur=0.0, noise=2.0,
             read="decode", graph=False),
        # a ragged batch of a middle size through a lens, odd frame width and count
        dict(name="rx_1152_13", kind="rx", n=1152, subch=720, span=128, w=1917, h=1439, frames=13, k1=0.02, blur=0.7, noise=3.0,
             read="decode", graph=False),
        # an offline decode of a recording: 32 frames of 4K a call, replayed from a graph
        dict(name="rx_1536_32", kind="rx", n=1536, subch=1024, span=128, w=3840, h=2160, frames=32, k1=0.0, blur=0.0, noise=2.0,
             read="decode", graph=True),
        # a tick of 32 camera streams of five formats: registration from the anchors, then the engine
        dict(name="tick_32", kind="tick", w=3840, h=2160, c0=10, c1=8, c2=6, c3=5, c4=3, blur=1.2, noise=3.0),
        # the transform alone on picture grids (a program with its own sampler)
        dict(name="spectrum_768_64", kind="spectrum", n=768, subch=320, span=128, frames=64, noise=3.0),
        # the registration from the anchors on frames a finder's corners gave
        dict(name="register_64", kind="register", n=1536, subch=1024, span=128, w=1920, h=1080, frames=64, blur=1.2, noise=3.0),
        # the registration refined through the adjoint of the receiver's front (Gauss-Newton, three steps)
        dict(name="field_24", kind="field", n=1536, subch=1024, span=128, w=1920, h=1080, frames=24, blur=1.2, noise=3.0),
        # the sender: pages of the largest picture
        dict(name="encode_32", kind="encode", n=1536, subch=1024, span=128, frames=32),
        # camera ingest in front of the receiver: 4K RAW10 frames developed to luma
        dict(name="develop_16", kind="ingest", fmt=RAW10, w=3840, h=2160, frames=16, bin=1),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ldpc", "ldpc", "rx", "rx", "rx", "tick", "spectrum", "register", "field", "encode", "ingest"])
    n = rng.choice(lz.PICTURES)
    span = rng.choice([128, 128, 256])
    if kind == "ldpc":
        lo = rng.uniform(1.0, 3.5)
        return dict(kind=kind, count=_log_int(rng, 1, 65536), rate=rng.choice([0, 0, 0, 6, 4, 3, 2]), lo_db=round(lo, 2),
                    hi_db=round(rng.uniform(lo, 4.0), 2), memory=rng.choice(["device", "device", "device", "pinned"]))
    if kind == "rx":
        w, h = rng.choice([(1280, 720), (1920, 1080), (2560, 1440), (3840, 2160)] if n <= 512 else
                          [(1920, 1440), (2560, 1440), (3840, 2160)])
        return dict(kind=kind, n=n, subch=SUBCH[n], span=span, w=w - rng.randrange(0, 9), h=h - rng.randrange(0, 9),
                    frames=_log_int(rng, 1, 32), k1=round(rng.uniform(-0.03, 0.03), 4), blur=round(rng.uniform(0.0, 1.0), 2),
                    noise=round(rng.uniform(1.0, 4.0), 2), read=rng.choice(["decode", "decode", "decode", "exact"]),
                    graph=rng.choice([False, True]))
    if kind == "tick":
        c = [rng.randrange(1, 11), rng.randrange(1, 9), rng.randrange(1, 7), rng.randrange(1, 6), rng.randrange(1, 4)]
        return dict(kind=kind, w=3840, h=2160, c0=c[0], c1=c[1], c2=c[2], c3=c[3], c4=c[4], blur=round(rng.uniform(0.5, 1.5), 2),
                    noise=round(rng.uniform(2.0, 4.0), 2))
    if kind == "spectrum":
        return dict(kind=kind, n=n, subch=SUBCH[n], span=span, frames=_log_int(rng, 1, 64 if n <= 768 else 24), noise=round(rng.uniform(1.0, 4.0), 2))
    if kind == "register":
        return dict(kind=kind, n=1536, subch=1024, span=128, w=1920, h=1080, frames=_log_int(rng, 1, 64),
                    blur=round(rng.uniform(0.5, 2.0), 2), noise=round(rng.uniform(2.0, 4.0), 2))
    if kind == "field":
        n = rng.choice([768, 1152, 1536])
        return dict(kind=kind, n=n, subch=SUBCH[n], span=128, w=1920, h=1080, frames=_log_int(rng, 1, 24),
                    blur=round(rng.uniform(0.5, 2.0), 2), noise=round(rng.uniform(2.0, 4.0), 2))
    if kind == "encode":
        return dict(kind=kind, n=n, subch=SUBCH[n], span=span, frames=_log_int(rng, 1, 32))
    fmt, bin_ = rng.choice([(RGBA8, 1), (RAW10, 1), (RAW10, 2), (RAW12, 1), (RAW12, 2), (P010, 1)])
    w, h = rng.choice([(1280, 720), (1920, 1080), (3840, 2160)])
    return dict(kind="ingest", fmt=fmt, w=w, h=h - 2 * rng.randrange(0, 5), frames=_log_int(rng, 1, 16), bin=bin_)


# ---------------------------------------------------------------- blocks, pictures and cameras

@functools.lru_cache(maxsize=None)
def _format(n, subch, span):
    return lz.Format(n, subch, span)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _generator(*seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence(seed).generate_state(1, np.uint64)[0] >> 2))
    return g


def _block_bits(rng, count):
    """count blocks (a 4-byte id, 472 random bytes) and their 3840 bits each: the bytes, then their CRC-32C."""
    rows = rng.integers(0, 256, (count, lz.BLOCK_BYTES), dtype=np.uint8)
    rows[:, :4] = np.arange(count, dtype="<u4").view(np.uint8).reshape(count, 4)
    crc = np.array([lz.crc32c(r.tobytes()) for r in rows], ">u4").view(np.uint8).reshape(count, 4)
    return rows, np.unpackbits(np.concatenate([rows, crc], axis=1), axis=1)


def _codewords(rate, bits):
    data = np.zeros((bits.shape[0], lz.CODE_K[rate]), np.uint8)
    data[:, :lz.INFO_BITS] = bits
    return lz.ldpc_encode_many(rate, data)


def _picture(fmt, rng, parity):
    """The n x n picture of a frame of random blocks, 0..1 (float32, on the GPU)."""
    _, bits = _block_bits(rng, fmt.blocks)
    slot = fmt.white.copy()
    for t in range(fmt.tiers):
        rate, _, nb = fmt.tier[t]
        nt = lz.CODE_NT[rate]
        idx = np.nonzero(fmt.block_tier == t)[0]
        seg = np.empty((idx.size, nb), np.uint8)
        seg[:, :nt] = _codewords(rate, bits[idx])[:, fmt.perm[t]]
        seg[:, nt:] = ((parity >> (idx & 1)) & 1)[:, None]
        at = fmt.block_slot[idx][:, None] + np.arange(nb)[None, :]
        slot[at] ^= seg
    a = 0.70710678
    sym = torch.from_numpy(slot.reshape(-1, 2).astype(np.float64)).cuda()
    sym = torch.complex(a - 2 * a * sym[:, 0], a - 2 * a * sym[:, 1])
    n = fmt.n
    S = torch.zeros(n * n, dtype=torch.complex128, device="cuda")
    S[torch.from_numpy(fmt.tix()).cuda()] = sym
    z = torch.fft.ifft2(S.view(n, n)).real * (2.0 * n * n)
    lim = 4.0 * math.sqrt(0.5 * fmt.subch * lz.SUB)
    return (0.5 + z.clamp(-lim, lim) * (0.5 / lim)).float()


def _view(rng, span, w, h, side_px, rot_deg, tilt_deg, scale):
    """A pinhole camera's homography, layout modules to image pixels, the layout whole inside the frame."""
    side = span + 30
    for k in range(200):
        rot, tilt = np.deg2rad(rng.uniform(-rot_deg, rot_deg)), np.deg2rad(rng.uniform(-tilt_deg, tilt_deg))
        phi, s = rng.uniform(0, np.pi), side_px * rng.uniform(*scale) / side * 0.995 ** k
        ax = np.array([np.cos(phi), np.sin(phi), 0.0])
        K = np.array([[0, -ax[2], ax[1]], [ax[2], 0, -ax[0]], [-ax[1], ax[0], 0]])
        R = np.array([[np.cos(rot), -np.sin(rot), 0], [np.sin(rot), np.cos(rot), 0], [0, 0, 1]]) @ (
            np.eye(3) + np.sin(tilt) * K + (1 - np.cos(tilt)) * (K @ K))
        M = np.array([[w, 0, w / 2], [0, w, h / 2], [0, 0, 1.0]]) @ np.column_stack([R[:, 0], R[:, 1], [0, 0, w]])
        H = M @ np.array([[s, 0, -s * side / 2], [0, s, -s * side / 2], [0, 0, 1]])
        H /= H[2, 2]
        q = H @ np.array([[0, 0, 1], [side, 0, 1], [side, side, 1], [0, side, 1.0]]).T
        u, v = q[0] / q[2], q[1] / q[2]
        if u.min() > 4 and u.max() < w - 5 and v.min() > 4 and v.max() < h - 5:
            return H
    raise ValueError("no view of this layout fits the frame")


def _through_lens(u, v, w, h, k1):
    cx, cy, R2 = w / 2, h / 2, (w * w + h * h) / 4
    g = 1 + k1 * ((u - cx) ** 2 + (v - cy) ** 2) / R2
    return cx + (u - cx) * g, cy + (v - cy) * g


def _mapped(H, k1, w, h, pts):
    """Where the camera sees layout points (k x 2)."""
    q = H @ np.column_stack([pts, np.ones(len(pts))]).T
    return np.column_stack(_through_lens(q[0] / q[2], q[1] / q[2], w, h, k1))


def _anchor_modules(span):
    a = span // 64
    return [math.floor(15 + span * (i + 0.5) / 7 - a / 2 + 0.5) for i in range(7)], a


def _nodes(span):
    side, pos, c = span + 30, [], 3.5
    while c < side - 3.5 - 8:
        pos.append(c)
        c += 16
    return np.array(pos + [side - 3.5])


def _registration(span, H, k1, w, h, mesh):
    """What a receiver holds: the homography through the corners as the camera sees them, then the node mesh: zeros, or
    with mesh the camera's displacements about it."""
    side = span + 30
    src = np.array([[0, 0], [side, 0], [side, side], [0, side]], np.float64)
    A, b = [], []
    for (x, y), (u, v) in zip(src, _mapped(H, k1, w, h, src)):
        A += [[x, y, 1, 0, 0, 0, -u * x, -u * y], [0, 0, 0, x, y, 1, -v * x, -v * y]]
        b += [u, v]
    Hp = np.append(np.linalg.solve(np.array(A), np.array(b)), 1.0)
    pos = _nodes(span)
    if not mesh:
        return np.concatenate([Hp, np.zeros(2 * pos.size ** 2)]).astype(np.float32)
    X, Y = np.meshgrid(pos, pos)
    pts = np.column_stack([X.ravel(), Y.ravel()])
    d = _mapped(H, k1, w, h, pts) - _mapped(Hp.reshape(3, 3), 0.0, w, h, pts)
    return np.concatenate([Hp, d.ravel()]).astype(np.float32)


def _blurred(img, sigma):
    r = max(1, int(3.0 * sigma + 0.5))
    k = np.exp(-0.5 * (np.arange(-r, r + 1) / sigma) ** 2)
    k /= k.sum()
    for dim in (0, 1):
        n = img.shape[dim]
        at = torch.arange(n, device=img.device)
        out = torch.zeros_like(img)
        for j in range(-r, r + 1):
            out += float(k[j + r]) * img.index_select(dim, (at + j).clamp(0, n - 1))
        img = out
    return img


def _captured(picture, kind, span, H, k1, blur, noise, w, h, gen):
    """The 8-bit luma frame (h x w, on the GPU) of a page holding the picture, two by two samples a pixel."""
    n = picture.shape[0]
    scale = n / span
    side = span + 30
    Hi = np.linalg.inv(H)
    m0, a = _anchor_modules(span)
    light = torch.zeros((h, w), device="cuda")
    cx, cy, R2 = w / 2, h / 2, (w * w + h * h) / 4
    for oy in (0.25, 0.75):
        for ox in (0.25, 0.75):
            V = (torch.arange(h, device="cuda", dtype=torch.float32) + oy)[:, None]
            U = (torch.arange(w, device="cuda", dtype=torch.float32) + ox)[None, :]
            u, v = U, V
            for _ in range(6 if k1 else 0):
                g = 1 + k1 * ((u - cx) ** 2 + (v - cy) ** 2) / R2
                u, v = cx + (U - cx) / g, cy + (V - cy) / g
            q = Hi[2, 0] * u + Hi[2, 1] * v + Hi[2, 2]
            mx, my = (Hi[0, 0] * u + Hi[0, 1] * v + Hi[0, 2]) / q, (Hi[1, 0] * u + Hi[1, 1] * v + Hi[1, 2]) / q
            sx, sy = (mx - 15) * scale - 0.5, (my - 15) * scale - 0.5
            x0, y0 = torch.floor(sx), torch.floor(sy)
            fx, fy = sx - x0, sy - y0
            x0, y0 = x0.long(), y0.long()
            xa, xb, ya, yb = x0.remainder(n), (x0 + 1).remainder(n), y0.remainder(n) * n, (y0 + 1).remainder(n) * n
            P = picture.reshape(-1)
            val = (P[ya + xa] * (1 - fx) + P[ya + xb] * fx) * (1 - fy) + (P[yb + xa] * (1 - fx) + P[yb + xb] * fx) * fy
            # the anchors' squares: light middle and rim, a dark ring
            dx, dy = torch.full_like(mx, 2.0), torch.full_like(my, 2.0)
            for m in m0:
                dx = torch.minimum(dx, (mx - (m + a / 2)).abs() / (a / 2))
                dy = torch.minimum(dy, (my - (m + a / 2)).abs() / (a / 2))
            r = torch.maximum(dx, dy)
            val = torch.where(r < 1, ((r < 0.25) | (r >= 0.6)).float(), val)
            # the border's cells outside the picture and its guard
            edge = torch.minimum(torch.minimum(mx, side - mx), torch.minimum(my, side - my))
            cell = kind[my.long().clamp(0, side - 1) * side + mx.long().clamp(0, side - 1)]
            val = torch.where(edge < 12, cell, val)
            val = torch.where(edge < 0, torch.where(edge < -2, 128.0 / 255.0, 1.0), val)
            light += 0.25 * val.clamp(0, 1) ** 2.2
    if blur > 0:
        light = _blurred(light, blur)
    grey = 255.0 * light.clamp(0, 1) ** (1 / 2.2)
    grey += noise * torch.randn(grey.shape, generator=gen, device="cuda")
    return grey.round().clamp(0, 255).to(torch.uint8)


def _cameras(n, subch, span, w, h, frames, k1, blur, noise, seed, side_px, rot=10.0, tilt=10.0, scale=(0.9, 1.05), mesh=True):
    """frames captures (frames x h x w uint8) of up to four distinct pictures, each its own view and noise, and their
    registrations (frames x floats); with them the views and lenses."""
    fmt = _format(n, subch, span)
    rng = np.random.default_rng(seed)
    kind = torch.from_numpy(np.where((lz.layout_kind(span, subch // 16, 30) & 3) == 2, 0.0, 1.0).astype(np.float32).ravel()).cuda()
    pics = [_picture(fmt, rng, k & 3) for k in range(min(frames, 4))]
    luma = torch.empty((frames, h, w), dtype=torch.uint8, device="cuda")
    regs, seen = [], []
    for k in range(frames):
        kk = k1 if k1 is not None else float(rng.uniform(-0.05, 0.05))
        H = _view(rng, span, w, h, side_px, rot, tilt, scale)
        luma[k] = _captured(pics[k % len(pics)], kind, span, H, kk, blur, noise, w, h, _generator(seed, k))
        regs.append(_registration(span, H, kk, w, h, mesh))
        seen.append((H, kk))
    return fmt, luma, torch.from_numpy(np.stack(regs)).cuda(), seen


def _side_px(n, span, h):
    """The layout's side as a camera frames it: no larger than one pixel a sample, inside the frame."""
    return min((span + 30) * n / span, 0.8 * h)


# ---------------------------------------------------------------- the kinds

def _prepare_ldpc(c, seed):
    """Codewords back to back in the profile's mix (rate 0) or of one code, codeword i at an Eb/N0 that steps by half a
    decibel from lo_db to hi_db, BPSK over AWGN, the receiver's int8 soft values. Up to 256 distinct codewords a code."""
    count, rng = c["count"], np.random.default_rng(seed)
    if c["rate"]:
        rates = np.full(count, c["rate"], np.int32)
    else:
        k = [int(count * f) for _, f in MIX[:-1]]
        rates = np.concatenate([np.full(m, r, np.int32) for (r, _), m in zip(MIX, k + [count - sum(k)])])
        rng.shuffle(rates)
    plan = lz.LdpcPlan(rates, 20, 9, 0.95)
    db = np.arange(c["lo_db"], c["hi_db"] + 1e-9, 0.5)
    ebn0 = torch.from_numpy(10.0 ** (db[np.arange(count) % db.size] / 10.0)).float().cuda()
    off = torch.from_numpy(plan.offsets).cuda()
    llr = torch.empty(plan.llr_bytes, dtype=torch.int8, device="cuda")
    gen = _generator(seed)
    for r in (6, 4, 3, 2):
        idx = np.nonzero(rates == r)[0]
        if not idx.size:
            continue
        n, k, nt = lz.CODE_N[r], lz.CODE_K[r], lz.CODE_NT[r]
        _, bits = _block_bits(rng, min(256, idx.size))
        sent = torch.from_numpy(1.0 - 2.0 * _codewords(r, bits).astype(np.float32)).cuda()
        for a in range(0, idx.size, 2048):
            at = torch.from_numpy(idx[a:a + 2048]).cuda()
            sigma2 = 1.0 / (2.0 * (lz.INFO_BITS / nt) * ebn0[at])[:, None]
            y = sent[torch.arange(a, a + at.numel(), device="cuda") % sent.shape[0]]
            y = y + sigma2.sqrt() * torch.randn((at.numel(), n), generator=gen, device="cuda")
            q = (16.0 * y / sigma2).round().clamp(-80, 80).to(torch.int8)
            if nt < n:   # the 7/8 code's bits that are never sent: known zeros
                q[:, k - (n - nt):k] = 127
            llr[(off[at][:, None] + torch.arange(n, device="cuda")[None, :]).reshape(-1)] = q.reshape(-1)
    s = {"plan": plan}
    if c["memory"] == "pinned":
        s["host"] = [torch.empty(plan.llr_bytes, dtype=torch.int8).pin_memory(), torch.empty(plan.llr_bytes // 8, dtype=torch.uint8).pin_memory(),
                     torch.empty(count, dtype=torch.int32).pin_memory(), torch.empty(count, dtype=torch.uint8).pin_memory()]
        s["host"][0].copy_(llr)
        return s
    s.update(llr=llr, bits=torch.zeros(plan.llr_bytes // 8, dtype=torch.uint8, device="cuda"),
             its=torch.zeros(count, dtype=torch.int32, device="cuda"), ok=torch.zeros(count, dtype=torch.uint8, device="cuda"))
    return s


def _run_ldpc(c, s):
    if c["memory"] == "pinned":
        llr, bits, its, ok = (t.numpy() for t in s["host"])
        s["plan"].run(llr, bits, its, ok, _stream())
        return {"bits": bits, "its": its, "ok": ok}
    s["plan"].run_dev(s["llr"].data_ptr(), s["bits"].data_ptr(), s["its"].data_ptr(), s["ok"].data_ptr(), _stream())
    return {"bits": s["bits"], "its": s["its"], "ok": s["ok"]}


def _prepare_rx(c, seed):
    fmt, luma, reg, _ = _cameras(c["n"], c["subch"], c["span"], c["w"], c["h"], c["frames"], c["k1"], c["blur"], c["noise"], seed,
                                 _side_px(c["n"], c["span"], c["h"]))
    rx = lz.Receiver(c["n"], c["subch"], c["span"], max_frames=c["frames"], read=c["read"])
    out, named = lz.rx_outputs(fmt, c["frames"])
    return {"rx": rx, "luma": luma, "reg": reg, "out": out, "named": named}


def _run_rx(c, s):
    fn = lz.lib().lizg_rx_finish_luma_graph if c["graph"] else lz.lib().lizg_rx_finish_luma_dev
    w, h = c["w"], c["h"]
    lz._check(fn(s["rx"]._h, ctypes.c_void_p(s["luma"].data_ptr()), w, h, w, w * h, ctypes.c_void_p(s["reg"].data_ptr()), c["frames"],
                 ctypes.byref(s["named"]), None, None, ctypes.c_void_p(_stream())), "finish_luma")
    return s["out"]


def _prepare_tick(c, seed):
    w, h = c["w"], c["h"]
    eng = lz.Engine()
    s = {"eng": eng, "fmts": [], "batches": [], "fork": torch.cuda.Event()}
    for i, (n, subch, span) in enumerate(TICK_FORMATS):
        k = c["c%d" % i]
        eng.add_format(n, subch, span, k)
        fmt, luma, corners, _ = _cameras(n, subch, span, w, h, k, None, c["blur"], c["noise"], seed * 8 + i, 1700.0, 15.0, 20.0, (0.8, 1.1), mesh=False)
        reg = torch.empty_like(corners)
        out, named = lz.rx_outputs(fmt, k)
        s["fmts"].append((luma, corners, reg, out, lz.Refiner(span, k), k, torch.cuda.Stream(), torch.cuda.Event()))
        s["batches"].append((i, luma.data_ptr(), w, h, w, w * h, reg.data_ptr(), k, named))
    return s


def _run_tick(c, s):
    """Each format's frames registered on a stream of its own, then every format decoded by the engine."""
    w, h = c["w"], c["h"]
    main = torch.cuda.current_stream()
    s["fork"].record(main)
    for luma, corners, reg, _, refiner, k, side, join in s["fmts"]:
        side.wait_event(s["fork"])
        with torch.cuda.stream(side):
            reg.copy_(corners)
        refiner.refine_dev(luma.data_ptr(), w, h, w * h, reg.data_ptr(), k, 3, None, None, side.cuda_stream)
        join.record(side)
        main.wait_event(join)
    s["eng"].run_dev(s["batches"], main.cuda_stream)
    return [{**{k: f[3][k] for k in ("blocks", "ok", "its", "est")}, "reg": f[2]} for f in s["fmts"]]


def _grids(c, seed):
    fmt = _format(c["n"], c["subch"], c["span"])
    rng = np.random.default_rng(seed)
    pics = [_picture(fmt, rng, k & 3) for k in range(min(c["frames"], 4))]
    gen, out = _generator(seed), torch.empty((c["frames"], fmt.n, fmt.n), device="cuda")
    ramp = torch.linspace(-8.0, 8.0, fmt.n, device="cuda")   # uneven light across the picture
    for k in range(c["frames"]):
        g = 255.0 * pics[k % len(pics)] + float(rng.uniform(-1, 1)) * ramp[None, :] + float(rng.uniform(-1, 1)) * ramp[:, None]
        g += c["noise"] * torch.randn(g.shape, generator=gen, device="cuda")
        out[k] = g.round().clamp(0, 255) / 255.0
    return fmt, out


def _prepare_spectrum(c, seed):
    fmt, grids = _grids(c, seed)
    return {"rx": lz.Receiver(c["n"], c["subch"], c["span"], max_frames=c["frames"]), "grids": grids,
            "coef": torch.zeros((c["frames"], fmt.subch * lz.SUB, 2), device="cuda")}


def _run_spectrum(c, s):
    lz._check(lz.lib().lizg_rx_spectrum_grid_dev(s["rx"]._h, ctypes.c_void_p(s["grids"].data_ptr()), c["frames"],
                                                 ctypes.c_void_p(s["coef"].data_ptr()), ctypes.c_void_p(_stream())), "spectrum_grid")
    return s["coef"]


def _exact_spectrum(c, seed):
    """The spectrum's used coefficients in 64 bits: the anchors' squares filled with the shading surface fitted to every
    eighth sample outside them, the five trends projected off, the transform, its points in order of (r^2, v, u)."""
    n, span, scale = c["n"], c["span"], np.float32(c["n"]) / np.float32(c["span"])
    _, grids = _grids(c, seed)
    z = grids.double()
    m0, a = _anchor_modules(span)
    sq = torch.zeros(n, dtype=torch.bool, device="cuda")
    for m in m0:
        lo, hi = math.floor(np.float32(m - 15) * scale) - 2, math.ceil(np.float32(m + a - 15) * scale) - 1 + 2
        sq[max(lo, 0):min(hi, n - 1) + 1] = True
    cc = (2.0 * torch.arange(n, dtype=torch.float64, device="cuda") + 1 - n) / n
    qq = cc * cc - (cc * cc).mean()
    one = torch.ones_like(cc)
    basis = torch.stack([torch.outer(*p) for p in ((one, one), (one, cc), (one, qq), (cc, one), (qq, one), (cc, cc))])   # [k, y, x]
    inside = torch.outer(sq, sq)
    B8, z8, keep = basis[:, ::8, ::8].reshape(6, -1), z[:, ::8, ::8].reshape(len(z), -1), ~inside[::8, ::8].reshape(-1)
    B8 = B8[:, keep]
    beta = torch.linalg.solve(B8 @ B8.T, B8 @ z8[:, keep].T)                       # 6 x frames
    hole = torch.einsum("kf,kyx->fyx", beta, basis)
    z = torch.where(inside, hole, z)
    for k in range(1, 6):
        t = basis[k]
        z = z - (z * t).sum((1, 2), keepdim=True) / (t * t).sum() * t
    C = torch.fft.fft2(z)
    h = n // 2
    u, v = torch.meshgrid(torch.arange(-h + 1, h), torch.arange(0, h), indexing="xy")
    u, v = u.reshape(-1), v.reshape(-1)
    use = (v > 0) | (u > 0)
    u, v = u[use], v[use]
    order = torch.argsort((u * u + v * v) * (4 * n * n) + v * (2 * n) + (u + h))[:c["subch"] * lz.SUB]
    got = C[:, v[order].cuda(), (u[order] % n).cuda()]
    return torch.view_as_real(got)


def _prepare_register(c, seed):
    w, h, k = c["w"], c["h"], c["frames"]
    _, luma, corners, _ = _cameras(c["n"], c["subch"], c["span"], w, h, k, None, c["blur"], c["noise"], seed, 950.0, 15.0, 20.0, (0.8, 1.1), mesh=False)
    s = {"refiner": lz.Refiner(c["span"], k), "luma": luma, "corners": corners, "reg": torch.empty_like(corners),
         "held": torch.zeros(k, dtype=torch.int32, device="cuda"), "lens": torch.zeros((k, 15), dtype=torch.float64, device="cuda"),
         "ok": torch.zeros((k, 49), dtype=torch.uint8, device="cuda")}
    for a in ("peak", "dx", "dy", "u", "v"):
        s[a] = torch.zeros((k, 49), device="cuda")
    s["anchors"] = lz.AnchorOut(*[s[a].data_ptr() for a in ("ok", "peak", "dx", "dy", "u", "v")])
    return s


def _run_register(c, s):
    w, h = c["w"], c["h"]
    s["reg"].copy_(s["corners"])
    s["refiner"].register_dev(s["luma"].data_ptr(), w, h, w * h, s["reg"].data_ptr(), c["frames"], None, None, s["held"].data_ptr(),
                              s["lens"].data_ptr(), s["anchors"], _stream())
    return {a: s[a] for a in ("reg", "held", "lens", "ok", "peak", "u", "v")}


def _prepare_field(c, seed):
    """Frames whose registration is off by a fraction of a pixel at every node, the anchors measured to a tenth."""
    w, h, k, span = c["w"], c["h"], c["frames"], c["span"]
    rng = np.random.default_rng(seed + 17)
    _, luma, reg, seen = _cameras(c["n"], c["subch"], span, w, h, k, None, c["blur"], c["noise"], seed, 950.0, 15.0, 20.0, (0.8, 1.1))
    off = np.zeros(tuple(reg.shape), np.float32)
    pos = _nodes(span)
    X, Y = np.meshgrid(pos / (span + 30), pos / (span + 30))
    for i in range(k):
        p = rng.uniform(-0.4, 0.4, (2, 4))
        d = [q[0] + q[1] * X + q[2] * Y + q[3] * np.sin(6.0 * X + 4.0 * Y) for q in p]
        off[i, 9:] = np.stack(d, -1).ravel()
    m0, a = _anchor_modules(span)
    pts = np.array([[x + a / 2, y + a / 2] for y in m0 for x in m0])
    uv = np.stack([_mapped(H, k1, w, h, pts) for H, k1 in seen]) + 0.1 * rng.standard_normal((k, 49, 2))
    s = {"field": lz.FieldRefiner(c["n"], c["subch"], span, chunk=k), "luma": luma, "start": reg + torch.from_numpy(off).cuda(), "reg": torch.empty_like(reg),
         "ok": torch.ones((k, 49), dtype=torch.uint8, device="cuda"), "u": torch.from_numpy(uv[..., 0].astype(np.float32)).cuda(),
         "v": torch.from_numpy(uv[..., 1].astype(np.float32)).cuda(), "loss": torch.zeros(k, device="cuda"),
         "improved": torch.zeros(k, dtype=torch.int32, device="cuda")}
    s["anchors"] = lz.AnchorOut(s["ok"].data_ptr(), *[s[a].data_ptr() for a in ("u", "u", "u", "u", "v")])
    return s


def _run_field(c, s):
    w, h = c["w"], c["h"]
    s["reg"].copy_(s["start"])
    s["field"].refine_dev(s["luma"].data_ptr(), w, h, w * h, s["reg"].data_ptr(), c["frames"], 3, s["anchors"], None, s["loss"].data_ptr(),
                          s["improved"].data_ptr(), _stream())
    return {"reg": s["reg"], "loss": s["loss"], "improved": s["improved"]}


def _prepare_encode(c, seed):
    enc = lz.Encoder(c["n"], c["subch"], c["span"], max_frames=c["frames"])
    fmt = _format(c["n"], c["subch"], c["span"])
    blocks = torch.randint(0, 256, (c["frames"], fmt.blocks, lz.BLOCK_BYTES), dtype=torch.uint8, device="cuda", generator=_generator(seed))
    return {"enc": enc, "blocks": blocks, "grey": torch.zeros((c["frames"], enc.W, enc.W), dtype=torch.uint8, device="cuda")}


def _run_encode(c, s):
    lz._check(lz.lib().lizg_encode_dev(s["enc"]._h, ctypes.c_void_p(s["blocks"].data_ptr()), c["frames"], 1, None,
                                       ctypes.c_void_p(s["grey"].data_ptr()), ctypes.c_void_p(_stream())), "encode")
    return s["grey"]


def _ingest_shape(c):
    """(bytes a row, output w, output h) of a w x h sensor's or camera's frame."""
    w, h = c["w"], c["h"]
    row = {RGBA8: 4 * w, P010: 2 * w, RAW10: w // 4 * 5, RAW12: w // 2 * 3}[c["fmt"]]
    return row, w // c["bin"], h // c["bin"]


def _prepare_ingest(c, seed):
    """Smooth scenes with sensor noise, packed as the camera packs them."""
    w, h, k = c["w"], c["h"], c["frames"]
    row, ow, oh = _ingest_shape(c)
    gen = _generator(seed)
    y, x = torch.arange(h, device="cuda", dtype=torch.float32)[:, None], torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    px = torch.empty((k, h, row), dtype=torch.uint8, device="cuda")
    bits = 12 if c["fmt"] == RAW12 else 10
    for i in range(k):
        v = 120 + 700 * x / w + 90 * torch.sin(y / (40.0 + i) + i) + 6 * torch.randn((h, w), generator=gen, device="cuda")
        v = (v.clamp(0, 1023) * (1 << (bits - 10))).round().int()
        if c["fmt"] == RGBA8:
            p = torch.stack([v >> 2, (v >> 2) * 9 // 10, (v >> 2) * 4 // 5, torch.full_like(v, 255)], -1)
        elif c["fmt"] == P010:
            p = torch.stack([(v << 6) & 255, v >> 2], -1)
        elif c["fmt"] == RAW10:
            g = v.view(h, w // 4, 4)
            p = torch.cat([g >> 2, ((g & 3) << torch.tensor([0, 2, 4, 6], device="cuda", dtype=torch.int32)).sum(-1, keepdim=True)], -1)
        else:
            g = v.view(h, w // 2, 2)
            p = torch.cat([g >> 4, (g[..., :1] & 15) | ((g[..., 1:] & 15) << 4)], -1)
        px[i] = p.to(torch.uint8).reshape(h, row)
    s = {"px": px, "out": torch.zeros((k, oh, ow), dtype=torch.uint8, device="cuda")}
    if c["fmt"] != RGBA8:
        top = float((1 << bits) - 1)
        black = 64.0 * (1 << (bits - 10))
        s["raw"] = lz.RawFrame(RAW_CODE[c["fmt"]], row, 2, 0, 0, c["bin"], (ctypes.c_float * 9)(black, black, black, black, top, 1.9, 1.0, 1.0, 1.6))
    return s


def _run_ingest(c, s):
    row, ow, oh = _ingest_shape(c)
    src, dst, st = ctypes.c_void_p(s["px"].data_ptr()), ctypes.c_void_p(s["out"].data_ptr()), ctypes.c_void_p(_stream())
    if c["fmt"] == RGBA8:
        rc = lz.lib().lizg_ingest_pixels_dev(src, c["w"], c["h"], row, row * c["h"], lz.LIZG_PIX_RGBA8, c["frames"], dst, st)
    else:
        rc = lz.lib().lizg_develop_dev(ctypes.byref(s["raw"]), src, row * c["h"], row * c["h"], c["frames"], 0, 0, ow, oh, dst, st)
    lz._check(rc, "ingest")
    return s["out"]


_PREPARE = {"ldpc": _prepare_ldpc, "rx": _prepare_rx, "tick": _prepare_tick, "spectrum": _prepare_spectrum, "register": _prepare_register,
            "field": _prepare_field, "encode": _prepare_encode, "ingest": _prepare_ingest}
_RUN = {"ldpc": _run_ldpc, "rx": _run_rx, "tick": _run_tick, "spectrum": _run_spectrum, "register": _run_register, "field": _run_field,
        "encode": _run_encode, "ingest": _run_ingest}


def prepare(case, seed):
    _format(128 * 3, 64, 128)   # the library loaded, its signatures known
    s = _PREPARE[case["kind"]](case, int(seed))
    s["case"] = case
    return s


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def exact(case, seed):
    """In 64 bits where the output is a computed number of its own: the spectrum. The decodes, pages and developed frames
    are whole numbers; a registration is the end of a search and has no value apart from it."""
    return _exact_spectrum(case, int(seed)) if case["kind"] == "spectrum" else None


# ---------------------------------------------------------------- the work that a pass cannot do without

def _ldpc_work(count_of, its):
    """(bytes in and out, integer operations) of codewords by rate, at `its` iterations a codeword: eight operations an
    edge (extrinsic, saturation, magnitude, the two minima, sign, message, posterior)."""
    b = sum(k * (lz.CODE_N[r] * 9 // 8 + 5) for r, k in count_of.items())
    return b, sum(8.0 * its * k * lz.CODE_EDGES[r] for r, k in count_of.items())


def _transform_flops(n):
    return 2.5 * n * n * math.log2(n * n)


def _frame_work(n, subch, span, w, h, side_px):
    """One frame through the receiver: the luma its picture covers, its blocks out; sampling, transform, decode."""
    f = _format(n, subch, span)
    dec = _ldpc_work({f.tier[t][0]: f.tier[t][1] for t in range(f.tiers)}, 3.0)[1]
    area = min((side_px * span / (span + 30)) ** 2, w * h)
    return area + f.blocks * (lz.BLOCK_BYTES + 13), 40.0 * n * n + _transform_flops(n) + dec


def work(case):
    c, k = case, case.get("frames", 1)
    if c["kind"] == "ldpc":
        counts = {c["rate"]: c["count"]} if c["rate"] else {r: c["count"] * f for r, f in MIX}
        b, f = _ldpc_work(counts, 6.0)
    elif c["kind"] == "rx":
        b, f = (k * x for x in _frame_work(c["n"], c["subch"], c["span"], c["w"], c["h"], _side_px(c["n"], c["span"], c["h"])))
    elif c["kind"] == "tick":
        each = [(c["c%d" % i], _frame_work(*t, c["w"], c["h"], 1615.0)) for i, t in enumerate(TICK_FORMATS)]
        b, f = sum(m * x[0] for m, x in each), sum(m * x[1] for m, x in each)
    elif c["kind"] == "spectrum":
        b, f = k * (4 * c["n"] ** 2 + 8 * c["subch"] * lz.SUB), k * _transform_flops(c["n"])
    elif c["kind"] == "register":
        b = k * 49 * (16 * 950 // 158) ** 2   # the pixels of the anchors' windows
        f = k * 49 * 2.0e5                    # a round of the search: sums over the window at every offset
    elif c["kind"] == "field":
        # a step: the picture sampled, transformed, its mismatch transformed back, its gradient at every sample; four looks
        b = k * 4 * min((950 * 128 / 158) ** 2, c["w"] * c["h"])
        f = k * (4 * (40.0 * c["n"] ** 2 + _transform_flops(c["n"])) + 3 * (60.0 * c["n"] ** 2 + _transform_flops(c["n"])))
    elif c["kind"] == "encode":
        fm = _format(c["n"], c["subch"], c["span"])
        W = (c["span"] + 34) * math.ceil(c["n"] / c["span"] - 1e-4)
        b, f = k * (fm.blocks * lz.BLOCK_BYTES + W * W), k * (_transform_flops(c["n"]) + 12.0 * W * W)
    else:
        row, ow, oh = _ingest_shape(c)
        b, f = k * (row * c["h"] + ow * oh), 0.0
    return {"bytes": float(b), "flops": float(f)}
