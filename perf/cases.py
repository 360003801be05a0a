"""The work a user of this framework has it do, as measurable cases: what a program holds before a call
(`prepare`), the call itself (`run`), what it cannot do without (`work`), and the values it should give
(`exact`, float64).

Three families of calls, each over its real range:

* the drop-in object (`TANConvolution`): one audio block at a time from device, pinned or ordinary host rows,
  several blocks per call (rendering), with and without an impulse-response swap, the non-uniform methods for
  long responses, and the direct FIR;
* the batched engine: many sessions per block, in each spectrum form, with swaps while it runs;
* the room-response producer that feeds both.

Calls go through the C entry points with the row tables built once, as a program that owns its buffers makes
them. Signals are uniform noise and responses exponentially decaying noise of unit energy, every delay line
filled with signal before the measured pass.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tan_b200 import convolution as cv
from tan_b200 import engine as eng
from tan_b200 import roomgen as rg

FS = 48000
SPECTRA = {"fp32": eng.SPECTRUM_FP32, "fp16": eng.SPECTRUM_FP16, "bf16": eng.SPECTRUM_BF16,
           "fp24": eng.SPECTRUM_FP24}
BIN_BYTES = {"fp32": (8, 8), "fp16": (4, 8), "bf16": (4, 8), "fp24": (6, 6)}  # spectrum, delay line


def listed():
    return [
        # a stereo reverb plugin in an audio callback: the smallest call, ordinary host buffers
        {"name": "stereo_host", "kind": "dropin", "channels": 2, "block": 1024, "ir": 8192, "blocks": 1,
         "rows": "host", "swap": False},
        # the headline workload's steady state: 64 channels of 65536 taps, audio already on the GPU
        {"name": "block_64ch", "kind": "dropin", "channels": 64, "block": 512, "ir": 65536, "blocks": 1,
         "rows": "device", "swap": False},
        # the same from page-locked host buffers: what an audio host pays per block, end to end
        {"name": "block_64ch_pinned", "kind": "dropin", "channels": 64, "block": 512, "ir": 65536, "blocks": 1,
         "rows": "pinned", "swap": False},
        # the time-varying step of the headline workload: every response replaced, then the crossfade block
        {"name": "swap_64ch", "kind": "dropin", "channels": 64, "block": 512, "ir": 65536, "blocks": 1,
         "rows": "device", "swap": True},
        # rendering: 32 blocks (the swap interval) in one call
        {"name": "render_64ch", "kind": "dropin", "channels": 64, "block": 512, "ir": 65536, "blocks": 32,
         "rows": "device", "swap": False},
        # rendering a stereo file from host memory, an odd length of response and a small block
        {"name": "render_stereo_host", "kind": "dropin", "channels": 2, "block": 256, "ir": 48001, "blocks": 64,
         "rows": "host", "swap": False},
        # a loaded server: 1024 sessions of 4 channels with 1 s responses
        {"name": "serve_4096ch", "kind": "engine", "sessions": 1024, "channels": 4, "block": 256, "ir_min": 48000,
         "ir_max": 48000, "spectrum": "fp32", "swaps": 0},
        # 1024 single-channel sessions of unequal lengths in the 24-bit spectrum form
        {"name": "serve_uneven_fp24", "kind": "engine", "sessions": 1024, "channels": 1, "block": 256,
         "ir_min": 4096, "ir_max": 262144, "spectrum": "fp24", "swaps": 0},
        # a lightly loaded server whose long sessions change their responses while it runs
        {"name": "serve_swaps", "kind": "engine", "sessions": 8, "channels": 8, "block": 256, "ir_min": 131072,
         "ir_max": 524288, "spectrum": "fp32", "swaps": 2},
        # very long responses at a small block: the non-uniform method, one period of its largest level
        {"name": "nonuniform_256ch", "kind": "nonuniform", "channels": 256, "block": 128, "ir": 1 << 20,
         "samples": 16384},
        # the direct method with a response per call
        {"name": "direct_16ch", "kind": "direct", "channels": 16, "ir": 4096, "samples": 2048},
        # a room response for a moved listener, both ears, 1 s
        {"name": "room_1s", "kind": "room", "width": 8.0, "height": 3.0, "length": 6.0, "samples": 48000,
         "bounces": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "dropin", "engine", "engine", "nonuniform", "direct", "room"])
    if kind == "dropin":
        while True:
            c = {"kind": kind, "channels": _log(rng, 1, 160), "block": rng.choice([128, 256, 512, 1024, 2048]),
                 "ir": _log(rng, 2000, 300000), "blocks": rng.choice([1, 1, _log(rng, 2, 70)]),
                 "rows": rng.choice(["device", "pinned", "host"]), "swap": rng.random() < 0.3}
            if c["channels"] * (c["ir"] + c["block"]) <= 12e6 and c["channels"] * c["block"] * c["blocks"] <= 1.5e6:
                return c
    if kind == "engine":
        while True:
            lo = _log(rng, 4096, 200000)
            c = {"kind": kind, "sessions": _log(rng, 4, 1024), "channels": rng.choice([1, 2, 3, 4, 6, 8]),
                 "block": rng.choice([128, 256, 512, 1024]), "ir_min": lo, "ir_max": min(524288, _log(rng, lo, 8 * lo)),
                 "spectrum": rng.choice(["fp32", "fp32", "fp24", "fp16", "bf16"])}
            c["swaps"] = rng.choice([0, 0, 1, min(4, c["sessions"])])
            taps = c["sessions"] * c["channels"] * (c["ir_min"] + c["ir_max"]) / 2
            if taps <= 150e6 and c["ir_max"] <= 2048 * c["block"]:
                return c
    if kind == "nonuniform":
        while True:
            c = {"kind": kind, "channels": _log(rng, 2, 200), "block": rng.choice([128, 256, 512]),
                 "ir": _log(rng, 60000, 1 << 20)}
            c["samples"] = c["block"] * _log(rng, 1, 16384 // c["block"])
            if c["channels"] * c["ir"] <= 120e6:
                return c
    if kind == "direct":
        ir = _log(rng, 100, 12000)
        return {"kind": kind, "channels": _log(rng, 1, 48), "ir": ir, "samples": _log(rng, 32, ir)}
    return {"kind": "room", "width": round(rng.uniform(4, 15), 2), "height": round(rng.uniform(2.4, 6), 2),
            "length": round(rng.uniform(4, 15), 2), "samples": _log(rng, 8000, 48000), "bounces": rng.choice([0, 0, 8])}


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _signal(g, channels, n):
    return torch.empty((channels, n), dtype=torch.float32, device="cuda").uniform_(-1.0, 1.0, generator=g)


def _responses(g, channels, n):
    """Decaying noise of unit energy, reverberation times of 0.2 to 1.5 s."""
    h = torch.empty((channels, n), dtype=torch.float32, device="cuda").normal_(generator=g)
    rt = torch.empty((channels, 1), dtype=torch.float32, device="cuda").uniform_(0.2, 1.5, generator=g)
    t = torch.arange(n, dtype=torch.float32, device="cuda")
    h *= torch.exp(t * (-math.log(1000.0) / FS) / rt)
    h /= h.norm(dim=1, keepdim=True)
    return h


def _ptrs(t):
    """Row pointers of a contiguous 2-D tensor (device or host)."""
    step = t.stride(0) * t.element_size()
    return (ctypes.c_void_p * t.shape[0])(*[t.data_ptr() + c * step for c in range(t.shape[0])])


def _ok(rc):
    if rc != 0:
        raise cv.TANError(rc, "perf case")


def _dropin_inputs(case, seed):
    g = _gen(seed)
    C, B, L = case["channels"], case["block"], case["ir"]
    hist = -(-L // B) * B
    x = _signal(g, C, hist + B * case["blocks"])
    irs = [_responses(g, C, L) for _ in range(2 if case["swap"] else 1)]
    return x, hist, irs


def _engine_lengths(case):
    """The sessions' response lengths, spread over the logarithm of their range."""
    n, lo, hi = case["sessions"], case["ir_min"], case["ir_max"]
    ratio = math.log(hi / lo)
    return [int(lo * math.exp(ratio * ((i * 0.6180339887498949) % 1.0))) for i in range(n)]


def _engine_inputs(case, seed):
    g = _gen(seed)
    C, B = case["channels"], case["block"]
    lens = _engine_lengths(case)
    hist = -(-max(lens) // B) * B
    x = _signal(g, C * len(lens), hist + B)
    irs = [_responses(g, C, n) for n in lens]
    new = [_responses(g, C, lens[s]) for s in range(case["swaps"])]
    return x, hist, lens, irs, new


def _direct_inputs(case, seed):
    g = _gen(seed)
    C, L, n = case["channels"], case["ir"], case["samples"]
    size = 1 << max(0, L - 1).bit_length()
    ir = torch.zeros((C, size), dtype=torch.float32)
    ir[:, :L] = _responses(g, C, L).cpu()
    return ir, _signal(g, C, n).cpu(), _signal(g, C, n).cpu(), size


def _room_inputs(case, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    damp = [float(v) for v in r.uniform(0.2, 0.8, 6)]
    dims = (case["width"], case["height"], case["length"])
    room = rg.Room(*dims, *damp)
    source = rg.Source(*[float(d * v) for d, v in zip(dims, r.uniform(0.15, 0.85, 3))])
    head = [float(d * v) for d, v in zip(dims, r.uniform(0.15, 0.85, 3))]
    k = np.arange(24)
    low = 0.25 * 0.75 ** k  # one-pole low pass of the head model and its complement
    high = (k == 0) - low
    ears = rg.listener(head, 0.16, float(r.uniform(-180, 180)), float(r.uniform(-20, 20)), 0.0, low, high)
    return room, source, ears


def _nonuniform_inputs(case, seed):
    g = _gen(seed)
    B = case["block"]
    hist = -(-case["ir"] // 16384) * 16384  # whole periods of the largest level
    return _signal(g, case["channels"], hist + case["samples"] // B * B), hist, [_responses(g, case["channels"], case["ir"])]


# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    ctx = cv.TANContext(0)
    s = {"kind": kind, "lib": cv.lib(), "ctx": ctx, "done": ctypes.c_size_t(0)}
    if kind in ("dropin", "nonuniform"):
        C, B = case["channels"], case["block"]
        if kind == "dropin":
            x, hist, irs = _dropin_inputs(case, seed)
            n, method = B * case["blocks"], cv.TAN_CONVOLUTION_METHOD_FFT_PARTITIONED_UNIFORM
        else:
            x, hist, irs = _nonuniform_inputs(case, seed)
            n, method = case["samples"], cv.TAN_CONVOLUTION_METHOD_FFT_PARTITIONED_NONUNIFORM
        conv = cv.TANConvolution(ctx)
        _ok(conv.Init(method, case["ir"], B, C))
        torch.cuda.synchronize()
        _ok(conv.UpdateResponseTDDevice(irs[0], case["ir"], None, cv.TAN_CONVOLUTION_OPERATION_FLAG_BLOCK_UNTIL_READY))
        old = x[:, :hist].contiguous()
        out = torch.empty_like(old)
        torch.cuda.synchronize()
        _ok(conv.ProcessDevice(old, out, hist)[0])
        _ok(conv.Synchronize())
        rows = case.get("rows", "device")
        if rows == "device":
            xin, y = x[:, hist:].contiguous(), torch.empty((C, n), dtype=torch.float32, device="cuda")
        elif rows == "pinned":
            xin, y = x[:, hist:].cpu().pin_memory(), torch.zeros((C, n), dtype=torch.float32).pin_memory()
        else:
            xin, y = x[:, hist:].cpu().contiguous(), torch.zeros((C, n), dtype=torch.float32)
        s.update(conv=conv, n=n, x=xin, y=y, px=_ptrs(xin), py=_ptrs(y), ir_len=case["ir"], turn=0,
                 call=s["lib"].tanb_convolution_process_device if rows == "device" else
                 s["lib"].tanb_convolution_process)
        if case.get("swap"):
            s.update(irs=irs, pir=[_ptrs(irs[1]), _ptrs(irs[0])])
    elif kind == "engine":
        C, B = case["channels"], case["block"]
        x, hist, lens, irs, new = _engine_inputs(case, seed)
        spec = SPECTRA[case["spectrum"]]
        budget = sum(eng.session_bytes(B, C, n, None, spec) for n in lens)
        e = eng.Engine(ctx, B, spec, budget_bytes=budget, max_channels=C * len(lens))
        sessions = []
        torch.cuda.synchronize()
        for n, h in zip(lens, irs):
            rc, sess = e.open_session(C, n)
            _ok(rc)
            _ok(sess.update_response_td_device(h))
            sessions.append(sess)
        _ok(e.synchronize())
        y = torch.empty((x.shape[0], B), dtype=torch.float32, device="cuda")
        out = torch.empty_like(x)  # the engine takes one row step for input and output
        torch.cuda.synchronize()
        for k in range(hist // B):
            _ok(s["lib"].tanb_engine_process_device(e._h, x.data_ptr() + 4 * k * B, out.data_ptr(), x.shape[1]))
        _ok(e.synchronize())
        xin = x[:, hist:].contiguous()
        swaps = [(sessions[i].id, [_ptrs(new[i]), _ptrs(irs[i])], lens[i]) for i in range(case["swaps"])]
        keep = [(new[i], irs[i]) for i in range(case["swaps"])]
        s.update(engine=e, sessions=sessions, x=xin, y=y, swaps=swaps, keep=keep, turn=0)
    elif kind == "direct":
        ir, x0, x1, _ = _direct_inputs(case, seed)
        conv = cv.TANConvolution(ctx)
        _ok(conv.Init(cv.TAN_CONVOLUTION_METHOD_TIME_DOMAIN, case["ir"], 128, case["channels"]))
        y = torch.zeros_like(x1)
        _ok(conv.ProcessDirect(ir.numpy(), x0.numpy(), y.numpy(), case["samples"])[0])
        s.update(conv=conv, ir=ir, x=x1, y=y, n=case["samples"], pir=_ptrs(ir), px=_ptrs(x1), py=_ptrs(y))
    else:
        room, source, ears = _room_inputs(case, seed)
        left, right = (torch.zeros(case["samples"], dtype=torch.float32, device="cuda") for _ in range(2))
        s.update(gen=rg.RoomGenerator(ctx, case["samples"]), room=room, source=source, ears=ears, left=left,
                 right=right, n=case["samples"], bounces=case["bounces"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, lib = s["kind"], s["lib"]
    if kind in ("dropin", "nonuniform"):
        h = s["conv"]._h
        if "pir" in s:  # every channel's response replaced by the other of its two
            _ok(lib.tanb_convolution_update_response_td_device(h, s["pir"][s["turn"]], s["ir_len"], None, 0))
            s["turn"] ^= 1
        _ok(s["call"](h, s["px"], s["py"], s["n"], None, ctypes.byref(s["done"])))
        return s["y"]
    if kind == "engine":
        e = s["engine"]._h
        for sid, rows, n in s["swaps"]:
            _ok(lib.tanb_engine_update_response_td_device(e, sid, rows[s["turn"]], n, 1))
        s["turn"] ^= 1
        _ok(lib.tanb_engine_process_device(e, s["x"].data_ptr(), s["y"].data_ptr(), 0))
        return s["y"]
    if kind == "direct":
        _ok(lib.tanb_convolution_process_direct(s["conv"]._h, s["pir"], s["px"], s["py"], s["n"],
                                                ctypes.byref(s["done"]), None))
        return s["y"]
    flags = rg.GENROOM_LIMIT_BOUNCES if s["bounces"] else 0
    _ok(s["gen"].response(s["room"], s["source"], s["ears"], FS, s["n"], s["left"], s["right"], flags, s["bounces"]))
    return {"left": s["left"], "right": s["right"]}


# ---------------------------------------------------------------------------

def _images(case):
    """Image sources per axis, as the producer enumerates them."""
    counts = []
    for d in (case["width"], case["height"], case["length"]):
        n = 1 + case["samples"] // int(np.float32(np.float32(d) / np.float32(340.0)) * np.float32(FS))
        n = min(n, case["bounces"]) if case["bounces"] else n
        counts.append((n, 2 * n if (2 * n) % 4 == 0 else 2 * n + 1))
    return counts


def work(case):
    """Bytes: the spectra of the responses in use, the delay line and the samples in and out, once per call;
    operations: the transforms and 8 per bin and partition."""
    kind = case["kind"]
    if kind in ("dropin", "engine"):
        B = case["block"]
        if kind == "dropin":
            nb, swapped, sb, xb = case["blocks"], case["swap"], 8, 8
            chans = [(-(-case["ir"] // B), case["channels"], swapped)]
        else:
            nb, (sb, xb) = 1, BIN_BYTES[case["spectrum"]]
            chans = [(-(-n // B), case["channels"], i < case["swaps"]) for i, n in enumerate(_engine_lengths(case))]
        fft = 5.0 * B * math.log2(2 * B)
        total, flops = 0.0, 0.0
        for P, C, swap in chans:
            total += C * (P * B * (sb + xb) + 8.0 * B * nb)
            flops += C * nb * (8.0 * P * B + 2 * fft)
            if swap:  # the new response's samples in, its spectra out, and both responses' products
                total += C * P * B * (4.0 + 2 * sb)
                flops += C * (P * fft + 8.0 * P * B + fft)
        return {"bytes": total, "flops": flops}
    if kind == "nonuniform":
        C, L, n = case["channels"], case["ir"], case["samples"]
        # the largest level's spectra and delay line are read in full once per 16384 samples
        return {"bytes": C * (16.0 * L * min(1.0, n / 16384.0) + 8.0 * n), "flops": C * (8.0 * L * n / 16384.0 +
                                                                              20.0 * n * math.log2(L))}
    if kind == "direct":
        C, L, n = case["channels"], case["ir"], case["samples"]
        return {"bytes": 4.0 * C * (2 * L + 2 * n), "flops": 2.0 * C * L * n}
    images = float(np.prod([c for _, c in _images(case)]))
    return {"bytes": 8.0 * case["samples"], "flops": 2 * 40.0 * images}


# ---------------------------------------------------------------------------

def _convolve_last(x, h, n):
    """The last n samples of x * h in float64, a few channels at a time."""
    size = 1 << int(x.shape[1] + h.shape[1] - 2).bit_length()
    step = max(1, (1 << 26) // size)
    out = torch.empty((x.shape[0], n), dtype=torch.float64, device="cuda")
    for c in range(0, x.shape[0], step):
        X = torch.fft.rfft(x[c:c + step].double(), size)
        X *= torch.fft.rfft(h[c:c + step].double(), size)
        out[c:c + step] = torch.fft.irfft(X, size)[:, x.shape[1] - n:x.shape[1]]
    return out


def _crossfade(old, new, block):
    y = new.clone()
    w = torch.arange(block, dtype=torch.float64, device="cuda") / block
    y[:, :block] = new[:, :block] * w + old[:, :block] * (1.0 - w)
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        x, hist, irs = _dropin_inputs(case, seed)
        n = x.shape[1] - hist
        y = _convolve_last(x, irs[0], n)
        if case["swap"]:
            y = _crossfade(y, _convolve_last(x, irs[1], n), case["block"])
        return y.cpu()
    if kind == "nonuniform":
        x, hist, irs = _nonuniform_inputs(case, seed)
        return _convolve_last(x, irs[0], x.shape[1] - hist).cpu()
    if kind == "engine":
        x, hist, lens, irs, new = _engine_inputs(case, seed)
        C, B = case["channels"], case["block"]
        y = torch.empty((x.shape[0], B), dtype=torch.float64, device="cuda")
        for i, n in enumerate(lens):
            xs = x[i * C:(i + 1) * C, x.shape[1] - (n + B):] if x.shape[1] > n + B else x[i * C:(i + 1) * C]
            v = _convolve_last(xs, irs[i], B)
            if i < case["swaps"]:
                v = _crossfade(v, _convolve_last(xs, new[i], B), B)
            y[i * C:(i + 1) * C] = v
        return y.cpu()
    if kind == "direct":
        ir, x0, x1, size = _direct_inputs(case, seed)
        n = case["samples"]
        line = torch.zeros((case["channels"], size), dtype=torch.float64)
        for k, x in enumerate((x0, x1)):  # the circular history after both calls
            line[:, (torch.arange(n) + k * n) % size] = x.double()
        y = torch.fft.irfft(torch.fft.rfft(line) * torch.fft.rfft(ir.double()), size)
        return y[:, (torch.arange(n) + n) % size]
    return _exact_room(case, seed)


def _exact_room(case, seed):
    """The image sum with arrival samples as the producer's single-precision positions give them (they are
    rounded to whole samples) and gains, filters and sums in float64."""
    room, source, ears = _room_inputs(case, seed)
    f32 = dict(dtype=torch.float32, device="cuda")
    es = float(np.float32(ears.ear_spacing))
    pi = np.float32(math.pi)
    f = np.float32
    sY, cY = (fn(f(f(ears.yaw) * pi) / f(180)) for fn in (np.sin, np.cos))
    sP, cP = (fn(f(f(ears.pitch) * pi) / f(180)) for fn in (np.sin, np.cos))
    m = np.array([[cY, 0, sY], [sP * sY, cP, -sP * cY], [-cP * sY, sP, cP * cY]], np.float32)  # no roll
    offs = np.array([[es / 2, 0, 0], [-es / 2, 0, 0], [es / 2, 0, -es / 2], [-es / 2, 0, -es / 2]], np.float32) @ m.T
    dims = [f(case[k]) for k in ("width", "height", "length")]
    src = [min(max(f(v), f(0)), d) for v, d in zip((source.x, source.y, source.z), dims)]
    damp = [(room.damp_right, room.damp_left), (room.damp_top, room.damp_bottom), (room.damp_front, room.damp_back)]
    idx, pos, amp = [], [], []
    for (n, extent), d, sp, (dp, dm) in zip(_images(case), dims, src, damp):
        i = torch.arange(extent, device="cuda") - n
        even = i % 2 == 0
        a = torch.where(even, i, i + 1).to(torch.float32)
        pos.append(a * torch.tensor(d, **f32) + torch.where(even, 1.0, -1.0).to(torch.float32) * torch.tensor(sp, **f32))
        plus = torch.where(i > 0, (i + 1) // 2, i.abs() // 2)
        minus = torch.where(i > 0, torch.div(i, 2, rounding_mode="floor"), (i - 1).abs() // 2)
        amp.append(torch.pow(torch.tensor(dp, dtype=torch.float64, device="cuda"), plus)
                   * torch.pow(torch.tensor(dm, dtype=torch.float64, device="cuda"), minus))
    n, speed = case["samples"], torch.tensor(340.0, **f32)
    cut = 2 * sum(int(f(d / f(340.0)) * f(FS)) for d in dims)
    taps = ears.filter_length
    lp = torch.tensor(list(ears.low_pass)[:taps], dtype=torch.float64, device="cuda")
    hp = torch.tensor(list(ears.high_pass)[:taps], dtype=torch.float64, device="cuda")
    out = torch.zeros((2, n + 64), dtype=torch.float64, device="cuda")
    for ear in range(2):
        head = [f(v) + f(o) for v, o in zip((ears.head_x, ears.head_y, ears.head_z), offs[ear])]
        ev = [float(v) for v in offs[2 + ear]]
        norm = math.sqrt(sum(v * v for v in ev))
        dx, dy = (pos[k] - torch.tensor(head[k], **f32) for k in (0, 1))
        for iz in range(pos[2].numel()):
            dz = pos[2][iz] - torch.tensor(head[2], **f32)
            d = torch.sqrt(((dx * dx)[None, :] + (dy * dy)[:, None]) + dz * dz)
            at = 1 + ((d / speed) * float(FS)).to(torch.int64)
            keep = at < n
            d64, at = d[keep].double(), at[keep]
            gain = (amp[2][iz] * amp[1][:, None] * amp[0][None, :])[keep]
            gain = gain * torch.where(d64 <= 2 * es, torch.full_like(d64, 2.0), 2.0 * (2 * es) / d64)
            early = at < cut
            out[ear].index_add_(0, at[~early], gain[~early])
            if bool(early.any()):
                dot = (ev[0] * dx.double()[None, :] + ev[1] * dy.double()[:, None] + ev[2] * dz.double())[keep][early]
                hf = (dot / (norm * d64[early]) + 1.0) / 2.0
                add = gain[early][:, None] * (lp[None, :] + hf[:, None] * hp[None, :])
                where = at[early][:, None] + torch.arange(taps, device="cuda")[None, :]
                out[ear].index_add_(0, where.reshape(-1), add.reshape(-1))
    return {"left": out[0, :n].cpu(), "right": out[1, :n].cpu()}
