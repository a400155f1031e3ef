"""Workloads that users of the RF backend run, through its public entry points.

Each case is one call sequence of a user's program: a capture (host or device
memory) decoded by a session, a whole-run handoff that writes files, a batch
of serving windows, a FLAC capture, a real-time pulse scan.  Captures are
synthetic VHS RF of the shapes the tests and the benchmark use
(``vhsd_gb300.synth``: VBI structure, bars / ramp / noise content,
pre-emphasis, FM, colour-under chroma, noise, dropouts, timebase wobble),
built here on the GPU so that long ones are quick to make.
"""
import ctypes
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "vhs-decode-dotnet_gb300"))
# A user who compares decodes fixes the FFT plan (the per-device tuner may
# otherwise choose another radix plan from one process to the next, whose
# rounding differs in the last bit).
os.environ.setdefault("VHSD_FFT_PLAN", "0")

from vhsd_gb300 import ldf, native, synth  # noqa: E402

BLOCK, STRIDE = 32768, 30720
OUT = {"PAL": (1135, 313), "NTSC": (910, 263)}      # output line length, field lines
SPEEDS = {"SP": native.TAPE_SP, "LP": native.TAPE_LP, "EP": native.TAPE_EP}
TAPES = {"VHS": native.FORMAT_VHS, "SVHS": native.FORMAT_SVHS}
PROFILES = {"PAL": native.PROFILE_PAL, "NTSC": native.PROFILE_NTSC}


def _session(name, **kw):
    """A session decode: `fields` fields of `system` `tape` at `speed`; the
    source is sampled at `mhz` x `decimation`; `source` is where the capture
    lies; `details`: the field's lines and dropouts are read too."""
    base = dict(name=name, kind="session", system="NTSC", tape="VHS", speed="SP", mhz=40.0, decimation=1,
                fields=4, source="pinned", dtype="int16", chroma=True, fp64=False, dropouts=0, wobble=0.0,
                details=False)
    base.update(kw)
    return base


def listed():
    return [
        # a real-time loop scans the sync stream it has on the device, a block at a time
        dict(name="pulse_scan_64k", kind="pulses", samples=65536),
        # a preview: a window of two fields from ordinary host memory, luma only
        _session("preview_pal_2_fields", system="PAL", fields=2, source="pageable", chroma=False, details=True),
        # a short clip with the default decode (luma and colour-under chroma)
        _session("pal_vhs_4_fields", system="PAL", fields=4, details=True),
        # the benchmark's capture: on the device already, luma and chroma to pinned host memory
        _session("ntsc_vhs_60_fields", fields=60, source="device", dropouts=200),
        # the same from pinned host memory with --skip_chroma (the cuda-fast backend's output)
        _session("ntsc_vhs_60_fields_luma", fields=60, chroma=False, dropouts=200),
        # the benchmark's long S-VHS capture (sub-deemphasis on every block), an unsteady tape
        _session("pal_svhs_100_fields", system="PAL", tape="SVHS", fields=100, source="device", wobble=0.005),
        # --decode-at-20msps: a 40 MSPS capture through the device decimator
        _session("ntsc_vhs_30_fields_at_20", fields=30, mhz=20.0, decimation=2, chroma=False, dropouts=40),
        # a long-play tape captured as float samples
        _session("ntsc_ep_float_9_fields", fields=9, speed="EP", dtype="float32", source="pageable", dropouts=8,
                 details=True),
        # the double-precision decode, for results that match the exact backend
        _session("pal_vhs_fp64_3_fields", system="PAL", fields=3, fp64=True, details=True),
        # a compressed .ldf capture of the benchmark's length to samples
        dict(name="flac_41m_samples", kind="flac", samples=41071507),
        # serving: four clients' windows of half a second, submitted together
        dict(name="serve_4_windows", kind="server", windows=4, ms=500),
        # the whole-run handoff: capture in, .tbc / _chroma.tbc / .tbc.json files out
        dict(name="run_ntsc_12_fields", kind="run", system="NTSC", fields=12, chroma=True, dropouts=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.1:
        return dict(kind="pulses", samples=_log(rng, 4096, 1 << 24))
    if pick < 0.2:
        return dict(kind="flac", samples=_log(rng, 100000, 41000000))
    if pick < 0.3:
        return dict(kind="server", windows=rng.randint(1, 6), ms=rng.randint(120, 600))
    if pick < 0.4:
        return dict(kind="run", system=rng.choice(["PAL", "NTSC"]), fields=_log(rng, 2, 40),
                    chroma=rng.random() < 0.7, dropouts=rng.randint(0, 60))
    case = _session("", system=rng.choice(["PAL", "NTSC"]), tape=rng.choice(["VHS", "VHS", "SVHS"]),
                    speed=rng.choice(["SP", "SP", "LP", "EP"]), source=rng.choice(["device", "pinned", "pageable"]),
                    dtype=rng.choice(["int16", "int16", "float32"]), chroma=rng.random() < 0.7,
                    wobble=rng.choice([0.0, 0.0, 0.005]), details=rng.random() < 0.5)
    del case["name"]
    rate = rng.random()
    if rate < 0.25:
        case.update(mhz=20.0, decimation=2)
    elif rate < 0.4:
        case.update(mhz=20.0)
    case["fp64"] = rng.random() < 0.15
    case["fields"] = _log(rng, 2, 10 if case["fp64"] else 90)
    case["dropouts"] = rng.randint(0, 2 * case["fields"])
    return case


# ------------------------------------------------------------------ captures

def _step(t, width):
    x = (t / width + 0.5).clamp_(0.0, 1.0)
    return 0.5 - 0.5 * torch.cos(math.pi * x)


def _capture(system, tape, mhz, fields, seed, dropouts=0, wobble=0.0):
    """int16 RF of `fields` fields on the GPU: the signal model of
    vhsd_gb300.synth, its phase from an integer accumulator and its band limit
    and pre-emphasis applied in the frequency domain."""
    make = {("PAL", "VHS"): synth.pal_vhs, ("NTSC", "VHS"): synth.ntsc_vhs,
            ("PAL", "SVHS"): synth.pal_svhs, ("NTSC", "SVHS"): synth.ntsc_svhs}[system, tape]
    cfg = make(fs=mhz * 1e6, fields=fields, snr_db=42.0 if tape == "SVHS" else 39.0, dropouts=dropouts)
    dev, f8 = torch.device("cuda"), torch.float64
    rng = np.random.default_rng(seed)
    gen = torch.Generator(dev).manual_seed(seed)
    g, pal, us, fs = synth._geometry(system), system == "PAL", 1.0 / mhz, mhz * 1e6
    line = g["line_us"] * mhz
    nlines = g["lines"]
    lead = cfg.lead_lines * line
    total = int(math.ceil((fields + 1.5) * nlines * line / 2 + lead))
    pos = torch.arange(total, device=dev, dtype=f8)
    if wobble:
        w = 2 * math.pi * cfg.wobble_hz / fs
        pos += wobble / w * torch.sin(w * pos + rng.uniform(0, 2 * math.pi))
    pos -= lead
    frame = torch.floor(pos / (nlines * line))
    pos -= frame * (nlines * line)
    frame = frame.long()
    half = torch.floor(pos / (line / 2)).long().clamp_(0, 2 * nlines - 1)
    row = half // 2                                     # frame line - 1
    tau_h = pos - half * (line / 2)
    tau = pos - row * line
    del pos
    edge = 0.2 / us
    kind = torch.from_numpy(synth._halfline_kinds(system).astype(np.int64)).to(dev)[half]
    widths = torch.tensor([0.0, g["hsync_us"] / us, g["eq_us"] / us, g["vsync_us"] / us], device=dev, dtype=f8)
    ire = cfg.vsync_ire * _step(tau_h, edge) * (1.0 - _step(tau_h - widths[kind], edge)) * (kind > 0)
    del tau_h, half, kind
    a0, a1 = g["active"][0] / us, g["active"][1] / us
    act = _step(tau - a0, edge) * (1.0 - _step(tau - a1, edge))
    act *= torch.tensor([synth._active_line(system, r + 1) for r in range(nlines)], device=dev)[row]
    second = torch.tensor([synth._field_of_line(system, r + 1) for r in range(nlines)], device=dev)[row]
    field = frame * 2 + second
    pattern = field % 3                                 # bars, ramp, noise
    x = ((tau - a0) / (a1 - a0)).clamp_(0.0, 1.0)
    bars = 75.0 * torch.tensor([1.0, 0.886, 0.701, 0.587, 0.413, 0.299, 0.114, 0.0], device=dev, dtype=f8)
    blocks = torch.from_numpy(rng.uniform(0.0, 100.0, (8, 40, 32))).to(dev)
    field_row = ((row - torch.where(second == 0, 0, nlines // 2 + 1)) // 8).clamp_(0, 39)
    col = (x * 8).long().clamp_(0, 7)
    content = torch.where(pattern == 0, bars[col], torch.where(
        pattern == 1, 100.0 * x, blocks[field % 8, field_row, (x * 32).long().clamp_(0, 31)]))
    ire += content * act
    del content, field_row
    # band limit (about 4.5 MHz) and the VHS pre-emphasis shelf
    nfft = 1 << (total - 1).bit_length()
    spec = torch.fft.rfft(ire, nfft)
    om = torch.arange(nfft // 2 + 1, device=dev, dtype=f8) * (2 * math.pi / nfft)
    b, a = synth._high_shelf(cfg.deemph_mid, cfg.deemph_gain, fs, cfg.deemph_q)
    z = torch.polar(torch.ones_like(om), -om)
    spec *= torch.exp(-0.5 * (om * fs / (2 * math.pi * 4.5e6)) ** 2)
    spec *= (b[0] + z * (b[1] + z * b[2])) / (a[0] + z * (a[1] + z * a[2]))
    del z, om
    ire = torch.fft.irfft(spec, nfft)[:total]
    del spec
    inc = torch.round((cfg.ire0 + cfg.hz_ire * ire) * (2.0 ** 32 / fs)).long()
    phase = (torch.cumsum(inc, 0) & 0xFFFFFFFF).double() * (2 * math.pi / 2 ** 32)
    del inc, ire
    rf = torch.cos(phase)
    del phase
    if dropouts:
        starts = rng.integers(int(lead), total - int(42 * mhz), dropouts)
        ends = starts + (rng.uniform(2.0, 40.0, dropouts) * mhz).astype(np.int64)
        delta = torch.zeros(total, device=dev, dtype=torch.int32)
        one = torch.ones(dropouts, device=dev, dtype=torch.int32)
        delta.index_add_(0, torch.from_numpy(starts).to(dev), one)
        delta.index_add_(0, torch.from_numpy(ends).to(dev), -one)
        rf = torch.where(torch.cumsum(delta, 0) > 0, cfg.dropout_level * rf, rf)
        del delta
    # line-locked colour-under chroma: the burst and the colour bars
    index = frame * nlines + row
    rot = torch.where(field % 2 == 0, 0 if pal else -1, -1 if pal else 1)
    b0, b1 = (5.6, 7.85) if pal else (5.3, 7.8)
    burst = _step(tau - b0 / us, edge) * (1.0 - _step(tau - b1 / us, edge))
    vsw = torch.where(index % 2 == 0, 1.0, -1.0).double() if pal else torch.ones(1, device=dev, dtype=f8)
    uv = torch.from_numpy(synth._BARS_UV).to(dev)
    u, v = uv[col, 0], uv[col, 1] * vsw
    amp = torch.hypot(u, v) * act * (pattern == 0)
    theta = torch.where(burst > amp, torch.pi * (1.0 - 0.25 * vsw) if pal else torch.full_like(vsw, math.pi),
                        torch.atan2(v, u))
    outlen, fsc = (1135, 4.43361875e6) if pal else (910, 315e6 / 88.0)
    psi = math.pi + torch.remainder(rot * index, 4) * (math.pi / 2) - theta \
        + 2 * math.pi * cfg.chroma_hz * outlen / (4.0 * fsc) * index
    level = 10.0 ** (cfg.chroma_db / 20.0)
    rf += level * (0.3 * burst + amp) * torch.cos(2 * math.pi * cfg.chroma_hz / fs * tau + psi)
    noise = math.sqrt(0.5 + 0.5 * level ** 2) / 10.0 ** (cfg.snr_db / 20.0)
    rf += noise * torch.randn(total, device=dev, generator=gen)
    rf *= cfg.peak / (1.0 + 1.3 * level + 4.5 * noise)
    return torch.round(rf).clamp_(-32768, 32767).to(torch.int16)


def _samples(system, mhz, fields):
    g = synth._geometry(system)
    line = g["line_us"] * mhz
    return int(math.ceil((fields + 1.5) * g["lines"] * line / 2 + 12.0 * line))


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _pin(t):
    out = _pinned(t.shape, t.dtype)
    out.copy_(t)
    return out


# ------------------------------------------------------------------ sessions

def _prepare_session(case, seed):
    rate = case["mhz"] * case["decimation"]
    rf = _capture(case["system"], case["tape"], rate, case["fields"], seed, case["dropouts"], case["wobble"])
    if case["dtype"] == "float32":
        rf = rf.float()
    sess = native.Session(PROFILES[case["system"]], len(rf), sample_rate_mhz=case["mhz"],
                          precision=native.PRECISION_FP64_PLAIN if case["fp64"] else native.PRECISION_FP32_FUSED,
                          tape_format=TAPES[case["tape"]], decimation=case["decimation"],
                          tape_speed=SPEEDS[case["speed"]])
    if case["source"] == "pinned":
        rf = _pin(rf)
    elif case["source"] == "pageable":
        rf = rf.cpu()
    outlen, lines = OUT[case["system"]]
    out = [_pinned((case["fields"] + 2, lines, outlen), torch.int16) for _ in range(2 if case["chroma"] else 1)]
    # (line, start, end) of up to 512 dropouts a field
    drops = np.zeros((case["fields"] + 2, 512, 3), np.int32) if case["details"] else None
    return dict(case=case, session=sess, rf=rf, out=out, drops=drops)


def _run_session(state):
    case, sess, rf, out = state["case"], state["session"], state["rf"], state["out"]
    if case["source"] == "device":
        r = sess.decode(None, device_ptr=rf.data_ptr(), count=len(rf), float_input=case["dtype"] == "float32",
                        chroma=case["chroma"])
    else:
        r = sess.decode(rf.numpy(), chroma=case["chroma"])
    n = r.fields
    sess.tbc_into(0, n, out[0].data_ptr())
    if case["chroma"]:
        sess.chroma_into(0, n, out[1].data_ptr())
    result = {"fields": n, "luma": out[0][:n]}
    if case["chroma"]:
        result["chroma"] = out[1][:n]
    if case["details"]:
        result["lines"] = np.concatenate([np.zeros(0)] + [sess.lines(i) for i in range(n)])
        drops = state["drops"]
        drops[:] = 0
        for i in range(n):
            d = sess.dropouts(i)[:drops.shape[1]]
            if d:
                drops[i, :len(d)] = d
        result["dropouts"] = drops[:n]
    return result


# -------------------------------------------------------------------- pulses

PULSE_HIGH = 3.4e6     # Hz: between the sync tip and blanking


def _prepare_pulses(case, seed):
    """A sync reference stream: pulses every line of 2542 samples, with noise."""
    n = case["samples"]
    gen = torch.Generator("cuda").manual_seed(seed)
    at = (torch.arange(n, device="cuda") + int(torch.randint(2542, (1,), device="cuda", generator=gen))) % 2542
    depth = ((at / 8.0).clamp(0, 1) - ((at - 188) / 8.0).clamp(0, 1))      # edges of 200 ns
    ref = (3.69e6 - 4.1e5 * depth + 3e4 * torch.randn(n, device="cuda", generator=gen)).float()
    cap = n // 8 + 64
    return dict(case=case, ref=ref, events=torch.zeros(cap, dtype=torch.int64, device="cuda"),
                total=torch.zeros(1, dtype=torch.int64, device="cuda"))


def _run_pulses(state):
    ref, events, total = state["ref"], state["events"], state["total"]
    native.check(native.load().vhsdecode_gb300_pulse_events_noalloc(
        ctypes.c_void_p(ref.data_ptr()), len(ref), PULSE_HIGH, ctypes.c_void_p(events.data_ptr()), len(events),
        ctypes.c_void_p(total.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"events": events, "total": total}


def _pulses_exact(case, seed):
    s = _prepare_pulses(case, seed)
    low = torch.cat([torch.zeros(1, dtype=torch.bool, device="cuda"), s["ref"].double() <= PULSE_HIGH])
    change = torch.nonzero(low[1:] != low[:-1])[:, 0]
    ev = 2 * change + (~low[1:][change]).long()
    events = s["events"].clone()
    events[:len(ev)] = ev
    return {"events": events, "total": torch.tensor([len(ev)], device="cuda")}


# ---------------------------------------------------------------------- FLAC

def _crc16_zeros(nbytes):
    """What `nbytes` zero bytes do to each of the CRC-16's 16 state bits."""
    def mul(p, q):           # p after q, as images of the 16 bits
        return [_gf_apply(p, v) for v in q]
    one = [ldf.CRC16[(1 << b) >> 8] ^ (((1 << b) << 8) & 0xFFFF) for b in range(16)]
    out = [1 << b for b in range(16)]
    while nbytes:
        if nbytes & 1:
            out = mul(one, out)
        one = mul(one, one)
        nbytes >>= 1
    return out


def _gf_apply(images, v):
    r = 0
    for b in range(16):
        if v >> b & 1:
            r ^= images[b]
    return r


FLAC_BLOCK, FLAC_BASE = 4096, 40


def _flac(samples, seed):
    """(stream bytes, samples): a 16-bit mono FLAC capture whose 4096-sample
    frames repeat FLAC_BASE encoded ones, each with its own number."""
    rf = _capture("NTSC", "VHS", 40.0, 1, seed)[:FLAC_BLOCK * FLAC_BASE].cpu().numpy()
    order = np.random.default_rng(seed)
    base = []
    for i in range(FLAC_BASE):
        x = rf[i * FLAC_BLOCK:(i + 1) * FLAC_BLOCK]
        body = ldf.write(x, FLAC_BLOCK, seed=seed + i)[42 + 6:-2]
        base.append((body, ldf.crc16(body), _crc16_zeros(len(body)), x))
    nfr = samples // FLAC_BLOCK
    tail = rf[:samples - nfr * FLAC_BLOCK]
    parts, data = [], []
    for i, k in enumerate(order.integers(0, FLAC_BASE, nfr)):
        body, crc, zeros, x = base[k]
        head = b"\xff\xf8\xc0\x08" + ldf._utf8_number(i)
        head += bytes([ldf.crc8(head)])
        c = _gf_apply(zeros, ldf.crc16(head)) ^ crc
        parts += [head, body, bytes([c >> 8, c & 0xFF])]
        data.append(x)
    if len(tail):
        parts.append(ldf._frame(tail.astype(np.int64), nfr, {"kind": "verbatim"}))
        data.append(tail)
    info = FLAC_BLOCK.to_bytes(2, "big") * 2 + bytes(6) + ((40000 << 44) | (15 << 36) | samples).to_bytes(8, "big")
    return b"".join([b"fLaC\x80\x00\x00\x22", info, bytes(16)] + parts), np.concatenate(data)


def _prepare_flac(case, seed):
    return dict(case=case, data=_flac(case["samples"], seed)[0])


def _run_flac(state):
    return {"samples": native.flac_decode(state["data"])}


# ------------------------------------------------------------------- serving

SERVE = [("PAL", "VHS", 40.0), ("NTSC", "VHS", 20.0), ("PAL", "SVHS", 40.0), ("NTSC", "VHS", 40.0)]


def _prepare_server(case, seed):
    windows = []
    for i in range(case["windows"]):
        system, tape, mhz = SERVE[i % len(SERVE)]
        g = synth._geometry(system)
        fields = max(2, int(case["ms"] * 1e3 / (g["lines"] * g["line_us"] / 2) - 1.5))
        rf = _pin(_capture(system, tape, mhz, fields, seed + 1000 * i, 2 * fields))
        outlen, lines = OUT[system]
        windows.append((system, tape, mhz, rf.numpy(),
                        _pinned((fields + 2) * lines * outlen, torch.int16).numpy().view(np.uint16)))
    server = native.Server(max(len(w[3]) for w in windows), workers=4)
    return dict(case=case, server=server, windows=windows)


def _run_server(state):
    server = state["server"]
    tickets = [server.submit(i, PROFILES[system], rf, seek=True, tbc_out=out, sample_rate_mhz=mhz,
                             tape_format=TAPES[tape])
               for i, (system, tape, mhz, rf, out) in enumerate(state["windows"])]
    result = {}
    for i, t in enumerate(tickets):
        r = server.wait(t)
        system, out = state["windows"][i][0], state["windows"][i][4]
        result["fields_%d" % i] = r.fields
        result["luma_%d" % i] = out[:r.fields * OUT[system][0] * OUT[system][1]].view(np.int16)
    return result


# ----------------------------------------------------------------- whole run

def _prepare_run(case, seed):
    rf = _capture(case["system"], "VHS", 40.0, case["fields"], seed, case["dropouts"]).cpu().numpy()
    # files go to memory where there is such a file system, so that no disk is timed
    folder = tempfile.TemporaryDirectory(dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
    address = rf.ctypes.data

    def read(user, destination, offset, count):
        count = max(0, min(count, len(rf) - offset))
        if count:
            ctypes.memmove(destination, address + 2 * offset, 2 * count)
        return count

    cfg = native.RunConfigV2()
    cfg.struct_size = ctypes.sizeof(cfg)
    cfg.profile = PROFILES[case["system"]]
    cfg.sample_rate_mhz = 40.0
    cfg.total_samples = len(rf)
    cfg.output_base_utf8 = os.path.join(folder.name, "capture").encode()
    cfg.overwrite = 1
    cfg.input_sample_format = native.INPUT_INT16
    cfg.device_decimation_factor = 1
    cfg.read_callback = native.READ_CB(read)
    cfg.decode_flags = native.DECODE_CHROMA if case["chroma"] else 0
    return dict(case=case, rf=rf, folder=folder, config=cfg, base=os.path.join(folder.name, "capture"),
                json=np.zeros(16384 + 2048 * case["fields"] + 128 * case["dropouts"], np.uint8))


def _run_run(state):
    r = native.RunResult()
    r.struct_size = ctypes.sizeof(r)
    native.check(native.load().vhsdecode_gb300_run(ctypes.byref(state["config"]), ctypes.byref(r)))
    base, json = state["base"], state["json"]
    json[:] = 0
    with open(base + ".tbc.json", "rb") as f:
        f.readinto(json)
    return {"fields": r.fields_written, "luma": np.memmap(base + ".tbc", np.int16, "r"),
            "chroma": np.memmap(base + "_chroma.tbc", np.int16, "r"),
            "json": json}


# ---------------------------------------------------------------------- cases

_PREPARE = {"session": _prepare_session, "pulses": _prepare_pulses, "flac": _prepare_flac,
            "server": _prepare_server, "run": _prepare_run}
_RUN = {"session": _run_session, "pulses": _run_pulses, "flac": _run_flac, "server": _run_server, "run": _run_run}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def exact(case, seed):
    if case["kind"] == "pulses":
        return _pulses_exact(case, seed)
    if case["kind"] == "flac":
        return {"samples": _flac(case["samples"], seed)[1]}
    return None      # decoded fields are whole numbers


def _decode_work(system, samples, decimation, sample_bytes, fields, chroma, svhs):
    outlen, lines = OUT[system]
    blocks = max(1, (samples // decimation - BLOCK) // STRIDE + 1)
    fft = 2.5 * BLOCK * 15                                   # a real transform of a block
    flops = blocks * ((9 if svhs else 5) * fft + 60.0 * BLOCK)   # transforms, demodulation and envelope
    pixels = fields * lines * outlen
    flops += pixels * 40.0                                   # 16 taps, position and conversion
    if chroma:
        flops += blocks * 2 * 4 * 9.0 * BLOCK + pixels * (32.0 + 2 * 4 * 9.0)   # band-passes and the second source
    return samples * sample_bytes + pixels * (4 if chroma else 2), flops


def work(case):
    kind = case["kind"]
    if kind == "pulses":
        return {"bytes": 4.0 * case["samples"] + 16.0 * (case["samples"] // 2542 + 1), "flops": 1.0 * case["samples"]}
    if kind == "flac":
        return {"bytes": 3.4 * case["samples"], "flops": 24.0 * case["samples"]}
    if kind == "server":
        bytes_, flops = 0.0, 0.0
        for i in range(case["windows"]):
            system, tape, mhz = SERVE[i % len(SERVE)]
            g = synth._geometry(system)
            fields = max(2, int(case["ms"] * 1e3 / (g["lines"] * g["line_us"] / 2) - 1.5))
            b, f = _decode_work(system, _samples(system, mhz, fields), 1, 2, fields, False, tape == "SVHS")
            bytes_, flops = bytes_ + b, flops + f
        return {"bytes": bytes_, "flops": flops}
    rate, dec = case.get("mhz", 40.0), case.get("decimation", 1)
    sub = case.get("tape") == "SVHS" or case.get("speed", "SP") != "SP"
    b, f = _decode_work(case["system"], _samples(case["system"], rate * dec, case["fields"]), dec,
                        4 if case.get("dtype") == "float32" else 2, case["fields"], case["chroma"], sub)
    return {"bytes": float(b), "flops": float(f)}
