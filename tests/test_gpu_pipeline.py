"""Decodes whose host and device work overlap, where the order of the two can go wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK, STRIDE = 32768, 30720


@pytest.mark.parametrize("mhz", [93.0, 100.0])
def test_last_launch_ends_before_the_one_ahead(gpu, mhz):
    # 41 blocks from pinned memory are demodulated by two launches, of 40 blocks
    # and of one, on two streams.  The first 40 hold dropouts, so the spike repair
    # makes the first launch the later one to end; a field's span is longer than
    # the capture at these rates, so no field work waits for either.
    import torch
    from vhsd_gb300 import native, synth
    rf, _ = synth.generate(synth.pal_vhs(fs=mhz * 1e6, fields=1, seed=4, snr_db=40.0))
    rf = np.resize(rf, 40 * STRIDE + BLOCK).copy()
    for b in range(1, 40):
        rf[b * STRIDE + 9000:b * STRIDE + 9400] //= 200
    pinned = torch.from_numpy(rf).pin_memory()
    with native.Session(native.PROFILE_PAL, len(rf), sample_rate_mhz=mhz) as s:
        for _ in range(20):
            r = s.decode(pinned.numpy())
            assert (r.fields, r.blocks, r.segments) == (0, 41, 2)
            assert r.repaired_blocks > 0 and r.demod_ms > 0.0


def _long_pulses(rf, cfg):
    """`rf` with hsync pulses of 9 us on five lines of every field."""
    from vhsd_gb300 import synth
    g = synth._geometry(cfg.system)
    line = g["line_us"] * cfg.fs / 1e6
    out = rf.copy()
    n = int(6e-6 * cfg.fs)
    tip = np.round(8000.0 * np.cos(2 * np.pi * np.arange(n) * (cfg.ire0 + cfg.hz_ire * cfg.vsync_ire) / cfg.fs))
    for field in range(int(cfg.fields) + 1):
        for k in (60, 100, 140, 180, 220):
            at = int((cfg.lead_lines + field * (g["lines"] // 2 + 1) + k) * line + 3e-6 * cfg.fs)
            if at + n <= len(out):
                out[at:at + n] = tip
    return out


def _rescues(capfd):
    return [int(line.split("rescue_fetches=")[1].split()[0]) for line in capfd.readouterr().err.splitlines()
            if "rescue_fetches=" in line]


def test_rescue_reads_finished_blocks(gpu, monkeypatch, capfd):
    # the long-hsync rescue reads sync samples of blocks that the running
    # demodulator has finished: the same fields, lines and pictures whichever way
    # the capture comes in, also right after a decode of another one (whose
    # samples an early read would find), and the fields of the double-precision
    # decode, which reads after its whole demodulation
    import torch
    from vhsd_gb300 import native, synth
    monkeypatch.setenv("VHSD_STAGE_TIMING", "1")
    cfg = synth.ntsc_vhs(fields=12, seed=11, snr_db=40.0)
    clean, _ = synth.generate(cfg)
    rf = _long_pulses(clean, cfg)
    pinned, dev = torch.from_numpy(rf).pin_memory(), torch.from_numpy(rf).cuda()
    with native.Session(native.PROFILE_NTSC, len(rf), precision=native.PRECISION_FP64_PLAIN) as s:
        r = s.decode(rf)
        spans = [(s.field(i).span_start, bool(s.field(i).is_first_field)) for i in range(r.fields)]
    assert len(spans) >= 11
    capfd.readouterr()
    want = None
    with native.Session(native.PROFILE_NTSC, len(rf)) as s:
        for source in ("device", "pinned", "pageable") * 4:
            s.decode(clean)
            capfd.readouterr()
            if source == "device":
                r = s.decode(None, device_ptr=dev.data_ptr(), count=len(rf))
            else:
                r = s.decode(pinned.numpy() if source == "pinned" else rf)
            assert _rescues(capfd)[0] > 0
            assert [(s.field(i).span_start, bool(s.field(i).is_first_field)) for i in range(r.fields)] == spans
            got = (s.tbc(), np.concatenate([s.lines(i) for i in range(r.fields)]))
            want = want or got
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), source


def test_rescue_does_not_wait_for_the_demodulator(gpu, monkeypatch, capfd):
    # 3000 blocks on the device, one launch, the first field only: its blocks
    # and the rescue's samples are there after a few of the 40 rounds of blocks
    import torch
    from vhsd_gb300 import native, synth
    monkeypatch.setenv("VHSD_STAGE_TIMING", "1")
    cfg = synth.ntsc_vhs(fields=4, seed=12, snr_db=40.0)
    rf = np.resize(_long_pulses(synth.generate(cfg)[0], cfg), 2999 * STRIDE + BLOCK)
    dev = torch.from_numpy(rf).cuda()
    with native.Session(native.PROFILE_NTSC, len(rf)) as s:
        times = []
        for _ in range(5):
            capfd.readouterr()
            r = s.decode(None, device_ptr=dev.data_ptr(), count=len(rf), max_fields=1)
            assert r.fields == 1 and r.segments == 1 and _rescues(capfd)[0] > 0
            times.append((r.host_ms, r.demod_ms))
        host, demod = np.median(times, axis=0)
        assert host < 0.5 * demod, (host, demod)


@pytest.mark.parametrize("mhz,fields,crowds,segments", [
    (40.0, 10, [(60, 2)], 1),                        # inside the second segment of blocks (of 40, 128 and the rest)
    (40.0, 10, [(20, 1), (200, 2)], 2),              # the first and the third
    (40.0, 10, [(165, 6)], 2),                       # across the end of the second
    (20.0, 14, [(10, 2), (36, 7)], 2),               # two in one segment, the later one across its end
])
def test_crowded_blocks_scan_their_segment(gpu, mhz, fields, crowds, segments):
    # blocks with more edges than a record holds (a 0.4 MHz square wave around
    # the threshold: 160 a chunk at 40 MSPS, 320 at 20): the rest of their segment
    # is scanned on the device, two kernels each, the others keep their records.
    # The fields are those of the double-precision decode's scan of its own
    # stream, whichever way the capture comes in.
    import torch
    from oracle import formats
    from vhsd_gb300 import native, synth
    clean, _ = synth.generate(synth.ntsc_vhs(fs=mhz * 1e6, fields=fields, seed=21, snr_db=40.0))
    fmt = formats.get("NTSC")["sys"]
    rf = clean.copy()
    for block, count in crowds:
        t = np.arange(count * STRIDE)
        ire = np.where((t * 0.8e6 / (mhz * 1e6)).astype(np.int64) % 2 == 0, -60.0, 20.0)
        wave = 8000.0 * np.cos(2 * np.pi * np.cumsum(fmt["ire0"] + fmt["hz_ire"] * ire) / (mhz * 1e6))
        rf[block * STRIDE + 8000:block * STRIDE + 8000 + len(t)] = np.round(wave)
    pinned, dev = torch.from_numpy(rf).pin_memory(), torch.from_numpy(rf).cuda()

    def spans(s, r):
        return [(s.field(i).span_start, bool(s.field(i).is_first_field)) for i in range(r.fields)]

    with native.Session(native.PROFILE_NTSC, len(rf), sample_rate_mhz=mhz,
                        precision=native.PRECISION_FP64_PLAIN) as s:
        want = spans(s, s.decode(rf))
    assert len(want) >= fields // 2
    pictures = None
    with native.Session(native.PROFILE_NTSC, len(rf), sample_rate_mhz=mhz) as s:
        for source in ("device", "pinned", "pageable"):
            launches = []
            for x in (clean, rf):
                if x is rf and source == "device":
                    r = s.decode(None, device_ptr=dev.data_ptr(), count=len(rf))
                else:
                    r = s.decode(pinned.numpy() if x is rf and source == "pinned" else x)
                assert r.fields > 0
                launches.append(r.kernel_launches - r.segments)
            assert launches[1] - launches[0] == 2 * segments, source
            assert spans(s, r) == want, source
            got = (s.tbc(), np.concatenate([s.lines(i) for i in range(r.fields)]))
            pictures = pictures or got
            assert all(np.array_equal(a, b) for a, b in zip(got, pictures)), source


def test_failed_decode_leaves_nothing_behind(gpu):
    # a segment with more edges than the host accepts (a 0.4 MHz wave for 128
    # blocks at 20 MSPS) fails the decode while thousands of blocks are still to
    # come; once the call has returned, nothing reads the caller's buffer any
    # more, and a decode on another stream is what it is in a new session
    import torch
    from oracle import formats
    from vhsd_gb300 import native, synth
    clean, _ = synth.generate(synth.ntsc_vhs(fs=20e6, fields=4, seed=31, snr_db=40.0))
    fmt = formats.get("NTSC")["sys"]
    t = np.arange(140 * STRIDE)
    ire = np.where((t * 0.8e6 / 20e6).astype(np.int64) % 2 == 0, -60.0, 20.0)
    wave = 8000.0 * np.cos(2 * np.pi * np.cumsum(fmt["ire0"] + fmt["hz_ire"] * ire) / 20e6)
    rf = np.resize(clean, 2999 * STRIDE + BLOCK)
    rf[36 * STRIDE:36 * STRIDE + len(t)] = np.round(wave)
    pinned = torch.from_numpy(rf).pin_memory()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with native.Session(native.PROFILE_NTSC, len(clean), sample_rate_mhz=20.0) as s:
        s.decode(clean)
        want = s.tbc()
    with native.Session(native.PROFILE_NTSC, len(rf), sample_rate_mhz=20.0) as s:
        for _ in range(3):
            s.set_stream(first.cuda_stream)
            with pytest.raises(native.NativeError, match="capacity"):
                s.decode(pinned.numpy())
            assert first.query()
            s.set_stream(second.cuda_stream)
            s.decode(clean)
            assert np.array_equal(s.tbc(), want)


@pytest.mark.parametrize("precision", ["FP32_FUSED", "FP64_PLAIN"])
def test_chroma_stream_needs_no_device_memory(gpu, precision):
    # reading the chroma channel of a decode allocates nothing on the device, so
    # it cannot fail where the decode did not; any range of it is the part of
    # the whole, across block ends too
    import torch
    from vhsd_gb300 import native, synth
    rf, _ = synth.generate(synth.ntsc_vhs(fields=2, seed=41, snr_db=40.0))
    rf = np.resize(rf, 199 * STRIDE + BLOCK)
    with native.Session(native.PROFILE_NTSC, len(rf), precision=getattr(native, "PRECISION_" + precision)) as s:
        r = s.decode(rf, chroma=True, demod_only=True)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        whole = s.stream(3, 0, r.stream_samples)
        assert torch.cuda.mem_get_info()[0] == free
        assert np.any(whole)
        for start, count in ((0, 1), (STRIDE - 1, 2), (5 * STRIDE, STRIDE), (7 * STRIDE + 11, 3 * STRIDE),
                             (r.stream_samples - 5, 5), (r.stream_samples, 0)):
            assert np.array_equal(s.stream(3, start, count), whole[start:start + count]), (start, count)


@pytest.mark.parametrize("blocks,limit,batch", [(128, 100, 64), (64, 3, 2), (64, 1, 1)])
def test_plain_workspace_takes_the_room_there_is(gpu, monkeypatch, blocks, limit, batch):
    # a device without room for the plain demodulator's whole batch gets half as
    # many blocks until they fit, down to one; the streams are the same (29
    # kernels a batch)
    from vhsd_gb300 import native, synth
    rf, _ = synth.generate(synth.pal_vhs(fields=1, seed=51, snr_db=40.0, dropouts=10))
    rf = np.resize(rf, (blocks - 1) * STRIDE + BLOCK)

    def streams():
        with native.Session(native.PROFILE_PAL, len(rf), precision=native.PRECISION_FP64_PLAIN) as s:
            r = s.decode(rf, demod_only=True)
            return r.kernel_launches, [s.stream(c, 0, r.stream_samples) for c in range(3)]

    kernels, want = streams()
    assert kernels == 29
    monkeypatch.setenv("VHSD_PLAIN_BATCH_LIMIT", str(limit))
    kernels, got = streams()
    assert kernels == 29 * (blocks // batch)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_chroma_finds_room_beside_the_plain_workspace(gpu, monkeypatch):
    # buffers that a later decode adds (here the chroma workspace, refused beside
    # a plain workspace of many blocks) take the room of the batches
    from vhsd_gb300 import native, synth
    rf, _ = synth.generate(synth.ntsc_vhs(fields=2, seed=52, snr_db=40.0))
    kw = dict(precision=native.PRECISION_FP64_PLAIN)
    with native.Session(native.PROFILE_NTSC, len(rf), **kw) as s:
        s.decode(rf, chroma=True)
        want = s.tbc(), s.chroma()
    monkeypatch.setenv("VHSD_FORCE_CHROMA_WORKSPACE_FAILURE", "batched")
    with native.Session(native.PROFILE_NTSC, len(rf), **kw) as s:
        s.decode(rf)
        s.decode(rf, chroma=True)
        assert all(np.array_equal(a, b) for a, b in zip((s.tbc(), s.chroma()), want))
