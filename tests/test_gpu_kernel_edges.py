"""Kernels at the sizes where their own tiling can go wrong, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCK, STRIDE = 32768, 30720


@pytest.mark.parametrize("system,mhz,insert", [("PAL", 40.0, 0), ("NTSC", 40.0, 0), ("NTSC", 20.0, 0),
                                               ("NTSC", 93.0, 0), ("PAL", 40.0, 301), ("NTSC", 40.0, -257)])
def test_float_tbc_matches_binary64(gpu, system, mhz, insert):
    # the float TBC of the device's own streams and lines, luma and chroma in
    # one pass, against the binary64 resampler: lines staged in shared memory
    # at several sample rates, and (samples inserted or cut in mid-field) lines
    # too long or too short for the stage.  The pair sums carry about 2^-46, so
    # a float output differs only within 2^-22 of a rounding boundary; 1e-5 of
    # the samples is 20 times that rate, and a uint16 then differs by 1.
    from oracle import field, formats, sync, tbc
    from vhsd_gb300 import native, synth
    make = synth.pal_vhs if system == "PAL" else synth.ntsc_vhs
    rf, info = synth.generate(make(fs=mhz * 1e6, fields=2, seed=3, snr_db=40.0))
    if insert:
        at = int(info["lead"] + 0.6 * info["field_samples"])
        rf = np.concatenate([rf[:at], rf[at - insert:]])   # repeats `insert` samples, or cuts them
    fmt = formats.get(system)
    sp = sync.SyncParams(fmt, mhz * 1e6)
    smoothing = fmt["sys"]["frame_lines"] / 2.0
    nominal = float(round(fmt["sys"]["line_period"] * sp.mhz))
    prof = native.PROFILE_PAL if system == "PAL" else native.PROFILE_NTSC
    with native.Session(prof, len(rf), sample_rate_mhz=mhz) as s:
        r = s.decode(rf, chroma=True)
        assert r.fields >= 2
        luma = s.tbc()
        for i in range(r.fields):
            fi = s.field(i)
            length = r.stream_samples - fi.span_start
            first = field.output_first_line(sp, bool(fi.is_first_field))
            args = (s.lines(i), first, sp.output_lines, sp.outlinelen, nominal, smoothing)
            hz = tbc.resample_field(s.stream(0, fi.span_start, length), *args)
            want = tbc.to_u16(hz, sp, formats.output_scale(fmt), fmt["sys"]["outputZero"]).astype(np.int64)
            diff = np.abs(luma[i].ravel().astype(np.int64) - want)
            assert diff.max() <= 1 and np.mean(diff != 0) <= 1e-5, (i, diff.max(), np.mean(diff != 0))
            want = tbc.resample_field(s.stream(3, fi.span_start, length), *args)
            got = s.chroma_stage(i, 0)
            assert np.mean(got != want) <= 1e-5, (i, np.mean(got != want))
            assert np.max(np.abs(got - want)) <= 2.0 ** -23 * np.max(np.abs(want))


@pytest.mark.parametrize("nblocks,dtype", [(1, "int16"), (1, "float32"), (7, "float32"), (33, "int16"),
                                           (800, "int16"), (801, "int16"), (865, "float32")])
def test_chroma_block_stage_edges(gpu, nblocks, dtype):
    # the block band-pass is bit-exact whatever the block's place in its CTA:
    # one block, a part of a warp, one more than a CTA, and both sides of the
    # line between 32 and 64 blocks a CTA (800 blocks); full-scale noise, so
    # every sample of the odd extension and of the last chunk matters
    from oracle import chroma, formats
    from vhsd_gb300 import native
    rng = np.random.default_rng(nblocks)
    rf = rng.integers(-32768, 32768, (nblocks - 1) * STRIDE + BLOCK).astype(np.int16)
    if dtype == "float32":
        rf = (rf + rng.random(len(rf), np.float32)).astype(np.float32)
    cp = chroma.ChromaParams(formats.get("NTSC"))
    with native.Session(native.PROFILE_NTSC, len(rf)) as s:
        s.decode(rf, demod_only=True, chroma=True)
        for b in sorted({0, min(nblocks - 1, 31), min(nblocks - 1, 32), min(nblocks - 1, 64), nblocks - 1}):
            want = chroma.chroma_stream(rf, cp, b, 1)
            assert np.array_equal(s.stream(3, b * STRIDE, STRIDE), want), b


@pytest.mark.parametrize("tape,nblocks", [("VHS", 1), ("VHS", 128), ("VHS", 129), ("SVHS", 129)])
def test_fp64_batches(gpu, tape, nblocks):
    # the double-precision demodulator takes the blocks in batches (at most 128
    # of equal size): a block's samples are the same wherever it lies in a
    # batch, and within 1 Hz of the oracle's (the bound of the stream tests;
    # both compute in binary64, whose rounding is below 1e-6 Hz, but a float
    # angle beside a rounding boundary moves a sample by up to 0.4 Hz).  Dropouts
    # make some blocks take the spike repair.
    from oracle import demod, filters, formats
    from vhsd_gb300 import native, synth
    make = synth.pal_svhs if tape == "SVHS" else synth.pal_vhs
    rf, _ = synth.generate(make(fields=4, seed=8, snr_db=40.0, dropouts=40))
    rf = np.resize(rf, (nblocks - 1) * STRIDE + BLOCK)
    fmt = formats.get("PAL", tape)
    filt = filters.FilterSet(fmt, 40e6)
    dmax = (fmt["sys"]["ire0"] + fmt["sys"]["hz_ire"] * 100.0) * 2.0
    kw = dict(precision=native.PRECISION_FP64_PLAIN,
              tape_format=native.FORMAT_SVHS if tape == "SVHS" else native.FORMAT_VHS)
    with native.Session(native.PROFILE_PAL, len(rf), **kw) as s:
        s.decode(rf, demod_only=True)
        for b in sorted({0, nblocks // 2 - 1, nblocks // 2, nblocks - 1} - {-1}):
            got = [s.stream(c, b * STRIDE, STRIDE) for c in range(3)]
            with native.Session(native.PROFILE_PAL, BLOCK, **kw) as one:
                one.decode(rf[b * STRIDE:b * STRIDE + BLOCK], demod_only=True)
                for c in range(3):
                    assert np.array_equal(got[c], one.stream(c, 0, STRIDE)), (b, c)
            want = demod.demod_stream(rf, filt, 40e6, dmax, b, 1)
            assert np.max(np.abs(got[0] - want[0])) < 1.0 and np.max(np.abs(got[1] - want[1])) < 1.0, b


@pytest.mark.parametrize("blocksize,kind", [(4096, "spikes"), (192, "spikes"), (4608, "noise"), (256, "mixed"),
                                            (16, "noise"), (1152, "quiet")])
def test_flac_frames_lossless(gpu, blocksize, kind):
    # four lanes a frame, eight frames a warp: codes far longer than the bits a
    # lane holds (a spike of 60000 in a silent partition is a 60000-bit run of
    # zeros), every predictor order beside constant and verbatim frames in one
    # warp, blocks shorter than a predictor, a short last frame
    from vhsd_gb300 import ldf, native
    rng = np.random.default_rng(blocksize)
    n = 24 * blocksize + 7
    x = np.zeros(n, np.int64)
    if kind == "noise":
        x = rng.integers(-32768, 32768, n)
    elif kind == "quiet":
        x = rng.integers(-1, 2, n)
    else:
        at = rng.integers(0, n, n // 150)
        x[at] = rng.integers(-32768, 32768, len(at))
    if kind == "mixed":
        t = np.arange(n)
        wave = (9000 * np.sin(t * 0.9) + 6000 * np.sin(t * 0.11) + rng.normal(0, 30, n)).astype(np.int64)
        frame = t // blocksize
        x = np.where(frame % 4 == 0, x, np.where(frame % 4 == 1, wave, np.where(frame % 4 == 2, 77, wave // 16)))
    x = x.astype(np.int16)
    assert np.array_equal(native.flac_decode(ldf.write(x, blocksize=blocksize, seed=blocksize)), x)


@pytest.mark.parametrize("n", [1, 31, 32, 1024, 1025, 8191, 8193, 262143, 262144, 262145])
def test_pulse_scan_lengths(gpu, n):
    # one warp, a ragged last word, one CTA, eight of them, and both sides of
    # the line between one cluster and two passes; runs of NaN across words,
    # warps and CTAs keep the state.  Integer work: identical.
    from oracle import native as onative
    from vhsd_gb300 import native
    rng = np.random.default_rng(n)
    x = rng.random(n) * 20.0 - 10.0
    x[rng.integers(0, 20, n) == 0] = np.nan
    for at in (n // 8 - 40, n // 2 - 700):
        if at > 0:
            x[at:at + 1400] = np.nan
    for high in (0.3, -9.9, 11.0):
        assert native.find_pulses(x, high, 1, 64) == onative.find_pulses(x, high, 1, 64)


@pytest.mark.parametrize("damage", ["none", "nan_block", "nan_start", "crowded"])
def test_pulse_edges_of_blocks(gpu, damage):
    # the fused demodulator's edge records against the plain path's scan of its
    # own stream: blocks without a sample (one NaN makes its whole block NaN;
    # the first block's, and with it the state before any sample), and chunks
    # with more edges than a record holds (a 0.4 MHz square wave around the
    # threshold: 160 a chunk), which sends the stream through the pulse scan.
    # Whole numbers: identical.
    from oracle import formats
    from vhsd_gb300 import native, synth
    rf, _ = synth.generate(synth.config("pal_small"))
    clean = rf.astype(np.float32)
    x = clean.copy()
    at = len(x) * 2 // 3
    if damage == "nan_block":
        x[at] = np.nan
    elif damage == "nan_start":
        x[5] = np.nan
    elif damage == "crowded":
        fmt = formats.get("PAL")["sys"]
        t = np.arange(100000)
        ire = np.where((t * 0.8e6 / 40e6).astype(np.int64) % 2 == 0, -60.0, 20.0)
        x[at:at + len(t)] = 8000.0 * np.cos(2 * np.pi * np.cumsum(fmt["ire0"] + fmt["hz_ire"] * ire) / 40e6)
    got = []
    for precision in (native.PRECISION_FP32_FUSED, native.PRECISION_FP64_PLAIN):
        with native.Session(native.PROFILE_PAL, len(x), precision=precision) as s:
            r = s.decode(x)
            got.append([(s.field(i).span_start, bool(s.field(i).is_first_field)) for i in range(r.fields)])
            if precision == native.PRECISION_FP32_FUSED:
                scanned = r.kernel_launches - s.decode(clean).kernel_launches
    assert got[0] and got[0] == got[1]
    if damage == "crowded":   # a clean decode of as many fields has no pulse scan
        assert scanned > 0
