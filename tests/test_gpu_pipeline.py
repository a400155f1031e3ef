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
