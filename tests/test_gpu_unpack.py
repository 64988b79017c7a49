"""Unpacking by 16-bit lanes and by whole words, and the mask's quartiles, bit for bit against the
oracle: channels that end inside a group, the largest sums that the narrow integers hold and the
first ones past them, zapped channels, pixels that are equal."""
import numpy as np
import pytest

from test_gpu_pipeline import oracle_rows

pytestmark = pytest.mark.gpu

# channels, samples per block, td, fd, zapthre
CASES = [
    (16, 64, 1, 1, 0.0), (20, 65, 1, 1, 4.0), (36, 127, 1, 2, 0.0), (100, 640, 2, 4, 4.0), (132, 1000, 5, 1, 4.0),
    (128, 4000, 40, 1, 0.0), (128, 4100, 41, 1, 0.0), (64, 2000, 20, 2, 0.0), (64, 2100, 21, 2, 0.0),
    (72, 640, 5, 8, 0.0), (144, 400, 2, 16, 0.0), (144, 600, 3, 16, 0.0), (1000, 500, 1, 2, 4.0),
    (999, 300, 1, 1, 4.0), (30, 300, 3, 3, 0.0), (18, 200, 2, 2, 0.0),
]


@pytest.mark.parametrize("C,ndump,td,fd,zap", CASES)
def test_blocks_match_oracle(tx, oracle, C, ndump, td, fd, zap):
    from transientx_gb300 import SinglePulse, synth
    ts = 1e-3
    fil = synth.Filterbank(C, ts, synth.band(C, 1500.0, 1200.0), 2 * ndump, 5, pulses=[], sines=[], impulses=[])
    rows = [SinglePulse(td=td, fd=fd, dms=0.0, ddm=1.0, ndm=4, maxw=0.05, bswidth=0.0)]
    orow = oracle_rows(oracle, rows, fil, ndump, tx, zapthre=zap)[0]
    rng = np.random.default_rng(C * td + fd)
    with tx.Search(rows, C, ts, fil.freqs, ndump, flags=tx.FLAG_KEEP_SERIES, zapthre=zap) as s:
        for b in range(2):
            raw = rng.integers(0, 256, (ndump, C)).astype(np.uint8)
            raw[:, C // 2] = 255
            raw[:-1, C - 1] = 255  # all but one sample at the top
            raw[:, C // 3] = np.where(np.arange(ndump) % 50 == 0, 255, 0)  # kurtosis: zapped
            s.push_block(raw)
            s.sync()
            orow.run(raw)
            np.testing.assert_array_equal(s.block(0), orow.block(), err_msg=f"block {b}")


@pytest.mark.parametrize("C,ndump,td,fd", [(8, 4, 4, 8), (8, 12, 4, 4), (64, 2048, 4, 4), (130, 515, 1, 1), (512, 4096, 2, 2)])
@pytest.mark.parametrize("levels", [1, 2, 40])
def test_mask_quartiles_match_oracle(tx, oracle, C, ndump, td, fd, levels):
    from transientx_gb300 import SinglePulse, synth
    ts = 1e-3
    fil = synth.Filterbank(C, ts, synth.band(C, 1500.0, 1200.0), 2 * ndump, 5, pulses=[], sines=[], impulses=[])
    rows = [SinglePulse(td=1, fd=1, dms=0.0, ddm=1.0, ndm=4, maxw=0.005, bswidth=0.0,
                        rfilist=[["mask", str(td), str(fd)]])]
    orow = oracle_rows(oracle, rows, fil, ndump, tx, zapthre=0.0)[0]
    rng = np.random.default_rng(levels)
    with tx.Search(rows, C, ts, fil.freqs, ndump, flags=tx.FLAG_KEEP_SERIES, zapthre=0.0) as s:
        for b in range(2):
            raw = (100 + rng.integers(0, levels, (ndump, C))).astype(np.uint8)
            raw[ndump // 2, :: max(1, C // 3)] = 250
            s.push_block(raw)
            s.sync()
            orow.run(raw)
            np.testing.assert_array_equal(s.block(0), orow.block(), err_msg=f"block {b}")
