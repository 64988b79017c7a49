"""The preprocessing passes at the edges of their tiles, bit for bit against the oracle: the
equalize apply that brings the first filter's downsampled block, the per-channel statistics
and fit of zdot (cached and uncached rows), the baseline's sums, the channel zap's sums."""
import numpy as np
import pytest

from test_gpu_pipeline import oracle_rows

pytestmark = pytest.mark.gpu

# channels, samples per block, td, fd, filters, baseline seconds, zapthre
CASES = [
    (64, 2048, 1, 1, [["kadaneF", "8", "4"], ["zdot"]], 0.1, 4.0),
    (61, 1999, 1, 1, [["kadaneF", "8", "4"], ["zdot"]], 0.1, 4.0),   # a rest in both axes
    (33, 1029, 1, 1, [["kadaneF", "4", "3"]], 0.0, 0.0),             # no baseline, 33 = 11 * 3
    (16, 1040, 1, 1, [["kadaneF", "16", "16"], ["zero"]], 0.05, 4.0),
    (130, 515, 1, 1, [["mask", "4", "2"], ["kadaneF", "8", "1"]], 0.02, 4.0),
    (40, 700, 1, 1, [["kadaneT", "4", "4"], ["kadaneF", "4", "4"]], 0.3, 4.0),
    (12, 7, 1, 1, [["kadaneF", "8", "4"]], 0.1, 0.0),                # a block shorter than td
    (3, 600, 1, 1, [["kadaneF", "8", "4"], ["zdot"]], 0.1, 4.0),     # fewer channels than fd
    (24, 1200, 3, 2, [["kadaneF", "5", "2"], ["zdot"]], 0.1, 4.0),   # td not a power of two
    (8, 16384, 1, 1, [["zdot"]], 0.0, 4.0),                          # the longest cached row
    (8, 16385, 1, 1, [["zdot"]], 0.0, 4.0),
    (5, 70001, 1, 1, [["kadaneF", "8", "1"], ["zdot"]], 4.5, 4.0),   # more than 64 runs, long baseline
    (260, 513, 1, 1, [["zdot"]], 0.1, 3.0),
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[1]}-{c[4][0][0]}{'-'.join(c[4][0][1:])}" for c in CASES])
def test_preprocessed_block_matches_oracle(tx, oracle, case):
    from transientx_gb300 import SinglePulse, synth
    C, ndump, td, fd, rfi, bw, zap = case
    ts = 1e-3
    f = synth.band(C, 1500.0, 1200.0)
    ndump = ndump // td * td
    fil = synth.Filterbank(C, ts, f, 2 * ndump, 3 + C, pulses=[(0.3 * ndump * ts, 10.0, 5e-3, 60.0)],
                           sines=[(C // 2, 15.0, 0.07, 0.3)],
                           impulses=[(0.6 * ndump * ts, 9, 12.0)])
    rows = [SinglePulse(td=td, fd=fd, dms=0.0, ddm=1.0, ndm=4, maxw=0.01, rfilist=rfi, bswidth=bw, widthlimit=0.05,
                        threKadaneF=5.0)]
    orow = oracle_rows(oracle, rows, fil, ndump, tx, zapthre=zap)[0]
    with tx.Search(rows, C, ts, f, ndump, flags=tx.FLAG_KEEP_SERIES, zapthre=zap) as s:
        for b in range(2):
            raw = fil.generate(b * ndump, ndump)
            s.push_block(raw)
            s.sync()
            orow.run(raw)
            np.testing.assert_array_equal(s.block(0), orow.block(), err_msg=f"block {b}")
            if rfi[0][0] == "kadaneF":
                np.testing.assert_array_equal(s.zap_ranges(0, 0), orow.zap_ranges(0))
