"""The channel zap's quartiles: values that one pass tells apart, that only the last digits do, and
equal ones, few channels and many, bit for bit against the oracle's blocks."""
import numpy as np
import pytest

from test_gpu_pipeline import oracle_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 8, 63, 256, 1025, 4100])
@pytest.mark.parametrize("kind", ["noise", "equal", "pairs", "nearly"])
def test_zapped_blocks_match_oracle(tx, oracle, C, kind):
    from transientx_gb300 import SinglePulse, synth
    ndump, ts = 256, 1e-3
    fil = synth.Filterbank(C, ts, synth.band(C, 1500.0, 1200.0), 2 * ndump, 5, pulses=[], sines=[], impulses=[])
    rows = [SinglePulse(td=1, fd=1, dms=0.0, ddm=1.0, ndm=3, maxw=0.01, bswidth=0.0)]
    orow = oracle_rows(oracle, rows, fil, ndump, tx, zapthre=3.0)[0]
    rng = np.random.default_rng(C)
    with tx.Search(rows, C, ts, fil.freqs, ndump, flags=tx.FLAG_KEEP_SERIES, zapthre=3.0) as s:
        for b in range(2):
            raw = rng.integers(60, 200, (ndump, C)).astype(np.uint8)
            if kind == "equal":
                raw[:] = raw[:, :1]
            elif kind == "pairs":
                raw[:, 1::2] = raw[:, : C // 2 * 2: 2]
            elif kind == "nearly":  # one sample differs by one
                raw[:] = raw[:, :1]
                raw[rng.integers(0, ndump, C), np.arange(C)] += 1
            raw[:, C // 2] = np.where(np.arange(ndump) % 40 == 0, 255, 100)
            s.push_block(raw)
            s.sync()
            orow.run(raw)
            np.testing.assert_array_equal(s.block(0), orow.block(), err_msg=f"block {b}")
