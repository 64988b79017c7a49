"""Stage 2 over the widths of DM groups that its chunks of 4 to 28 DMs divide, evenly or not, against
the subband series summed in order on the host: the same additions, so bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("G", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 24, 25, 28, 30, 33, 36, 40, 56, 64])
def test_series_are_the_ordered_sums_of_the_subbands(tx, G, prec):
    C, nsub, ndump, ndm = 48, 6, 700, 2 * G + (G + 1) // 2
    f = 1500.0 - 5.0 * np.arange(C)
    row = tx.SinglePulse(td=1, fd=1, dms=2.0, ddm=0.4, ndm=ndm, maxw=0.005, nsub=nsub, dm_group=G)
    rng = np.random.default_rng(G)
    with tx.Search([row], C, 2e-4, f, ndump, precision=prec, flags=tx.FLAG_KEEP_SERIES, zapthre=0.0) as s:
        n = int(s.row_info(0).offset // ndump) + 3
        checked = 0
        for _ in range(n):
            s.push_block(rng.integers(60, 200, (ndump, C)).astype(np.uint8))
            s.sync()
            if not s.row_info(0).gated:
                continue
            got = s.timdata(0)
            for k in range(ndm):
                sub = s.subdata(k)
                want = np.zeros(sub.shape[1], np.float32)
                for b in range(nsub):
                    want = want + sub[b]
                np.testing.assert_array_equal(got[k], want, err_msg=f"DM {k}")
            checked += 1
        assert checked >= 1
