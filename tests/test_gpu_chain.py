"""Blocks pushed one after another, so that each block's kernels overlap the ends of those before
them, against blocks with a wait after each: the same series, points and masks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,ndump,prec", [(16, 96, "fp32"), (64, 512, "fp32"), (100, 1000, "fp16"), (256, 4096, "bf16")])
@pytest.mark.parametrize("rfi", [[], [["kadaneF", "8", "4"], ["zdot"]], [["mask", "2", "2"], ["kadaneT", "4", "4"], ["zero"]]])
def test_blocks_in_a_row_equal_blocks_apart(tx, C, ndump, prec, rfi):
    f = 1500.0 - 300.0 / C * np.arange(C)
    rows = [tx.SinglePulse(td=t, fd=1, dms=0.0, ddm=2.0, ndm=40 * t, maxw=0.01, thre=4.0, bswidth=0.05, rfilist=rfi)
            for t in (1, 2, 4)]
    rng = np.random.default_rng(C)
    blocks = [rng.integers(60, 200, (ndump, C)).astype(np.uint8) for _ in range(24)]
    out = []
    for apart in (True, False):
        with tx.Search(rows, C, 5e-4, f, ndump, precision=prec, flags=tx.FLAG_KEEP_SERIES, zapthre=4.0,
                       cand_capacity=1 << 18) as s:
            for b in blocks:
                s.push_block(b)
                if apart:
                    s.sync()
            s.sync()
            out.append([(s.mask(), s.block(r), s.timdata(r), s.candidates(r)) for r in range(3) if s.row_info(r).gated])
    assert len(out[0]) == len(out[1]) >= 1
    for a, b in zip(*out):
        for u, v in zip(a, b):
            np.testing.assert_array_equal(u, v)
