"""Stage 1 from tensor memory, and stage 2 as it is by default, against the shared-memory shapes over
plans at their edges: the same additions in the same order, so the series are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# channels, subbands, DM group, DMs, samples per block, DM step, what it is
PLANS = [
    (16, 16, 1, 5, 600, 1.0, "one channel a subband, one DM a group"),
    (64, 8, 4, 260, 512, 1.0, "65 groups of 4: a second pass of one group"),
    (64, 8, 4, 256, 511, 1.0, "64 groups, a tile but one sample"),
    (61, 7, 5, 23, 1000, 2.0, "uneven subbands, a last group of 3"),
    (48, 4, 16, 33, 37, 0.5, "a block shorter than a lane row, 17th DM alone"),
    (96, 3, 24, 200, 1537, 0.05, "32 channels a subband, groups of 24"),
    (40, 2, 33, 100, 900, 0.3, "groups wider than 32"),
    (32, 4, 8, 40, 640, 0.0, "no delay at all"),
    (64, 2, 2, 64, 700, 4.0, "wide delay steps between groups"),
    (64, 2, 2, 64, 700, 8.0, "steps too wide for the windows"),
    (256, 16, 56, 120, 2050, 0.2, "two DM chunks a group"),
]


def _run(tx, plan, prec, shape, monkeypatch):
    C, nsub, G, ndm, ndump, ddm, _ = plan
    if shape:
        monkeypatch.setenv("TXG_DEDISP_SHAPE", shape)
    else:
        monkeypatch.delenv("TXG_DEDISP_SHAPE", raising=False)
    f = 1500.0 - 0.5 * 600 / C * np.arange(C)
    row = tx.SinglePulse(td=1, fd=1, dms=3.0 if ddm else 0.0, ddm=ddm, ndm=ndm, maxw=0.01, nsub=nsub, dm_group=G, thre=7.0)
    rng = np.random.default_rng(C + ndm)
    out = []
    with tx.Search([row], C, 1e-3, f, ndump, precision=prec, flags=tx.FLAG_KEEP_SERIES, zapthre=0.0) as s:
        n = int(s.row_info(0).offset // ndump) + 3
        for b in range(n):
            s.push_block(rng.integers(90, 160, (ndump, C)).astype(np.uint8))
            s.sync()
            if s.row_info(0).gated:
                out.append(s.timdata(0).copy())
    return out


@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("plan", PLANS, ids=[p[-1].replace(" ", "-") for p in PLANS])
def test_tensor_memory_kernels_equal_the_shared_memory_ones(tx, plan, prec, monkeypatch):
    want = _run(tx, plan, prec, "s1=18,s2=1,s2kb=18", monkeypatch)
    got = _run(tx, plan, prec, "", monkeypatch)
    assert len(want) == len(got) >= 2
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
