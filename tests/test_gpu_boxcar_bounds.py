"""The search that skips widths by upper bounds (points only, threshold 4 or more) against the
tracked search over every width (dense output): the same arithmetic decides both, so the points
are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, rng):
    x = rng.normal(0, 20, (10, n)).astype(np.float32)
    x[1, n // 3:n // 3 + 5] += 200            # a narrow pulse
    x[2, n // 4:n // 4 + max(1, n // 6)] += 30  # a wide one
    x[3] = np.cumsum(x[3]) * 0.2              # red noise: no bound holds for long
    x[4] = 3.0                                # no variance
    x[5, :1] += 400                           # at the row's ends
    x[5, -1:] += 400
    x[6] = 0.0
    x[6, ::7] = 60.0                          # equal scores
    x[7, n // 2] = np.inf                     # only the IQR statistics stay finite
    x[8, n - 1 - n // 5] = np.nan
    x[9, n // 2:] *= 30                       # most of the power in one half
    return x


# sizes: one block and its edges, chunks that start in the same bank (512 k), a row whose bounds do
# not fit beside it (51000), segmented rows, and a segment of so many samples that the
# statistics' pieces get smaller (250000)
@pytest.mark.parametrize("n", [1, 2, 31, 64, 127, 128, 129, 257, 512, 1537, 8192, 13156, 40000, 51000, 62496, 250000])
@pytest.mark.parametrize("iqr", [False, True])
def test_bounded_search_gives_the_tracked_searchs_points(tx, n, iqr):
    x = _rows(n, np.random.default_rng(n))
    widths = np.unique(np.concatenate([tx.width_ladder(1e-4, 0.05, 0.1, 1e-4), [127, 128, 129, 130, min(n, 900), min(n + 3, 901)]]))
    widths = np.concatenate([widths, np.arange(1, 41, 3)])  # more than a warp's, and not in order
    for thre in (4.0, 7.0):
        _, _, want = tx.boxcar(x, widths, iqr=iqr, thre=thre, dense=True, cand_capacity=1 << 22)
        _, _, got = tx.boxcar(x, widths, iqr=iqr, thre=thre, dense=False, cand_capacity=1 << 22)
        np.testing.assert_array_equal(got, want)
