"""ccm_calculate_weights on bit planes: widths around the plane words (32 columns) and
their shared-memory chunks (256), row counts around the 64-row tiles, thresholds at
both ends, duplicated rows, and states above 31 (all eight planes).  The weights are
1 / (count - 1) of integer counts: equal bit for bit."""
import numpy as np
import pytest

from ccmpred_b200 import calculate_weights

pytestmark = pytest.mark.gpu


def weights(msa, threshold):
    """src/reweighting.c:9-58: a row counts itself twice, idthres = ceil(float product)."""
    N, L = msa.shape
    idthres = int(np.ceil(np.float64(np.float32(threshold) * np.float32(L))))
    count = np.zeros(N, np.float32)
    for i in range(N):
        same = (msa == msa[i]).sum(axis=1)
        count[i] = (same > idthres).sum() + (same[i] > idthres)
    with np.errstate(divide="ignore"):
        return (1.0 / (count - np.float32(1.0)).astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("states", [21, 256])
@pytest.mark.parametrize("L,N", [(1, 2), (31, 63), (32, 64), (33, 65), (255, 130), (256, 200),
                                 (257, 129), (300, 500), (513, 77)])
def test_counts(gpu, L, N, states):
    rng = np.random.default_rng(L * 1000 + N)
    msa = rng.integers(0, states, (N, L), dtype=np.uint8)
    src = rng.integers(0, N, N // 2)
    near = msa[src]
    change = rng.random(near.shape) < rng.uniform(0.0, 0.4, (len(src), 1))
    near[change] = rng.integers(0, states, int(change.sum()), dtype=np.uint8)
    msa[: len(src)] = near
    for threshold in (0.0, 0.5, 0.62, 0.8, 0.95, 1.0):
        assert np.array_equal(calculate_weights(msa, threshold).view(np.uint32),
                              weights(msa, threshold).view(np.uint32)), threshold
