"""Sequence weights at thresholds and row counts past what an int, or a grid, holds."""
import ctypes

import numpy as np
import pytest

from ccmpred_b200 import CcmError, _lib, calculate_weights, lib, synth

pytestmark = pytest.mark.gpu


def identity_limit(threshold, L):
    """(int)ceil of the float product, as x86-64 converts what an int does not hold."""
    p = np.ceil(np.float64(np.float32(threshold) * np.float32(L)))
    return int(p) if abs(p) < 2 ** 31 else -2 ** 31


@pytest.mark.parametrize("threshold", [float("nan"), float("inf"), -float("inf"), 1e30, -1e30,
                                       4e8, -4e8, 2e8, -2e8, -0.01, 0.0, 1.0, 1.01])
def test_thresholds(gpu, threshold):
    import torch
    L, N = 10, 150
    msa = synth.generate(synth.MSAConfig("lim", L, N, dup_frac=0.3, seed=1))
    ids = (msa[:, None] == msa[None]).sum(2)
    with np.errstate(all="ignore"):
        over = ids > identity_limit(threshold, L)
        expect = np.float32(1.0 / np.float64(over.sum(1) + np.diag(over) - 1.0))
    assert np.array_equal(calculate_weights(msa, threshold), expect)
    d_msa = torch.from_numpy(msa).cuda()
    d_w = torch.empty(N, device="cuda")
    assert lib().ccm_calculate_weights_noalloc(d_msa.data_ptr(), L, N, ctypes.c_float(threshold),
                                               d_w.data_ptr(), None) == _lib.CCM_OK
    torch.cuda.synchronize()
    assert np.array_equal(d_w.cpu().numpy(), expect)


@pytest.mark.parametrize("N", [64 * 65535 + 1, 64 * 92682])
def test_more_tiles_than_a_grid_holds(gpu, N):
    """65536 blocks of rows have more tiles of pairs than a grid has blocks; those of 92682
    are 2^32 + 55607, which as an unsigned number would pass for a few."""
    with pytest.raises(CcmError) as err:
        calculate_weights(np.zeros((N, 1), np.uint8))
    assert err.value.code == _lib.CCM_ERR_CUDA
    msa = synth.generate(synth.MSAConfig("lim", 10, 70, seed=2))
    assert np.isfinite(calculate_weights(msa)).all()  # nothing of it is left behind
