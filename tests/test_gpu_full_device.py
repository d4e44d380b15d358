"""Allocations that a full device refuses are reported by the call that made them and by
no later one."""
import numpy as np
import pytest

from ccmpred_b200 import CcmError, Evaluator, _lib, calculate_weights, release_memory, synth


@pytest.mark.gpu
def test_failed_allocation_is_not_reported_twice(gpu):
    import torch
    L, N = 400, 300
    msa = synth.generate(synth.MSAConfig("full", L, N, seed=95))
    x = synth.random_x(L, 96)
    xd = torch.from_numpy(x).cuda()
    gd, g = torch.empty_like(xd), np.empty_like(x)
    many = np.zeros((1 << 20, 400), np.uint8)  # its planes take 512 MB
    with Evaluator(msa) as ev:
        f = ev.evaluate(xd, gd)
        w = calculate_weights(msa)
        torch.cuda.synchronize()
        release_memory()
        hold = torch.empty(torch.cuda.mem_get_info(0)[0] - (384 << 20), dtype=torch.uint8, device="cuda")
        try:
            with pytest.raises(CcmError) as err:
                ev.evaluate(x, g)  # two copies of 430 MB
            assert err.value.code == _lib.CCM_ERR_NOMEM
            assert ev.evaluate(xd, gd) == f
            with pytest.raises(CcmError):
                calculate_weights(many)
            assert ev.evaluate(xd, gd) == f
            assert np.array_equal(calculate_weights(msa), w)
        finally:
            del hold
            torch.cuda.empty_cache()
        assert ev.evaluate(x, g) == f and np.array_equal(g, gd.cpu().numpy())
