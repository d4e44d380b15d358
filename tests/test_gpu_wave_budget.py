"""The waves of a batch count memory that the library's pool keeps mapped, but nobody
uses, as free: earlier calls do not make the waves smaller."""
import ctypes

import pytest

from ccmpred_b200 import Evaluator, _lib, lib, synth


@pytest.mark.gpu
def test_kept_memory_counts_as_free(gpu):
    def driver_free():
        free = ctypes.c_size_t()
        assert lib().ccm_device_info(0, None, 0, ctypes.byref(free), None) == _lib.CCM_OK
        return free.value

    msa = synth.generate(synth.MSAConfig("wb", 300, 20000, seed=3))
    assert lib().ccm_release_memory(0) == _lib.CCM_OK
    free, budget = driver_free(), lib().ccm_debug_wave_budget(0)
    assert abs(budget - 0.6 * free) < 128 << 20
    with Evaluator(msa):
        # (what a context holds is taken)
        assert lib().ccm_debug_wave_budget(0) < budget - (256 << 20)
    assert driver_free() < free - (256 << 20)  # kept
    assert abs(lib().ccm_debug_wave_budget(0) - budget) < 64 << 20
    assert lib().ccm_release_memory(0) == _lib.CCM_OK
