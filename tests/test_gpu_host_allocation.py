"""A host-pointer evaluation whose device copy of x, or of g, cannot be allocated is an
error, and the next call on the context is whole again."""
import numpy as np
import pytest

from ccmpred_b200 import CcmError, Evaluator, _lib, lib, synth


@pytest.mark.gpu
@pytest.mark.parametrize("nth", [1, 2])
def test_failed_copies(gpu, nth):
    L, N = 20, 200
    msa = synth.generate(synth.MSAConfig("ha", L, N, seed=90))
    x = synth.random_x(L, 91)
    g, ref = np.empty_like(x), np.empty_like(x)
    with Evaluator(msa) as ev:
        f = ev.evaluate(x, ref)
    with Evaluator(msa) as ev:
        for n in ([nth, 1] if nth == 2 else [nth, 2, 1]):
            lib().ccm_debug_fail_allocation(n)
            with pytest.raises(CcmError) as err:
                ev.evaluate(x, g)
            assert lib().ccm_debug_fail_allocation(0) == 0
            assert err.value.code == _lib.CCM_ERR_NOMEM
        for _ in range(2):
            g.fill(np.nan)
            assert ev.evaluate(x, g) == f and np.array_equal(g, ref)
