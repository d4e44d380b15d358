"""Which contexts cut their backward's tiles, and what becomes of a context when one of
its allocations fails: the sums of cut tiles are done without (with the same bits),
anything else is an error that leaves nothing behind."""
import ctypes

import pytest

from ccmpred_b200 import CcmError, Evaluator, _lib, lib, release_memory, synth

pytestmark = pytest.mark.gpu


def cut(ev):
    parts = ctypes.c_int()
    return lib().ccm_debug_cut_tiles(ev.handle, ctypes.byref(parts)), parts.value


def alignment(L, N):
    return synth.generate(synth.MSAConfig("cs", L, N, n_pairs=L // 8, dup_frac=0.2, seed=30 + L))


@pytest.mark.parametrize("L,N,gradient,max_sms,expect", [
    (12, 2500, "tied", 0, (1, 3)),
    (12, 9999, "tied", 0, (1, 6)),
    (12, 6000, "partial", 0, (1, 4)),
    (12, 32768, "tied", 0, (1, 8)),    # the most rows and parts
    (12, 32800, "tied", 0, (0, 1)),
    (60, 800, "tied", 0, (0, 1)),      # too few rows
    (60, 4001, "tied", 28, (1, 4)),
    (60, 6000, "partial", 44, (3, 4)),
    (60, 6000, "partial", 2, (0, 1)),  # no tiles left over
    (60, 6000, "tied", 0, (15, 4)),
    (97, 6000, "tied", 0, (36, 2)),    # 36 tiles on 74 pairs
    (102, 6000, "tied", 0, (0, 1)),    # 45: none can be two
])
def test_schedules(gpu, L, N, gradient, max_sms, expect):
    with Evaluator(alignment(L, N), gradient=gradient, max_sms=max_sms) as ev:
        assert cut(ev) == expect
    with Evaluator(alignment(L, N), gradient=gradient, max_sms=max_sms, mem_limit=1 << 32) as ev:
        assert cut(ev) == (0, 1)


def test_allocations_that_fail(gpu):
    import torch
    L, N = 12, 9999
    msa = alignment(L, N)
    x = torch.from_numpy(synth.random_x(L, 31)).cuda()
    g, ref = torch.empty_like(x), torch.empty_like(x)
    with Evaluator(msa) as ev:
        f = ev.evaluate(x, ref)
        # (the first of a process also load their kernels, the solve's and torch's)
        ev.minimize(x.clone(), max_iterations=1)
        assert torch.equal(ref, ref.clone())
    torch.cuda.synchronize()
    release_memory()
    free = torch.cuda.mem_get_info(0)[0]
    uncut = failed = 0
    for nth in range(1, 100):
        lib().ccm_debug_fail_allocation(nth)
        try:
            ev = Evaluator(msa)
        except CcmError as err:
            assert err.code == _lib.CCM_ERR_NOMEM
            failed += 1
            continue
        finally:
            left = lib().ccm_debug_fail_allocation(0)
        with ev:
            uncut += cut(ev) == (0, 1)
            assert ev.evaluate(x, g) == f and torch.equal(g, ref)
        if left:
            break
    assert left and failed > 10 and uncut == 1
    with Evaluator(msa) as ev:
        for nth in range(1, 7):  # the optimizer's vectors and records
            y = x.clone()
            lib().ccm_debug_fail_allocation(nth)
            with pytest.raises(CcmError) as err:
                ev.minimize(y, max_iterations=1)
            assert lib().ccm_debug_fail_allocation(0) == 0
            assert err.value.code == _lib.CCM_ERR_NOMEM
            assert ev.evaluate(x, g) == f and torch.equal(g, ref)
        assert ev.minimize(x.clone(), max_iterations=1, epsilon=0.0).iterations == 1
    torch.cuda.synchronize()
    release_memory()
    assert torch.cuda.mem_get_info(0)[0] >= free - (8 << 20)
