"""The backward's epilogue is made to wait 1000 clock cycles on a barrier that nothing
arrives on.  It records the timeout in the device's record and, by itself, in the one
that a waiting host reads (f may be in it already), and returns; with the knob cleared
the same context evaluates with the bits of a fresh one.  Every tile has a CTA pair of
its own here."""
import ctypes

import pytest

from ccmpred_b200 import CcmError, Evaluator, _lib, lib, synth

BACKWARD = 2  # bit of the record's status


@pytest.mark.gpu
@pytest.mark.parametrize("path,L,N,gradient", [
    ("tc_i8sp", 60, 800, "tied"), ("tc_i8sp", 60, 800, "partial"),
    ("tc_i8sp", 12, 2500, "tied"),  # one tile, cut in three parts
    ("tc_i8x3", 60, 800, "tied"),
])
def test_backward_wait_runs_out(gpu, path, L, N, gradient):
    import torch
    msa = synth.generate(synth.MSAConfig("bw", L, N, n_pairs=L // 15, seed=20))
    x = torch.from_numpy(synth.random_x(L, 21)).cuda()
    ref, g = torch.empty_like(x), torch.empty_like(x)
    with Evaluator(msa, path=path, gradient=gradient) as ev:
        f = ev.evaluate(x, ref)
    with Evaluator(msa, path=path, gradient=gradient) as ev:
        for _ in range(2):
            assert lib().ccm_debug_set_backward_wait_limit(ev.handle, 1000) == _lib.CCM_OK
            with pytest.raises(CcmError) as err:
                ev.evaluate(x, g)
            assert err.value.code == _lib.CCM_ERR_DEVICE and "timed out" in str(err.value)
            ev.evaluate_async(x, g)
            assert ev.result().status == BACKWARD
            host = x.cpu().numpy()
            with pytest.raises(CcmError) as err:
                ev.evaluate(host, host.copy())
            assert err.value.code == _lib.CCM_ERR_DEVICE
            if gradient == "tied":
                r = _lib.CcmCgResult()
                p = _lib.CcmCgParams()
                lib().ccm_cg_params_default(ctypes.byref(p))
                rc = lib().ccm_conjugrad_gpu(ev.handle, g.copy_(x).data_ptr(), x.numel(),
                                             ctypes.byref(p), _lib.PROGRESS(0), None, ctypes.byref(r))
                assert rc == _lib.CCM_ERR_DEVICE
            assert lib().ccm_debug_set_backward_wait_limit(ev.handle, 0) == _lib.CCM_OK
            assert ev.evaluate(x, g) == f and torch.equal(g, ref)
        assert lib().ccm_debug_set_backward_wait_limit(ev.handle, -1) == _lib.CCM_ERR_INVALID
    torch.cuda.synchronize()
