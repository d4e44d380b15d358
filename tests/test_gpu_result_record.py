"""The result record of a synchronous evaluation, which the kernels write to the host
themselves: equal to the device's record on every path, also with asynchronous
evaluations of other points around it."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth


@pytest.mark.gpu
@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "tc_bf16x3", "simt_f32"])
@pytest.mark.parametrize("L,N", [(7, 3), (40, 700)])
def test_record_is_the_devices(gpu, path, L, N):
    import torch
    msa = synth.generate(synth.MSAConfig("record", L, N, n_pairs=1, dup_frac=0.1, seed=9))
    with Evaluator(msa, path=path) as ev:
        xs = [torch.from_numpy(synth.random_x(L, 500 + i)).cuda() for i in range(3)]
        g = torch.empty(nvar_padded(L), device="cuda")
        f = []
        for x in xs:
            f.append(ev.evaluate(x, g))
            r = ev.result()
            assert (r.fx, r.status) == (f[-1], 0)
        assert len(set(f)) == 3
        for i in range(6):  # sums in double, in any order
            ev.evaluate_async(xs[(i + 1) % 3], g)
            assert ev.evaluate(xs[i % 3], g) == pytest.approx(f[i % 3], rel=1e-12)
            ev.evaluate_async(xs[(i + 2) % 3], g)
        h = np.empty(nvar_padded(L), np.float32)
        assert ev.evaluate(xs[1].cpu().numpy(), h) == pytest.approx(f[1], rel=1e-12)
