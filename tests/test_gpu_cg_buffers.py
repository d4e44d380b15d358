"""The whole solve with buffers chosen on the device (the sparse path without a progress
callback) equals the per-iteration graphs bit for bit where its vector passes have edges:
odd widths, an x that is only 4-byte aligned, nonzero padding (every element visited),
and solves that end at once or after one trial."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nsingle_padded, nvar_padded, synth
from ccmpred_b200.host import init_bias

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,N", [(1, 20), (5, 64), (32, 257), (43, 600)])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("padding", [0.0, 1e-3])
@pytest.mark.parametrize("iterations", [0, 1, 9])
def test_whole_solve_equals_iterations(gpu, L, N, shift, padding, iterations):
    import torch
    msa = synth.generate(synth.MSAConfig("cgb", L, N, dup_frac=0.2, seed=70 + L))
    x0 = init_bias(msa)
    x0[nsingle_padded(L):].reshape(21, L, 32, L)[2, L // 2, 30, 0] = padding
    got = []
    with Evaluator(msa) as ev:
        for progress in (None, lambda *a: False):
            buf = torch.zeros(nvar_padded(L) + 4, device="cuda")
            x = buf[shift:shift + nvar_padded(L)]
            x.copy_(torch.from_numpy(x0))
            r = ev.minimize(x, max_iterations=iterations, epsilon=0.0, progress=progress)
            got.append((r.status, r.iterations, r.evaluations, r.fx, r.gnorm, x.cpu().numpy()))
    assert got[0][:5] == got[1][:5]
    assert np.array_equal(got[0][5].view(np.uint32), got[1][5].view(np.uint32))
