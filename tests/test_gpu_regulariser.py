"""The regulariser is an FP64 sum of FP64 squares at every width, whether 4 divides it or
not: exact products, some 1e5 additions of 1e-16 each and a difference of two sums of its
own size; and it does not overflow where a float square would."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nsingle_padded, synth


@pytest.mark.gpu
@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "tc_bf16x3", "simt_f32"])
@pytest.mark.parametrize("L", [12, 13])
@pytest.mark.parametrize("large", [0.0, 3e19])
def test_regulariser(gpu, path, L, large):
    import torch
    msa = synth.generate(synth.MSAConfig("reg", L, 60, seed=50))
    x = synth.random_x(L, 51) * np.float32(30)
    nsp = nsingle_padded(L)
    if large:
        x[nsp + 5 * 32 * L * L + 3] = large
    lam1, lam2 = np.float32(0.01), np.float32(0.2) * np.float32(L - 1)
    d = x.astype(np.float64)
    exact = float(lam1) * np.sum(d[:nsp] ** 2) + 0.5 * float(lam2) * np.sum(d[nsp:] ** 2)
    xd = torch.from_numpy(x).cuda()
    with Evaluator(msa, path=path) as ev:
        f = ev.evaluate(xd, torch.empty_like(xd))
        reg = ev.result().reg
    assert np.isfinite(f)
    assert abs(reg - exact) <= 1e-10 * max(abs(f), exact)
