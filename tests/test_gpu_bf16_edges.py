"""The split-bf16 paths at the edges of their 12-column groups and 256-row tiles, and
with vectors that are only 4-byte aligned, against the FP64 oracle (bounds as in
test_gpu_parity: 1e-6 in f, 1e-5 of the whole gradient)."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["tc_bf16x2", "tc_bf16x3"])
@pytest.mark.parametrize("L,N", [(1, 5), (11, 256), (12, 257), (13, 40), (24, 511), (61, 300)])
def test_edges(gpu, oracle_mod, path, L, N):
    import torch
    msa = synth.generate(synth.MSAConfig("bf", L, N, n_pairs=L // 8, dup_frac=0.2, seed=300 + L))
    w = oracle_mod.oracle_weights(msa, 0.8)
    lam2 = 0.2 * max(L - 1, 1)
    x = synth.random_x(L, 400 + L)
    f64, g64 = oracle_mod.oracle_evaluate(msa, w, 0.01, lam2, x)
    n = nvar_padded(L)
    with Evaluator(msa, weights=w, lambda_pair=lam2, path=path) as ev:
        bufs = torch.zeros(2, n + 4, device="cuda")
        for shift in (0, 1):
            xd, gd = bufs[0, shift:shift + n], bufs[1, shift:shift + n]
            xd.copy_(torch.from_numpy(x))
            gd.fill_(float("nan"))
            f = ev.evaluate(xd, gd)
            assert abs(f - f64) < 1e-6 * abs(f64)
            assert np.linalg.norm(gd.cpu().numpy() - g64) < 1e-5 * np.linalg.norm(g64)
