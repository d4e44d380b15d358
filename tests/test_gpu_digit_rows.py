"""The digits of W on both sides of the rule that takes four rows a step instead of
eight (L <= 89), against the FP64 oracle."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 9, 63, 72, 73, 89, 90, 112, 113])
def test_digit_rows(gpu, oracle_mod, L):
    import torch
    msa = synth.generate(synth.MSAConfig("rows", L, 40, n_pairs=L // 8, dup_frac=0.2, seed=700 + L))
    w = oracle_mod.oracle_weights(msa, 0.8)
    lam2 = 0.2 * (L - 1)
    x = synth.random_x(L, 800 + L)
    f64, g64 = oracle_mod.oracle_evaluate(msa, w, 0.01, lam2, x)
    with Evaluator(msa, weights=w, lambda_pair=lam2) as ev:
        g = torch.empty(nvar_padded(L), device="cuda")
        f = ev.evaluate(torch.from_numpy(x).cuda(), g)
        assert abs(f - f64) < 1e-6 * abs(f64)
        assert np.linalg.norm(g.cpu().numpy() - g64) < 1e-5 * np.linalg.norm(g64)
