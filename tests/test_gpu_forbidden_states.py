"""Single fields of minus infinity, which forbid a state: their probability is exactly
zero, as with -1e30, also where they are all the states that one thread of the softmax
holds; the rest of the gradient is what it is with -1e30."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, synth


@pytest.mark.gpu
@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "tc_bf16x3", "simt_f32"])
@pytest.mark.parametrize("states", [range(0, 1), range(0, 12), range(11, 20), range(0, 20)])
def test_minus_infinity_fields(gpu, path, states):
    import torch
    L, N = 30, 300
    states = list(states)
    free = [a for a in range(21) if a not in states]
    msa = synth.generate(synth.MSAConfig("forbid", L, N, n_pairs=3, dup_frac=0.2, seed=40))
    cols = [0, 8, 9, 17, 29]
    for j in cols:
        msa[:, j] = np.array(free)[msa[:, j] % len(free)]
    x = torch.from_numpy(synth.random_x(L, 41)).cuda()
    at = torch.tensor([a * L + j for a in states for j in cols], device="cuda")
    got = []
    with Evaluator(msa, path=path) as ev:
        for v in (-1e30, -float("inf")):
            x[at] = v
            g = torch.empty_like(x)
            ev.evaluate(x, g)
            g[at] = 0.0  # 2 lambda v and a zero
            got.append(g)
    assert torch.isfinite(got[0]).all()
    assert torch.equal(got[0], got[1])
