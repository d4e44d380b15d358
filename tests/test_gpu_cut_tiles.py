"""The sparse path's backward with tiles of its last wave cut along the rows: gradient
and f are those of the uncut schedule, bit for bit.  One CTA pair (two SMs) never cuts,
since every tile is then a wave of its own."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth


@pytest.mark.gpu
@pytest.mark.parametrize("L,N,gradient,max_sms", [
    (12, 2500, "tied", 0),       # one tile, three parts
    (12, 9999, "tied", 0),       # one tile, eight parts, rows not a multiple of a K block
    (12, 6000, "partial", 0),
    (12, 32768, "tied", 0),      # the most rows that are cut
    (12, 32800, "tied", 0),      # past them: the K chunks of an uncut tile
    (60, 4001, "tied", 28),      # fifteen tiles on fourteen pairs: one wave and one cut tile
    (60, 6000, "partial", 44),   # 25 tiles on 22 pairs
])
def test_cut_tiles_are_bit_identical(gpu, L, N, gradient, max_sms):
    import torch
    msa = synth.generate(synth.MSAConfig("cut", L, N, n_pairs=L // 8, dup_frac=0.2, seed=300 + L))
    w = np.random.default_rng(7).uniform(0.05, 1, N).astype(np.float32)
    x = torch.from_numpy(synth.random_x(L, 400 + L)).cuda()
    got = []
    for sms in (2, max_sms):
        with Evaluator(msa, weights=w, lambda_pair=0.2 * (L - 1), gradient=gradient,
                       max_sms=sms) as ev:
            g = torch.full((nvar_padded(L),), float("nan"), device="cuda")
            for _ in range(3):
                f = ev.evaluate(x, g)
                got.append((f, g.cpu().numpy().copy()))
    for f, g in got[1:]:
        assert f == got[0][0] and np.array_equal(g, got[0][1])


@pytest.mark.gpu
def test_memory_cap_goes_without(gpu):
    """A context with a memory cap keeps to the uncut schedule, with the same bits."""
    import torch
    L, N = 12, 9999
    msa = synth.generate(synth.MSAConfig("cap", L, N, n_pairs=1, dup_frac=0.2, seed=13))
    x = torch.from_numpy(synth.random_x(L, 14)).cuda()
    got = []
    for limit in (0, 40 << 20):  # the eight parts' sums and the operands do not both fit
        with Evaluator(msa, mem_limit=limit) as ev:
            g = torch.empty(nvar_padded(L), device="cuda")
            got.append((ev.evaluate(x, g), g.cpu().numpy()))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
