"""x and g that are only 4-byte aligned: the gradient has the bits of an aligned call, f
differs by the order of the regulariser's sum at most (FP64 sums of float squares)."""
import pytest

from ccmpred_b200 import Evaluator, synth

pytestmark = pytest.mark.gpu


def shifted(t, by):
    import torch
    buf = torch.full((t.numel() + 8,), float("nan"), dtype=t.dtype, device=t.device)
    view = buf[by:by + t.numel()]
    view.copy_(t)
    return buf, view


@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "simt_f32"])
@pytest.mark.parametrize("L,N", [(12, 257), (61, 300), (64, 700)])
def test_evaluate(gpu, path, L, N):
    import torch
    msa = synth.generate(synth.MSAConfig("al", L, N, n_pairs=L // 8, dup_frac=0.2, seed=700 + L))
    x = torch.from_numpy(synth.random_x(L, 800 + L)).cuda()
    g = torch.empty_like(x)
    with Evaluator(msa, path=path) as ev:
        f = ev.evaluate(x, g)
        for dx, dg in [(1, 0), (0, 1), (3, 2), (2, 4)]:
            (_, xs), (whole, gs) = shifted(x, dx), shifted(g, dg)
            assert abs(ev.evaluate(xs, gs) - f) <= 1e-6 * abs(f)
            assert torch.equal(gs, g)
            assert torch.isnan(whole[:dg]).all() and torch.isnan(whole[dg + g.numel():]).all()
