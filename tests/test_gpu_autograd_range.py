"""An f beyond float's range is an infinite loss, not an error, and has its gradient."""
import pytest

from ccmpred_b200 import Evaluator, synth


@pytest.mark.gpu
@pytest.mark.parametrize("value", [1e21, -1e21, float("inf"), float("nan")])
def test_loss_beyond_float(gpu, value):
    import torch
    from ccmpred_b200 import autograd
    L = 9
    ev = Evaluator(synth.generate(synth.MSAConfig("ar", L, 30, seed=70)), gradient="partial")
    V = torch.randn(L, 20, device="cuda") * 0.1
    W = (torch.randn(L, L, 21, 21, device="cuda") * 0.01).requires_grad_()
    V[3, 4] = value
    V.requires_grad_()
    got = []
    for call in (lambda: autograd.PseudoLikelihoodFunction.apply(autograd.pack(V, W), ev),
                 lambda: autograd.pseudo_likelihood(V, W, ev)):
        f = call()
        got.append((f.detach(), *torch.autograd.grad(f, (V, W))))
    assert not torch.isfinite(got[0][0])
    for a, b in zip(*got):
        assert torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))
    ev.close()
