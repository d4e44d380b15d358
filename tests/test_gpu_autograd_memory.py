"""The autograd wrapper's backward allocates the gradients that are asked for only."""
import pytest

from ccmpred_b200 import Evaluator, synth


@pytest.mark.gpu
@pytest.mark.parametrize("need_w", [False, True])
def test_partial_needs(gpu, need_w):
    import torch
    from ccmpred_b200 import autograd
    L = 60
    w_bytes = 4 * (21 * L) ** 2
    ev = Evaluator(synth.generate(synth.MSAConfig("am", L, 40, seed=60)), gradient="partial")
    V = torch.randn(L, 20, device="cuda").mul_(0.1).requires_grad_()
    W = torch.randn(L, L, 21, 21, device="cuda").mul_(0.01).requires_grad_(need_w)
    for _ in range(2):
        V.grad = W.grad = None
        f = autograd.pseudo_likelihood(V, W, ev)
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        f.backward()
        grown = torch.cuda.max_memory_allocated() - before
        assert (grown >= w_bytes) == need_w
    assert (W.grad is None) != need_w and torch.isfinite(V.grad).all()
    ev.close()
