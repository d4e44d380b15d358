"""Saved-tensor hooks around the autograd wrapper: the gradient that it keeps may come
back in other memory, with other strides or in another type."""
import pytest

from ccmpred_b200 import Evaluator, synth


def strided(t):
    import torch
    return torch.stack([t, t.new_full(t.shape, float("nan"))], 1)[:, 0]


HOOKS = {
    "cpu": (lambda t: t.cpu(), lambda t: t.cuda()),
    "strided": (strided, lambda t: t),
    "double": (lambda t: t.double(), lambda t: t),
    "shifted": (lambda t: t.new_empty(t.numel() + 1)[1:].copy_(t), lambda t: t),
}


@pytest.mark.gpu
@pytest.mark.parametrize("hook", list(HOOKS))
def test_saved_tensor_hooks(gpu, hook):
    import torch
    from ccmpred_b200 import autograd
    L = 9
    ev = Evaluator(synth.generate(synth.MSAConfig("ah", L, 30, seed=80)), gradient="partial")
    V = (torch.randn(L, 20, device="cuda") * 0.1).requires_grad_()
    W = (torch.randn(L, L, 21, 21, device="cuda") * 0.01).requires_grad_()
    plain = torch.autograd.grad(autograd.pseudo_likelihood(V, W, ev), (V, W))
    with torch.autograd.graph.saved_tensors_hooks(*HOOKS[hook]):
        f = autograd.pseudo_likelihood(V, W, ev)
    for a, b in zip(plain, torch.autograd.grad(f, (V, W))):
        assert torch.equal(a, b.to(a.dtype))
    ev.close()
