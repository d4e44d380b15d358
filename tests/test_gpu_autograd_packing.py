"""The packing kernels of the autograd wrapper against its torch operations (pack,
unpack): every stride order of V and W, both types, partial needs, a scaled and a
second-order backward, batched gradients; bit for bit, being copies (and one product)."""
import itertools

import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth

pytestmark = pytest.mark.gpu


def general(V, W, ev):
    from ccmpred_b200 import autograd
    return autograd.PseudoLikelihoodFunction.apply(autograd.pack(V, W), ev)


@pytest.mark.parametrize("path", ["tc_i8sp", "simt_f64"])
@pytest.mark.parametrize("L", [1, 7, 8, 16, 17, 40])
def test_forms_of_the_parameters(gpu, path, L):
    import torch
    from ccmpred_b200 import autograd
    dtype = torch.float64 if path == "simt_f64" else torch.float32
    ev = Evaluator(synth.generate(synth.MSAConfig("pk", L, 30, seed=L)), path=path, gradient="partial",
                   lambda_pair=0.4)
    gen = torch.Generator(device="cuda").manual_seed(L)
    big = torch.randn(L, L, 21, 42, generator=gen, device="cuda", dtype=dtype) * 0.05
    base = big[..., ::2]
    forms = [base.permute(p).contiguous().permute([p.index(i) for i in range(4)])
             for p in itertools.permutations(range(4))]
    forms += [base, big[..., 21:], base.new_zeros(1, 1, 21, 21).expand(L, L, 21, 21)]
    V0 = torch.randn(20, L, generator=gen, device="cuda", dtype=dtype) * 0.1
    for n, W0 in enumerate(forms):
        V0n = V0.T if n % 2 else V0.T.contiguous()
        got = []
        for call in (general, autograd.pseudo_likelihood):
            V, W = V0n.detach().requires_grad_(n % 3 != 1), W0.detach().requires_grad_(n % 3 != 2)
            f = call(V, W, ev)
            (f * 3.0).backward()
            got.append((f.detach(), V.grad, W.grad))
        for a, b in zip(*got):
            assert (a is None) == (b is None)
            assert a is None or torch.equal(a, b)
    x = torch.full((nvar_padded(L),), float("nan"), device="cuda", dtype=dtype)
    from ccmpred_b200._lib import check, lib
    check(lib().ccm_pack_parameters(V0.T.data_ptr(), autograd._strides(V0.T), base.data_ptr(),
                                    autograd._strides(base), L, x.element_size(), x.data_ptr(), None))
    assert torch.equal(x, autograd.pack(V0.T, base))
    ev.close()


def test_other_ways_through_backward(gpu):
    import torch
    from ccmpred_b200 import autograd
    L = 9
    ev = Evaluator(synth.generate(synth.MSAConfig("pk", L, 30, seed=3)), gradient="partial")
    V = (torch.randn(L, 20, device="cuda") * 0.1).requires_grad_()
    W = (torch.randn(L, L, 21, 21, device="cuda") * 0.01).requires_grad_()
    s = torch.tensor(2.0, device="cuda", requires_grad=True)
    second, batched = [], []
    for call in (general, autograd.pseudo_likelihood):
        f = call(V, W, ev)
        dV, dW = torch.autograd.grad(f * s, (V, W), create_graph=True)
        second.append(torch.autograd.grad(dV.sum() + dW.square().sum(), s)[0])
        f = call(V, W, ev)
        batched.append(torch.autograd.grad(f, (V, W), torch.tensor([1.0, -2.0], device="cuda"),
                                           is_grads_batched=True))
    assert torch.equal(*second)
    assert all(torch.equal(a, b) for a, b in zip(*batched))
    # what the kernels do not take goes the general way, with its errors
    with pytest.raises(AssertionError):
        autograd.pseudo_likelihood(V.cpu(), W.cpu(), ev)
    with pytest.raises(ValueError):
        autograd.pseudo_likelihood(V, W, Evaluator(ev.msa))
    ev.close()
