"""Calls on torch tensors under a side stream, and evaluators on a caller's non-blocking
stream: they wait for what torch's current stream still has to do to their inputs."""
import pytest

from ccmpred_b200 import Evaluator, synth

pytestmark = pytest.mark.gpu
L, N = 40, 400
SLOW = 20_000_000  # clock cycles, some 10 ms


def alignment():
    return synth.generate(synth.MSAConfig("st", L, N, n_pairs=4, dup_frac=0.2, seed=900))


# (torch's stream, the evaluator's): "side" is a torch stream (non-blocking), None the default
@pytest.mark.parametrize("current,own", [(None, None), ("side", None), (None, "side"),
                                         ("side", "side"), ("side", "same")])
@pytest.mark.parametrize("path", ["tc_i8sp", "simt_f32"])
def test_late_inputs(gpu, current, own, path):
    import torch
    from ccmpred_b200 import autograd
    x = torch.from_numpy(synth.random_x(L, 901)).cuda()
    V, W = (t.clone() for t in autograd.unpack(x, L))
    with Evaluator(alignment(), path=path, gradient="partial") as ev:
        g = torch.empty_like(x)
        f = ev.evaluate(x, g)
        grads = autograd.unpack(g, L)
    with Evaluator(alignment(), path=path) as ev:
        solved = x.clone()
        r = ev.minimize(solved, max_iterations=2, epsilon=0.0)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    where = torch.cuda.default_stream() if current is None else side
    handle = {None: None, "side": other.cuda_stream, "same": side.cuda_stream}[own]
    torch.cuda.synchronize()
    with torch.cuda.stream(where):
        def late(t):
            out = torch.zeros_like(t)
            torch.cuda._sleep(SLOW)
            out.copy_(t)
            return out
        with Evaluator(alignment(), path=path, gradient="partial", stream=handle) as ev:
            g2 = torch.empty_like(x)
            assert ev.evaluate(late(x), g2) == f and torch.equal(g2, g)
            v, w = late(V).requires_grad_(), late(W).requires_grad_()
            torch.cuda._sleep(SLOW)
            out = autograd.pseudo_likelihood(v, w, ev)
            out.backward()
            assert abs(out.item() - f) <= 1e-6 * abs(f)
            assert torch.equal(v.grad, grads[0]) and torch.equal(w.grad, grads[1])
            xs = late(x).requires_grad_()
            autograd.PseudoLikelihoodFunction.apply(xs, ev).backward()
            assert torch.equal(xs.grad, g)
        with Evaluator(alignment(), path=path, stream=handle) as ev:
            y = late(x)
            assert ev.minimize(y, max_iterations=2, epsilon=0.0).fx == r.fx
            assert torch.equal(y, solved)
    torch.cuda.synchronize()
