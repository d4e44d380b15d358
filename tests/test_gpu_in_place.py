"""x and g in one buffer: every path evaluates at the buffer's contents and leaves the
gradient in it, with the bits of a call on two buffers."""
import pytest

from ccmpred_b200 import Evaluator, synth


@pytest.mark.gpu
@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "tc_bf16x3", "simt_f32",
                                  "simt_f64"])
@pytest.mark.parametrize("L,N,gradient,shift", [
    (1, 5, "tied", 0), (12, 300, "tied", 0), (13, 257, "partial", 0), (61, 513, "tied", 1),
    (64, 700, "partial", 0), (12, 9999, "tied", 0),  # (the last one's backward tile is cut)
])
def test_gradient_over_its_point(gpu, path, L, N, gradient, shift):
    import torch
    msa = synth.generate(synth.MSAConfig("in", L, N, n_pairs=L // 8, dup_frac=0.2, seed=500 + L))
    dtype = torch.float64 if path == "simt_f64" else torch.float32
    x = torch.from_numpy(synth.random_x(L, 600 + L)).to("cuda", dtype)
    g = torch.empty_like(x)
    if path == "tc_i8x3":
        shift = 0
    one = torch.empty(x.numel() + shift, dtype=dtype, device="cuda")[shift:]
    with Evaluator(msa, lambda_pair=0.2 * L, gradient=gradient, path=path) as ev:
        f = ev.evaluate(x, g)
        for _ in range(2):
            one.copy_(x)
            assert ev.evaluate(one, one) == f
            assert torch.equal(one, g)
        assert ev.evaluate(x, one) == f and torch.equal(one, g)  # and on two again
