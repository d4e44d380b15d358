"""x and g that are only 4-byte aligned: the gradient has the bits of an aligned call, f
differs by the order of the regulariser's sum at most (FP64 sums of float squares); a
solve from such an x takes the same steps to FP64 rounding of its scalars."""
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


@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "simt_f32"])
@pytest.mark.parametrize("progress", [None, lambda *a: False])
def test_minimize(gpu, path, progress):
    import torch
    L, N = 24, 300
    msa = synth.generate(synth.MSAConfig("al", L, N, n_pairs=3, dup_frac=0.2, seed=724))
    x = torch.from_numpy(synth.random_x(L, 824)).cuda()
    with Evaluator(msa, path=path) as ev:
        _, xs = shifted(x, 1)
        a = ev.minimize(x, max_iterations=3, epsilon=0.0, progress=progress)
        b = ev.minimize(xs, max_iterations=3, epsilon=0.0, progress=progress)
        assert (a.iterations, a.evaluations) == (b.iterations, b.evaluations)
        assert abs(a.fx - b.fx) <= 1e-6 * abs(a.fx)
        # three steps: float rounding of x, carried through three gradients of 1e-5
        assert torch.linalg.norm(xs - x) <= 1e-4 * torch.linalg.norm(x)


def test_libconjugrad_gpu(gpu):
    """conjugrad_gpu under libconjugrad's name, with an evaluation of its own."""
    import ctypes

    import torch
    from ccmpred_b200 import _lib, lib
    L = 12
    msa = synth.generate(synth.MSAConfig("al", L, 200, n_pairs=1, dup_frac=0.2, seed=725))
    x = torch.from_numpy(synth.random_x(L, 825)).cuda()
    got = []
    with Evaluator(msa, path="simt_f32") as ev:
        def evaluate(inst, xp, gp, n):
            fx = ctypes.c_double()
            assert lib().ccm_evaluate(ev.handle, xp, gp, n, ctypes.byref(fx)) == _lib.CCM_OK
            return fx.value
        cb = _lib.EVALUATE(evaluate)
        for by in (0, 1):
            _, xs = shifted(x, by)
            fx = ctypes.c_float()
            p = lib().conjugrad_init()
            p.contents.max_iterations, p.contents.epsilon = 3, 0.0
            torch.cuda.synchronize()
            lib().conjugrad_gpu(xs.numel(), xs.data_ptr(), ctypes.byref(fx),
                                ctypes.cast(cb, ctypes.c_void_p), None, None, p)
            got.append((fx.value, xs.clone()))
    assert abs(got[0][0] - got[1][0]) <= 1e-6 * abs(got[0][0])
    assert torch.linalg.norm(got[0][1] - got[1][1]) <= 1e-4 * torch.linalg.norm(got[0][1])
