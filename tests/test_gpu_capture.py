"""Evaluations captured into a CUDA graph (plain edges between their kernels) against the
same ones in a stream (dependent launches): the same bits, replay after replay."""
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth


@pytest.mark.gpu
@pytest.mark.parametrize("path", ["tc_i8sp", "tc_i8x3", "tc_bf16x2", "tc_bf16x3"])
@pytest.mark.parametrize("L,N", [(7, 3), (50, 700)])
def test_captured_evaluations(gpu, path, L, N):
    import torch
    msa = synth.generate(synth.MSAConfig("graph", L, N, n_pairs=1, dup_frac=0.1, seed=11))
    with Evaluator(msa, path=path) as ev:
        xs = [torch.from_numpy(synth.random_x(L, 600 + i)).cuda() for i in range(2)]
        gs = [torch.empty(nvar_padded(L), device="cuda") for _ in xs]
        want = []
        for x, g in zip(xs, gs):
            f = ev.evaluate(x, g)
            want.append((f, g.clone()))
        stream = torch.cuda.ExternalStream(ev.stream)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for x, g in zip(xs, gs):
                ev.evaluate_async(x, g)
        for _ in range(3):
            for g in gs:
                g.fill_(float("nan"))
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            r = ev.result()
            assert (r.fx, r.status) == (want[-1][0], 0)
            for g, (_, w) in zip(gs, want):
                assert torch.equal(g, w)
        del graph
