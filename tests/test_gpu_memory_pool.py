"""The library's memory pool: evaluations, solves and sequence weights from several host
threads at once, with the pool's unused memory given back in between, equal those of one
thread bit for bit."""
import threading

import numpy as np
import pytest

from ccmpred_b200 import Evaluator, _lib, calculate_weights, lib, synth

pytestmark = pytest.mark.gpu


def work(L, N, seed):
    import torch
    msa = synth.generate(synth.MSAConfig("pool", L, N, dup_frac=0.3, seed=seed))
    w = calculate_weights(msa, 0.8)
    with Evaluator(msa, weights=w) as ev:
        x = torch.from_numpy(synth.random_x(L, seed + 1)).cuda()
        g = torch.empty_like(x)
        f = ev.evaluate(x, g)
        r = ev.minimize(x, max_iterations=3, epsilon=0.0)
        return f, r.fx, w, g.cpu().numpy(), x.cpu().numpy()


@pytest.mark.parametrize("threads", [1, 4])
def test_threads_share_the_pool(gpu, threads):
    sizes = [(20, 300, 1), (45, 700, 2), (64, 257, 3), (31, 1500, 4)]
    alone = [work(*s) for s in sizes]
    assert lib().ccm_release_memory(0) == _lib.CCM_OK
    got = [None] * len(sizes)

    def run(k):
        for i in range(k, len(sizes), threads):
            for _ in range(2):
                got[i] = work(*sizes[i])
                assert lib().ccm_release_memory(0) == _lib.CCM_OK

    pool = [threading.Thread(target=run, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    for a, b in zip(alone, got):
        assert a[:2] == b[:2]
        assert all(np.array_equal(u.view(np.uint32), v.view(np.uint32)) for u, v in zip(a[2:], b[2:]))


def test_release_rejects_a_bad_device(gpu):
    assert lib().ccm_release_memory(-1) == _lib.CCM_ERR_INVALID
    assert lib().ccm_release_memory(64) == _lib.CCM_ERR_INVALID
