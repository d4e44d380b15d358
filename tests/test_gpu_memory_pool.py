"""The library's memory pool: evaluations, solves and sequence weights from several host
threads at once, with the pool's unused memory given back in between, equal those of one
thread bit for bit."""
import threading

import numpy as np
import pytest

from ccmpred_b200 import Evaluator, _lib, calculate_weights, lib, synth

pytestmark = pytest.mark.gpu


def buffers(L, seed):
    import torch
    x = torch.from_numpy(synth.random_x(L, seed + 1)).cuda()
    return x, torch.empty_like(x)


def work(L, N, seed, x, g):
    """(Only calls of the library: an operation on the legacy stream, as torch's own are,
    is refused while another thread's solve captures its graph.)"""
    msa = synth.generate(synth.MSAConfig("pool", L, N, dup_frac=0.3, seed=seed))
    w = calculate_weights(msa, 0.8)
    with Evaluator(msa, weights=w) as ev:
        f = ev.evaluate(x, g)
        r = ev.minimize(x, max_iterations=3, epsilon=0.0)
        return f, r.fx, w


@pytest.mark.parametrize("threads", [1, 4])
def test_threads_share_the_pool(gpu, threads):
    import torch
    sizes = [(20, 300, 1), (45, 700, 2), (64, 257, 3), (31, 1500, 4)]
    alone, first = [], []
    for L, N, seed in sizes:
        x, g = buffers(L, seed)
        alone.append(work(L, N, seed, x, g))
        first.append((x, g))
    assert lib().ccm_release_memory(0) == _lib.CCM_OK
    got = [[None, None] for _ in sizes]
    own = [[buffers(L, seed) for _ in range(2)] for L, _, seed in sizes]
    torch.cuda.synchronize()

    def run(k):
        for i in range(k, len(sizes), threads):
            for rep in range(2):
                got[i][rep] = work(*sizes[i], *own[i][rep])
                assert lib().ccm_release_memory(0) == _lib.CCM_OK

    pool = [threading.Thread(target=run, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    torch.cuda.synchronize()
    for a, vectors, both, mine in zip(alone, first, got, own):
        for b, vecs in zip(both, mine):
            assert a[:2] == b[:2] and np.array_equal(a[2], b[2])
            for u, v in zip(vectors, vecs):
                assert torch.equal(u.view(torch.int32), v.view(torch.int32))


def test_release_rejects_a_bad_device(gpu):
    assert lib().ccm_release_memory(-1) == _lib.CCM_ERR_INVALID
    assert lib().ccm_release_memory(64) == _lib.CCM_ERR_INVALID
