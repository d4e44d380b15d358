"""What a context may hold under a memory cap, to the byte: its operands and records, and
nothing for schedules that a capped context does not take."""
import numpy as np
import pytest

from ccmpred_b200 import CcmError, Evaluator, _lib, synth

RECORD = 32  # ccm_result


def up(n, to):
    return -(-n // to) * to


def simt_bytes(L, N):
    return N * L + 4 * N + RECORD + 4 * (N * 21 * L + (21 * L) ** 2 + 20 * L) + 8 * (N + 21 * L)


def sparse_bytes(L, N):
    Np, KP, SB = up(N, 256), up(21 * L, 256), up(21 * L + 1, 256)
    T = -(-L // 9)
    b = SB // 256
    return (N * L + 4 * N + RECORD
            + 3 * KP * 192 * T + 5 * Np * SB + Np * KP + Np * KP // 8  # W, one-hot and R, A, metadata
            + 4 * up(21 * L, 4) + 4 * 21 * L                           # column maxima, twice
            + 8 * 8 * (Np // 128) * T + 8 * 21 * L + 8 * 48 + 4        # partials
            + 4 * 20 * L + 8 * b * (b + 1) // 2)                       # g1, tiles


@pytest.mark.gpu
@pytest.mark.parametrize("path,size", [("simt_f32", simt_bytes), ("tc_i8sp", sparse_bytes)])
@pytest.mark.parametrize("L,N", [(1, 2), (12, 9999), (40, 500)])
def test_exact_cap(gpu, path, size, L, N):
    import torch
    msa = synth.generate(synth.MSAConfig("cap", L, N, seed=5))
    cap = size(L, N)
    x = torch.from_numpy(synth.random_x(L, 6)).cuda()
    g = torch.empty_like(x)
    with Evaluator(msa, path=path, mem_limit=cap) as ev:
        assert np.isfinite(ev.evaluate(x, g))
    with pytest.raises(CcmError) as err:
        Evaluator(msa, path=path, mem_limit=cap - 1)
    assert err.value.code == _lib.CCM_ERR_NOMEM
