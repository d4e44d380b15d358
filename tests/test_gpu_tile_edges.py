"""The sparse integer path at the edges of its tiles: widths whose 21 L + 1 natural
slots end just below, at and just above a multiple of the backward's 256-slot tiles
and whose column groups end inside a forward tile, row counts around the 256-row
pairs, and a gradient buffer that is only 4-byte aligned.  Against the FP64 oracle."""
import numpy as np
import pytest

from ccmpred_b200 import Evaluator, nvar_padded, synth

Q = 21


def natural_offset(n, s, KB, mats):
    """Byte of (row n, slot s) in the backward's storage: 128-slot x 32-row tiles,
    `mats` matrices of a tile side by side, 32 bytes per slot, the 16-byte halves of
    slots with bit 2 set exchanged."""
    return ((s >> 7) * KB + (n >> 5)) * (mats * 4096) + (s & 127) * 32 + ((n & 31) ^ ((s & 4) << 2))


@pytest.mark.parametrize("mats", [2, 3])
def test_natural_storage_is_a_bijection(mats):
    Npad, SB = 256, 512
    n, s = np.arange(Npad)[:, None], np.arange(SB)[None, :]
    off = natural_offset(n, s, Npad // 32, mats)
    every = np.concatenate([(off + 4096 * m).ravel() for m in range(mats)])
    assert np.array_equal(np.sort(every), np.arange(mats * Npad * SB))


@pytest.mark.gpu
@pytest.mark.parametrize("gradient", ["tied", "partial"])
@pytest.mark.parametrize("L,N", [(1, 3), (12, 257), (13, 255), (37, 256), (61, 513), (85, 31),
                                 (97, 1025)])
def test_tile_edges(gpu, oracle_mod, L, N, gradient):
    import torch
    msa = synth.generate(synth.MSAConfig("edge", L, N, n_pairs=L // 8, dup_frac=0.2, seed=100 + L))
    w = oracle_mod.oracle_weights(msa, 0.8)
    lam2 = 0.2 * max(L - 1, 1)
    x = synth.random_x(L, 200 + L)
    f64, g64 = oracle_mod.oracle_evaluate(msa, w, 0.01, lam2, x)
    with Evaluator(msa, weights=w, lambda_pair=lam2, gradient=gradient) as ev:
        xd = torch.from_numpy(x).cuda()
        buf = torch.full((nvar_padded(L) + 4,), float("nan"), device="cuda")
        for shift in (0, 1) if L % 4 else (0,):
            gd = buf[shift:shift + nvar_padded(L)]
            f = ev.evaluate(xd, gd)
            g = gd.cpu().numpy().astype(np.float64)
            assert abs(f - f64) < 1e-6 * abs(f64)
            if gradient == "partial":
                # tied = partial + its transpose without the self blocks, the
                # single fields alike
                nsp = g.size - Q * L * 32 * L
                P = g[nsp:].reshape(Q, L, 32, L)[:, :, :Q].reshape(Q * L, Q * L)
                T = np.zeros((Q, L, 32, L))
                S = (P + P.T).reshape(Q, L, Q, L)
                W = x[nsp:].reshape(Q, L, 32, L).astype(np.float64)
                i = np.arange(L)
                S[:, i, :, i] = 2 * lam2 * W[:, i, :Q, i]
                T[:, :, :Q] = S
                g = np.concatenate([g[:nsp], T.ravel()])
            assert np.linalg.norm(g - g64) < 1e-5 * np.linalg.norm(g64)
        assert torch.isnan(buf[shift + nvar_padded(L):]).all()
