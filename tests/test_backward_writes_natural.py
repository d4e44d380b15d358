"""The write set of the sparse path's backward on natural slots (CPU restatement of the
index arithmetic of bwd_output_natural): slot q L + l of state q in column l, the ones
slot at 21 L.  With the tied gradient every coupling entry (s1, s2) of two different
alignment columns gets exactly one addition of its sum, directly or mirrored, and every
other addition is a zero that stays inside its row of 32 L; with the partial one every
entry gets its sum, self blocks included.  Every single field is stored once."""
import numpy as np
import pytest

Q = 21


def writes(L, sym):
    nat = Q * L
    blocks = -(-(nat + 1) // 256)
    g2 = np.zeros((nat, 32 * L), dtype=np.int64)  # additions of a sum
    g1 = np.zeros((Q - 1) * L, dtype=np.int64)
    for Qb in range(blocks):
        for P in range(Qb + 1 if sym else blocks):
            s1, s2 = np.meshgrid(P * 256 + np.arange(256), Qb * 256 + np.arange(256), indexing="ij")
            # the accumulators that are zeroed in their registers
            zero = s2 >= nat
            if sym:
                zero = zero | ((s2 - s1) % L == 0)
                if P != Qb:  # mirrored: row s2 of g2, column s1
                    m = s2 < nat
                    assert (s1[m] < nat).all()
                    np.add.at(g2, (s2[m], s1[m]), ~zero[m])
                at = (s2 == nat) & (s1 < (Q - 1) * L)
                np.add.at(g1, s1[at], 1)
            else:
                at = (s1 == nat) & (s2 < (Q - 1) * L)
                np.add.at(g1, s2[at], 1)
            # direct, four columns at a time: both triangles of a diagonal tile
            d = (s1 < nat) & (s2 - s2 % 4 < nat)
            assert (s2[d] < 32 * L).all()
            np.add.at(g2, (s1[d], s2[d]), ~zero[d])
    return g2, g1


@pytest.mark.parametrize("L", [1, 2, 12, 13, 25, 37])
@pytest.mark.parametrize("sym", [True, False])
def test_one_addition_per_entry(L, sym):
    g2, g1 = writes(L, sym)
    expect = np.zeros_like(g2)
    expect[:, :Q * L] = 1
    if sym:
        l = np.arange(Q * L) % L
        expect[:, :Q * L] = l[:, None] != l[None, :]
    assert np.array_equal(g2, expect)
    assert (g1 == 1).all()
