"""Residue products of small blocks packed several to a tile, at the edges of their epilogue: blocks that straddle
the warps' row quarters, one block to many per tile, a last tile with fewer blocks, padded accumulator rows, output
runs that start on an odd entry, overwriting and adding, K on both sides of the limit (64) below which the middle
sum needs no reduction; bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from test_gpu_kernels import cu, np_

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,M,N,K,pad,fresh", [(7, 21, 21, 48, 0, True), (7, 21, 21, 80, 3, True), (5, 43, 17, 64, 0, False),
                                                (3, 64, 64, 16, 0, True), (9, 1, 1, 16, 0, True), (33, 1, 3, 32, 1, False),
                                                (2, 63, 3, 96, 0, True), (130, 5, 5, 16, 0, True), (4, 31, 64, 48, 0, True)])
def test_packed_products(nb, M, N, K, pad, fresh):
    from sdpvibe_b200.mpmat import ctx
    rng = np.random.default_rng(nb * M + N)
    T = O.tables(8)
    R = ctx(8)
    m = T.m32.astype(np.int64)[:, None, None]
    a = rng.integers(0, 1 << 30, size=(T.n, nb * M, K)) % m
    b = rng.integers(0, 1 << 30, size=(T.n, nb * N, K)) % m
    a[:, 0] = m[:, 0] - 1                                            # largest digits
    b[:, 0] = m[:, 0] - 1
    old = (rng.integers(0, 1 << 30, size=(T.n, nb * M, N + pad)) % m).astype(np.int16)
    acc = cu(old)
    split = lambda x: (cu((x >> 7).astype(np.uint8)), cu((x & 127).astype(np.uint8)))
    Ah, Al = split(a)
    Bh, Bl = split(b)
    R.accumulate(Ah, Al, Bh, Bl, acc[:, :, :N] if not pad else acc, nb=nb, fresh=fresh, unsigned=True)
    got = np_(acc)
    for q in range(nb):
        want = np.einsum("gik,gjk->gij", a[:, q * M:(q + 1) * M], b[:, q * N:(q + 1) * N])
        if not fresh:
            want = want + old[:, q * M:(q + 1) * M, :N]
        assert np.array_equal(got[:, q * M:(q + 1) * M, :N], (want % m).astype(np.int16)), q
    assert np.array_equal(got[:, :, N:], old[:, :, N:])
