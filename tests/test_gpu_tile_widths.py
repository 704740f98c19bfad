"""Base tiles over the limb counts: bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from test_gpu_kernels import _spd_tiles, cu, np_

pytestmark = pytest.mark.gpu


def _factor_and_invert(W, WL, LF):
    """(factor, pivot reciprocals, inverse) of the kernels, and of the oracle"""
    from sdpvibe_b200 import _lib
    nb = W.shape[0]
    tri = np.tril(np.ones((32, 32), bool))
    RA, RR = O.chol_tiles(W, 32, WL, LF)
    RA = np.where(tri[None, :, :, None], RA, 0).astype(np.uint32)
    RX = O.trinv_tiles(RA, RR, 32, WL, LF)
    A, RINV = cu(W.view(np.int32)), torch.zeros((nb, 32, WL), dtype=torch.int32, device="cuda")
    _lib.call("sdpv_chol_tiles", _lib.ptr(A), _lib.ptr(RINV), nb, 32, WL, LF, _lib.stream())
    Lw, X, S = A.clone(), torch.empty_like(A), torch.empty_like(A)
    Lw[:, torch.from_numpy(~tri).cuda()] = 0
    _lib.call("sdpv_trinv_tiles", _lib.ptr(Lw), _lib.ptr(RINV), _lib.ptr(X), _lib.ptr(S), nb, 32, WL, LF, _lib.stream())
    return [np_(t).view(np.uint32) for t in (Lw, RINV, X)], [RA, RR, RX]


@pytest.mark.parametrize("L,ill", [(41, False), (41, True), (57, False), (70, False)])
def test_widest_tiles(L, ill):
    """over 64 words: products of up to three times 32 columns, each with its own range of words (the ill conditioned
    tiles' pivots go down to 2^(-16 L): from L = 48 on the squares of their reciprocals leave the 24 words above the point)"""
    got, want = _factor_and_invert(_spd_tiles(np.random.default_rng(L + 100 * ill), 2, L, ill), L + 24, L)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def _invert(Lw, RR, WL, LF):
    """the kernel's inverse and the oracle's"""
    from sdpvibe_b200 import _lib
    nb = Lw.shape[0]
    A = cu(Lw.view(np.int32))
    X, S = torch.empty_like(A), torch.empty_like(A)
    _lib.call("sdpv_trinv_tiles", _lib.ptr(A), _lib.ptr(cu(RR.view(np.int32))), _lib.ptr(X), _lib.ptr(S), nb, 32, WL, LF,
              _lib.stream())
    return np_(X).view(np.uint32), O.trinv_tiles(Lw, RR, 32, WL, LF)


def _words(v, n):
    return [(v >> (32 * w)) & 0xffffffff for w in range(n)]


@pytest.mark.parametrize("L,extra", [(2, 24), (3, 24), (4, 24), (5, 24), (9, 24), (16, 24), (23, 24), (24, 24), (25, 24), (26, 24),
                                     (28, 24), (33, 24), (39, 24), (40, 24), (7, 1), (8, 2), (25, 1), (26, 6)])
def test_inverse_around_the_unrolled_products(L, extra):
    """every parity and both ends of the limb counts whose products are unrolled; entries of the factor below 1, just 1
    and above, of the inverse on both sides of 2^32 (as far as the words above the point go), zeros and single bits; few
    words above the point"""
    rng = np.random.default_rng(L * 31 + extra)
    nb, WL, one = 3, L + extra, 1 << (32 * L)
    Lw, RR = np.zeros((nb, 32, 32, WL), np.uint32), np.zeros((nb, 32, WL), np.uint32)
    top = 40 if extra > 8 else 3                                     # largest reciprocals: 2^top
    for b in range(nb):
        for i in range(32):
            r = one + int.from_bytes(rng.bytes(4 * L), "little") % one
            if b == 1 and i % 11 == 3:
                r <<= top
            RR[b, i] = _words(r, WL)
            for j in range(i + 1):
                v = int.from_bytes(rng.bytes(4 * L), "little") % one >> (6 if extra > 8 else 9)
                if b == 2 and extra > 8 and (i + j) % 13 == 5:
                    v = one + (v if j % 2 else 0)                    # 1 and a little above
                if (i * 7 + j) % 17 == 0:
                    v = 0 if j % 2 else 1
                Lw[b, i, j] = _words(-v if rng.random() < 0.5 and i != j else v, WL)
    got, want = _invert(Lw, RR, WL, L)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L,extra", [(24, 2), (24, 4), (24, 5), (26, 2), (26, 4), (26, 5)])
def test_inverse_with_few_words_above_the_point(L, extra):
    """entries of the inverse over 2^32 in tiles of 2 to 5 words above the point: nothing past an entry's words is read"""
    rng = np.random.default_rng(L + extra)
    WL, one = L + extra, 1 << (32 * L)
    Lw, RR = np.zeros((1, 32, 32, WL), np.uint32), np.zeros((1, 32, WL), np.uint32)
    for i in range(32):
        RR[0, i] = _words((one << 33) + int.from_bytes(rng.bytes(4 * L), "little"), WL) if i == 0 else _words(one, WL)
        for j in range(i):
            Lw[0, i, j] = _words(int.from_bytes(rng.bytes(4 * L), "little") % one >> 40, WL)
        Lw[0, i, i] = _words(one, WL)
    got, want = _invert(Lw, RR, WL, L)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("L", [4, 7, 16, 24, 27, 34, 40])
@pytest.mark.parametrize("ill", [False, True])
def test_tiles_by_limb_count(L, ill):
    got, want = _factor_and_invert(_spd_tiles(np.random.default_rng(L + 100 * ill), 2, L, ill), L + 24, L)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
