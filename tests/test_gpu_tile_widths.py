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
