"""Entrywise MPF products, sums and renormalisation at the edges of the shared-memory column arithmetic: limb
counts around multiples of four (the product's word blocks) and at both ends of the range, operands that are
normalised, unnormalised, zero, the lowest two's-complement value, and products whose guard word is all ones;
every pair of a set of mantissas, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def _mantissas(L, rng):
    nb = 32 * L - 2
    one = 1 << (nb - 1)
    vals = [0, 1, 3, one, one + 1, (1 << nb) - 1, (1 << nb) - 2, (1 << (32 * L - 1)) - 1, 1 << (nb // 2),
            (1 << nb) - (1 << (nb // 2)), one + (1 << (nb // 3)), (one | 0xffffffff) & ((1 << nb) - 1)]
    vals += [int.from_bytes(rng.bytes(4 * L), "little") % one + one for _ in range(5)]       # normalised
    vals += [int.from_bytes(rng.bytes(4 * L), "little") % (1 << max(1, nb - k)) for k in (3, 40, nb // 2)]
    vals = vals + [-v for v in vals if v] + [-(1 << (32 * L - 1))]
    return vals


@pytest.mark.parametrize("L", [1, 2, 4, 5, 8, 10, 25, 26, 27, 28, 50, 160])
def test_mul_add_norm_all_pairs(L):
    from sdpvibe_b200 import mpf
    rng = np.random.default_rng(L)
    vals = _mantissas(L, rng)
    m = O.to_limbs(vals, L)
    q = len(vals)
    a, b = np.repeat(np.arange(q), q), np.tile(np.arange(q), q)
    Am, Bm = np.ascontiguousarray(m[:, a]), np.ascontiguousarray(m[:, b])
    zero = np.array([v == 0 for v in vals])
    gap = rng.choice([-32 * L - 200, -32 * L - 3, -32 * L, -65, -33, -32, -31, -1, 0, 0, 1, 32, 64, 32 * L], size=q * q)
    Ae = np.where(zero[a], -(1 << 40), rng.integers(-50, 50, size=q * q))
    Be = np.where(zero[b], -(1 << 40), Ae.clip(-100) + gap)
    A = mpf.MPF(torch.from_numpy(Am).cuda(), torch.from_numpy(Ae).cuda())
    B = mpf.MPF(torch.from_numpy(Bm).cuda(), torch.from_numpy(Be).cuda())
    for got, want in ((mpf.mul(A, B), O.mpf_mul(Am, Ae, Bm, Be)), (mpf.add(A, B), O.mpf_add(Am, Ae, Bm, Be, 1)),
                      (mpf.add(A, B, -1), O.mpf_add(Am, Ae, Bm, Be, -1)),
                      (mpf.normalize(A.m, A.e, L), O.mpf_norm(Am, Ae, L))):
        assert np.array_equal(got.m.cpu().numpy(), want[0])
        assert np.array_equal(got.e.cpu().numpy(), want[1])


def test_mul_scalar_operand_and_wide_norm():
    from sdpvibe_b200 import mpf
    rng = np.random.default_rng(7)
    L = 26
    m = O.to_limbs(_mantissas(L, rng), L)
    e = np.zeros(m.shape[1], np.int64)
    A = mpf.MPF(torch.from_numpy(m).cuda(), torch.from_numpy(e).cuda())
    B = A[17:18]
    want = O.mpf_mul(m, e, np.repeat(m[:, 17:18], m.shape[1], 1), e)
    got = mpf.mul(A, B)
    assert np.array_equal(got.m.cpu().numpy(), want[0]) and np.array_equal(got.e.cpu().numpy(), want[1])
    for LI in (1, 27, 54, 160):
        x = O.to_limbs(_mantissas(LI, rng), LI)
        ex = np.arange(x.shape[1], dtype=np.int64)
        want = O.mpf_norm(x, ex, L)
        got = mpf.normalize(torch.from_numpy(x).cuda(), torch.from_numpy(ex).cuda(), L)
        assert np.array_equal(got.m.cpu().numpy(), want[0]) and np.array_equal(got.e.cpu().numpy(), want[1])
