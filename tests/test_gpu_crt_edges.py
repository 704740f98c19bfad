"""CRT reconstruction at the edges of its kernel: one and two digit chunks and K tiles, resident and streamed
digit tables (contexts of up to and over 128 moduli), the 64-bit digit sums (over 168 moduli), the largest
context it takes, entry counts around the 128-entry tiles and over several tiles per CTA; extreme values, bit
for bit against the oracle.  The float quotient of the pre-pass is checked for every modulus on the CPU."""
import random

import numpy as np
import pytest
import torch

import oracle as O


def test_float_quotient_needs_one_correction():
    """q = round(a float(inv / m)) in float32 leaves |a inv - q m| <= m (1/2 + 2^-8): every modulus of the largest
    context, extreme and random int16 residues"""
    T = O.tables(58)
    rng = np.random.default_rng(0)
    for m, inv in zip(T.mods, T.inv):
        m, inv = int(m), int(inv)
        a = np.concatenate([np.arange(0, 300), np.arange(m - 300, m), rng.integers(0, m, 3000)])
        t = (a.astype(np.float32).astype(np.float64) * float(np.float32(inv / m)) + 12582912.0).astype(np.float32)
        q = t.astype(np.float64) - 12582912.0
        x = a.astype(np.int64) * inv - q.astype(np.int64) * m
        assert np.abs(x).max() <= m / 2 + m / 256
        y = np.where(x < 0, x + m, x)
        assert (y >= 0).all() and (y < m).all() and ((y - a * inv) % m == 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("L,count", [(1, 1), (8, 127), (14, 128), (26, 129), (29, 40000), (30, 40000), (39, 131), (8, 60001), (14, 76000), (26, 151552), (28, 37889),
                                     (40, 20000), (58, 700)])
def test_crt_shapes(L, count):
    from sdpvibe_b200.mpmat import ctx
    rng = random.Random(L)
    T = O.tables(L)
    R = ctx(L)
    lim = T.M // 4
    base = [rng.randrange(-lim + 1, lim) >> rng.randrange(0, T.M.bit_length() - 3) for _ in range(min(count, 120))]
    special = [0, lim - 1, -lim + 1, -1, 1, -(1 << 64), 1 << 31, (1 << (32 * L - 2)) - 1]
    base[:min(len(special), len(base))] = special[:len(base)]
    pick = np.array([rng.randrange(len(base)) for _ in range(count)])
    pick[:min(count, len(base))] = np.arange(min(count, len(base)))
    one = np.array([[v % p for v in base] for p in T.mods], np.int16)
    acc = np.ascontiguousarray(one[:, pick]).reshape(T.n, 1, count)
    Wd, bl = O.crt_block(T, one.reshape(T.n, 1, -1), len(base), 0, len(base), 1)
    rexp = np.array([17], np.int64)
    cexp = np.arange(count, dtype=np.int64) - 5
    rm, re_ = O.mpf_norm(Wd, np.zeros(len(base), np.int64), L)
    re_ = np.where(re_[pick] == -(1 << 40), re_[pick], re_[pick] + 17 + cexp)
    cu = lambda a: torch.from_numpy(a).cuda()
    m, e = R.crt_norm(cu(acc), count, 0, count, 1, cu(rexp), cu(cexp), L)
    assert np.array_equal(m.cpu().numpy(), rm[:, pick]) and np.array_equal(e.cpu().numpy(), re_)
    W2, bl2, _ = R.crt_block(cu(acc), count, 0, count, 1)
    assert np.array_equal(W2.cpu().numpy(), Wd[:, pick]) and np.array_equal(bl2.cpu().numpy(), bl[pick])
