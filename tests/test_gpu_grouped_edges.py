"""Grouped factorisations and solves at the edges of their support kernels: right-hand-side counts around the
column sets of 8 and 32, zero columns (left shifts of the whole width in the column rounding), columns of very
different magnitude, one-row blocks and blocks over several tiles, small and wide limb counts; against the oracle."""
import numpy as np
import pytest

import oracle as O
from oracle import mp as OM
from test_gpu_kernels import _normal_mpf_np, cu, np_

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,n,nr", [(8, 1, 1), (8, 33, 7), (26, 64, 9), (26, 97, 33), (10, 70, 40), (50, 34, 8)])
def test_solve_edges(L, n, nr):
    from sdpvibe_b200.mpf import MPF, Chol, EZ
    rng = np.random.default_rng(n + nr)
    nb = 2
    vals, exps = [], []
    for b in range(nb):
        G = rng.integers(-40, 41, size=(n, n)).astype(object)
        d = rng.integers(-20, 21, size=n)
        A = G.dot(G.T) + np.eye(n, dtype=object) * (50 * n)
        for i in range(n):
            for j in range(n):
                vals.append(int(A[i, j]))
                exps.append(int(d[i] + d[j]))
    m, e = O.mpf_norm(O.to_limbs(vals, L), np.array(exps, np.int64), L)
    Am, Ae = m.reshape(L, nb, n, n), e.reshape(nb, n, n)
    Bm, Be = _normal_mpf_np(rng, L, (nb, n, nr), -20, 20)
    Be = Be + 40 * L * (np.arange(nr) - nr // 2)                     # magnitudes far apart by column
    Bm[:, 0, :, 0] = 0                                               # a zero column
    Be[0, :, 0] = EZ
    Bm[:, 1, n // 2:, nr - 1] = 0                                    # and a half zero one
    Be[1, n // 2:, nr - 1] = EZ
    ref = OM.Chol(Am, Ae)
    ch = Chol(MPF(cu(Am), cu(Ae)))
    assert np.array_equal(np_(ch.Lt.limbs), ref.Lt)
    B = MPF(cu(Bm), cu(Be))
    for (rm, re_), got in ((ref.solve_lower(Bm, Be), ch.solve_lower(B)), (ref.solve(Bm, Be), ch.solve(B))):
        assert np.array_equal(np_(got.m), rm) and np.array_equal(np_(got.e), re_)
