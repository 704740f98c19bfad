"""The fused operand set-up of a product (exponents and alignment of both sides in two launches) against the
separate kernels (sdpv_top_max, sdpv_align) for all four orders, at the edges of its launch shapes: vectors of one
entry, contiguous vectors around the warp / CTA limit of 512, strided ones split over several CTAs, single
columns, batches, zero vectors and unnormalised entries; and whole products in those shapes against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (5, 7, 64, 9), (5, 7, 65, 9), (1, 5, 512, 3), (1, 3, 513, 2), (1, 33, 1100, 31), (3, 9, 41, 1), (2, 1, 600, 40),
          (4, 21, 44, 17), (1, 1, 1030, 1), (2, 40, 7, 65)]


def _rand(shape, L, seed):
    from sdpvibe_b200 import mpf
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = int(np.prod(shape))
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (L, n), dtype=torch.int32, device="cuda", generator=g)
    e = torch.randint(-60, 60, (n,), device="cuda", generator=g)
    A = mpf.normalize(w, e, L)
    A.m[:, ::7] = 0                                                 # zeros
    A.e[::7] = mpf.EZ
    A.m[max(0, L - 2):, 3::11] = 0                                  # short mantissas (not normalised)
    A = A.reshape(*shape)
    A.m[..., 0, :] = 0                                              # a zero row
    A.e[..., 0, :] = mpf.EZ
    return A


@pytest.mark.parametrize("tA", [False, True])
@pytest.mark.parametrize("tB", [False, True])
@pytest.mark.parametrize("nb,M,K,N", SHAPES)
def test_operands_match_separate_kernels(nb, M, K, N, tA, tB):
    from sdpvibe_b200 import _lib, mpf
    L = 10
    A, B = _rand((nb, K, M) if tA else (nb, M, K), L, 1), _rand((nb, N, K) if tB else (nb, K, N), L, 2)
    ld, ldE = (K + 3) // 4 * 4, N + 3
    X = torch.zeros((L, nb * (M + N), ld), dtype=torch.int32, device="cuda")
    Ea, Eb = (torch.full((nb, n), 77, dtype=torch.int64, device="cuda") for n in (M, ldE))
    _lib.call("sdpv_gemm_operands", *(_lib.ptr(t) for t in (A.m, A.e, B.m, B.e)), L, nb, M, K, N, int(tA), int(tB), ld,
              _lib.ptr(X), _lib.ptr(Ea), _lib.ptr(Eb), ldE, _lib.stream())
    ea = mpf._row_exponents(mpf.top_max(A, over_rows=tA), L)
    eb = mpf._row_exponents(mpf.top_max(B, over_rows=not tB), L)
    assert torch.equal(Ea, ea) and torch.equal(Eb[:, :N], eb)
    assert nb == 1 or bool((Eb[:-1, N:] < -(1 << 40)).all() | (Eb[:-1, N:] == 77).all())
    Xa = mpf.aligned(A, ea, per_col=tA, transpose=tA).reshape(L, nb * M, K)
    Xb = mpf.aligned(B, eb, per_col=not tB, transpose=not tB).reshape(L, nb * N, K)
    assert torch.equal(X[:, :nb * M, :K], Xa) and torch.equal(X[:, nb * M:, :K], Xb)
    assert bool((X[:, :, K:] == 0).all())                            # entries past K stay untouched


@pytest.mark.parametrize("nb,M,K,N,tA,tB", [(1, 6, 1100, 3, True, False), (3, 9, 41, 1, False, False),
                                            (2, 70, 5, 65, True, True), (1, 1, 530, 9, False, True)])
def test_products_match_oracle(nb, M, K, N, tA, tB):
    from oracle import mp as OM
    from sdpvibe_b200 import mpf
    L = 10
    A, B = _rand((nb, K, M) if tA else (nb, M, K), L, 3), _rand((nb, N, K) if tB else (nb, K, N), L, 4)
    C = mpf.gemm(A, B, tA, tB)
    for b in range(nb):
        cm, ce = OM.mpf_gemm(A.m[:, b].cpu().numpy(), A.e[b].cpu().numpy(), B.m[:, b].cpu().numpy(),
                             B.e[b].cpu().numpy(), tA, tB)
        assert np.array_equal(C.m[:, b].cpu().numpy(), cm) and np.array_equal(C.e[b].cpu().numpy(), ce)
