"""Products with few columns without residues: the Toeplitz operand's layout (CPU: images, the strided reads of the
MMA and the order of the digit sums restated in numpy, against Python integers), and the GPU path against the residue
path over the forms it takes (limb counts at the edges of its K steps and row groups, one to four columns in either
order, blocks of columns that are not full, one to many ranges of k, zeros and unnormalised entries) and the oracle."""
import numpy as np
import pytest


def _digits(v, n):
    """signed base-256 digits of v: the bytes of v + 0x80..80, less 128"""
    u = (v + int.from_bytes(b"\x80" * n, "little")) % (1 << (8 * n))
    return [b - 128 for b in u.to_bytes(n, "little")]


@pytest.mark.parametrize("L", [1, 5, 8, 26, 32])
def test_toeplitz_layout(L):
    rng = np.random.default_rng(L)
    n, ks, nh = 4 * L, (4 * L + 31) // 32, 2 * ((L + 3) // 4)
    nc = 2 * ks + nh - 1
    val = lambda: int(rng.integers(0, 1 << 62)) ** (L // 2 + 1) % (1 << (32 * L - 2)) * int(rng.choice([-1, 1]))
    a, x = [val() for _ in range(3)], val()
    z = np.zeros(16 * nh + 400, np.int64)                            # digit d at 200 + d
    z[200:200 + n] = _digits(x, n)
    image = np.array([[[[z[200 + 16 * nh - 1 - 8 * p - r - b - 16 * m] for b in range(16)] for r in range(8)]
                       for m in range(nc)] for p in range(2)])
    for v in a:
        row = np.zeros(128, np.int64)
        row[:n] = _digits(v, n)
        total = 0
        for p in range(2):
            for h in range(nh):
                for r in range(8):
                    # K step s reads core matrices 2 s + c + h, c = 0, 1: equal strides along K and along the rows
                    d = sum(int(row[32 * s + 16 * c:32 * s + 16 * c + 16] @ image[p, 2 * s + c + h, r])
                            for s in range(ks) for c in range(2))
                    total += d << (8 * (16 * nh - 1 - 16 * h - 8 * p - r))
        assert total == v * x


def _workspace(L, M, K, N):
    import ctypes
    from sdpvibe_b200 import _lib
    need = ctypes.c_int64()
    assert _lib.lib().sdpv_gemm_tall_workspace(L, M, K, N, ctypes.byref(need)) == 0
    return need.value


@pytest.mark.parametrize("L,M,K,N", [(32, 128, 65536, 4), (26, 128, 65536, 3), (26, 1000, 7380, 4), (26, 600, 7380, 4), (8, 128, 4096, 4)])
def test_workspace_stays_below_the_matrix(L, M, K, N):
    """the columns' images are held in pairs where all of them would take more than a quarter of the matrix"""
    assert _workspace(L, M, K, N) < K * M * (4 * L + 8)
    assert _workspace(L, M, K, N) <= max(_workspace(L, M, K, 2), K * M * (4 * L + 8) / 4 + _workspace(L, M, K, 2))


@pytest.mark.parametrize("L", [5, 26, 32])
@pytest.mark.parametrize("M", [1000, 6400, 9600, 10000, 12000, 15000, 18800, 19000, 40000])
@pytest.mark.parametrize("K", [1000, 7380])
def test_split_fills_the_processors(L, M, K):
    """blocks of 128 columns times ranges of k: the rounds of one CTA per SM (148) take at most 1.35 times the steps
    that an even split would (one range per block: up to 1.97), and no range has more values of k than int32 sums hold"""
    nh = 2 * ((L + 3) // 4)
    image = 2 * (2 * ((4 * L + 31) // 32) + nh - 1) * 128
    blocks = (M + 127) // 128
    ranges, rest = divmod(_workspace(L, M, K, 1) - (K * image + 255) // 256 * 256, 16 * nh * blocks * 128 * 4)
    assert rest == 0
    kper = -(-K // ranges)
    assert kper <= 32000 // L
    assert -(-blocks * ranges // 148) * kper <= 1.35 * blocks * K / 148


def _rand(shape, L, seed):
    import torch
    from sdpvibe_b200 import mpf
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = int(np.prod(shape))
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (L, n), dtype=torch.int32, device="cuda", generator=g)
    A = mpf.normalize(w, torch.randint(-40, 40, (n,), device="cuda", generator=g), L)
    A.m[:, ::13] = 0                                                 # zeros
    A.e[::13] = mpf.EZ
    A.m[max(1, L - 2):, 5::17] = 0                                   # short mantissas (not normalised)
    A.m[:, 7::19] = 0                                                # zero mantissas with an exponent
    A = A.reshape(*shape)
    A.m[..., 0] = 0                                                  # a zero column
    A.e[..., 0] = mpf.EZ
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("L,M,K,N,tB", [(1, 5, 3, 1, False), (2, 130, 40, 2, True), (8, 33, 2100, 4, False),
                                        (26, 1000, 530, 1, False), (26, 257, 300, 3, True), (26, 1, 5000, 1, False),
                                        (31, 128, 64, 2, False), (32, 129, 1100, 1, True), (10, 64, 65536, 1, False),
                                        (24, 20000, 17, 1, False), (26, 130, 900, 2, False), (29, 132, 700, 3, True),
                                        (26, 10000, 200, 4, False), (5, 12001, 130, 3, True)])
def test_tall_matches_residue_path(monkeypatch, L, M, K, N, tB):
    import torch
    from sdpvibe_b200 import mpf
    A, B = _rand((K, M), L, 1), _rand((N, K) if tB else (K, N), L, 2)
    got = mpf._gemm_tall(A, B, L, M, K, N, tB)
    monkeypatch.setattr(mpf, "TALL_MIN", 1 << 60)
    want = mpf.gemm(A, B, transA=True, transB=tB)
    assert torch.equal(got.m, want.m) and torch.equal(got.e, want.e)


@pytest.mark.gpu
def test_tall_matches_oracle_and_refuses():
    from oracle import mp as OM
    from sdpvibe_b200 import mpf
    L, M, K, N = 26, 140, 1000, 2
    A, B = _rand((K, M), L, 3), _rand((K, N), L, 4)
    C = mpf.gemm(A, B, transA=True)                                   # by the rule on sizes
    cm, ce = OM.mpf_gemm(A.m.cpu().numpy(), A.e.cpu().numpy(), B.m.cpu().numpy(), B.e.cpu().numpy(), True, False)
    assert np.array_equal(C.m.cpu().numpy(), cm) and np.array_equal(C.e.cpu().numpy(), ce)
    for shape in ((33, 8, 8, 1), (26, 8, 8, 5), (26, 8, 65537, 1)):
        assert mpf._gemm_tall(A, B, *shape, False) is None
