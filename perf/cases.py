"""The work that programs on top of this package have it do, as timed cases.

The sizes are those of the package's own benchmark workloads and solver (832-bit numbers, L = 26 limbs, a Gram
matrix of 274 columns, 600 uneven SPD blocks of 8 ... 160 rows, SDP blocks of up to 41 points and 21-row bases
against up to 1000 free variables, 256 x 256 products at 768 bits), with small calls beside them.  Numbers are
full-width random mantissas with exponents spread over a few binades, as intermediate results of a solver are.
Results are limb planes and exponents: every operation is defined bit by bit, so outputs are whole numbers.
"""
import math

import numpy as np
import torch

from sdpvibe_b200 import mpf
from sdpvibe_b200.adjoint import gemm_vjp
from sdpvibe_b200.sdp_io import decode_bigfloats, encode_bigfloats, limbs_for_precision
from sdpvibe_b200.solver import SDP, Solver, copy_lower_to_upper
from sdpvibe_b200.synthetic import damped_bases, ising_like_shapes

DEV = "cuda"


def listed():
    return [
        # one small product: a scalar-sized step between host decisions; latency and launches are all there is
        dict(name="gemm_small", op="gemm", L=10, nb=1, M=17, K=12, N=20, transA=False, transB=False),
        # the benchmark's single product: 256 x 256 x 256 at 768 bits
        dict(name="gemm_256", op="gemm", L=24, nb=1, M=256, K=256, N=256, transA=False, transB=False),
        # constraint sums of one chunk of the solver: V diag(a) V^T for both parities of 180 blocks of dimension 1
        dict(name="gemm_blocks", op="gemm", L=26, nb=360, M=21, K=41, N=21, transA=False, transB=True),
        # the primal residual of the same chunk, B^T x: one column against 7380 x 1000
        dict(name="gemm_matvec", op="gemm", L=26, nb=1, M=1000, K=7380, N=1, transA=True, transB=False),
        # the backward pass of a ragged product (cotangents of both factors)
        dict(name="gemm_backward", op="gemm_vjp", L=26, nb=1, M=150, K=274, N=91, transA=False, transB=False),
        # Q = sum_c P_c^T P_c over four chunks, the benchmark's Gram step
        dict(name="gram_274", op="gram", L=26, N=274, rows=7250, chunks=4),
        # Cholesky and solve of the 600 uneven blocks of the benchmark, 8 right-hand sides
        dict(name="chol_blocks", op="chol", L=26, blocks=600, nmin=8, nmax=160, nrhs=8),
        # one matrix the size of Q, two right-hand sides: the serial chain of one factorisation
        dict(name="chol_single", op="chol", L=26, blocks=1, nmin=274, nmax=274, nrhs=2),
        # entrywise products of one chunk's pairings (2 x 180 blocks of 41 x 41)
        dict(name="mul_pairings", op="mul", L=26, n=605160),
        # entrywise sums at twice the working precision (the precision checks run there), an odd count
        dict(name="add_wide", op="add", L=50, n=150001),
        # a block file's matrix of 66 x 1000 numbers read at 1024 bits of file precision
        dict(name="decode_block", op="decode", L=26, n=66000, precision=1024),
        # the solver itself: two iterations of a 20-block SDP with 60 free variables
        dict(name="solver_small", op="solver", L=26, blocks=20, N=60, iters=2),
    ]


LIMBS = (8, 10, 16, 20, 24, 26, 26, 26, 26, 28, 34, 50)


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "gemm_vjp", "gram", "chol", "chol", "mul", "add", "codec", "solver"])
    L = rng.choice(LIMBS)
    if op == "gemm":
        shape = rng.choice(["square", "blocks", "vector"])
        tA, tB = rng.random() < 0.5, rng.random() < 0.5
        if shape == "square":
            return dict(op=op, L=L, nb=1, M=_log(rng, 4, 300), K=_log(rng, 4, 300), N=_log(rng, 4, 300), transA=tA,
                        transB=tB)
        if shape == "blocks":
            return dict(op=op, L=L, nb=_log(rng, 2, 360), M=_log(rng, 4, 64), K=_log(rng, 4, 64), N=_log(rng, 4, 64),
                        transA=tA, transB=tB)
        return dict(op=op, L=min(L, 28), nb=1, M=_log(rng, 32, 1000), K=_log(rng, 32, 7300), N=rng.choice([1, 1, 2, 3]),
                    transA=tA, transB=False)
    if op == "gemm_vjp":
        return dict(op=op, L=L, nb=1, M=_log(rng, 8, 200), K=_log(rng, 8, 300), N=_log(rng, 8, 200),
                    transA=rng.random() < 0.5, transB=rng.random() < 0.5)
    if op == "gram":
        return dict(op=op, L=min(L, 28), N=_log(rng, 16, 270), rows=_log(rng, 100, 7200), chunks=rng.randint(1, 4))
    if op == "chol":
        L = min(L, 34)
        if rng.random() < 0.4:
            n = _log(rng, 8, 270)
            return dict(op=op, L=L, blocks=1, nmin=n, nmax=n, nrhs=rng.randint(1, 9))
        nmax = _log(rng, 12, 150)
        return dict(op=op, L=L, blocks=_log(rng, 4, 300), nmin=rng.randint(4, nmax), nmax=nmax, nrhs=rng.randint(1, 9))
    if op in ("mul", "add"):
        return dict(op=op, L=L, n=_log(rng, 100, 600000) // (2 if L > 28 else 1))
    if op == "codec":
        return dict(op=rng.choice(["decode", "encode"]), L=L, n=_log(rng, 100, 60000),
                    precision=32 * (L - 1) + 64 * rng.randint(0, 4))
    return dict(op="solver", L=rng.choice([8, 16, 24, 26]), blocks=rng.randint(3, 18), N=rng.randint(5, 55), iters=1)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7fffffff)


def _rand(g, shape, L, spread=8):
    """random normalised numbers: full-width mantissas of either sign, values over 2 spread binades"""
    n = int(np.prod(shape))
    w = torch.randint(-(1 << 31), (1 << 31) - 1, (L, n), dtype=torch.int32, device=DEV, generator=g)
    e = torch.randint(-spread, spread + 1, (n,), dtype=torch.int64, device=DEV, generator=g) - 32 * L
    return mpf.normalize(w, e, L).reshape(*shape)


def _spd(g, ns, npad, L):
    """blocks G G^T + n I of the given sizes, each padded to npad with the identity"""
    nb = len(ns)
    G = _rand(g, (nb, npad, npad), L, spread=1)
    n = torch.tensor(ns, device=DEV)[:, None]
    inside = torch.arange(npad, device=DEV)[None] < n                              # (nb, npad)
    keep = inside[:, :, None] & inside[:, None, :]
    G = mpf.MPF(G.m * keep[None].to(torch.int32), torch.where(keep, G.e, torch.full_like(G.e, mpf.EZ)))
    A = mpf.gemm(G, G, transB=True)
    d = torch.where(inside, n.double(), torch.ones((), dtype=torch.float64, device=DEV))
    return mpf.add(A, mpf.from_float(torch.diag_embed(d), L))


def _sizes(case):
    """block sizes of a batched Cholesky, by padded size (multiples of 32): part of the case, not of the seed"""
    rng = np.random.default_rng(case["blocks"])
    by = {}
    for n in rng.integers(case["nmin"], case["nmax"] + 1, size=case["blocks"]):
        by.setdefault(-(-int(n) // 32) * 32, []).append(int(n))
    return sorted(by.items())


def _gemm_shapes(case):
    M, K, N, nb = case["M"], case["K"], case["N"], case["nb"]
    a, b = ((K, M) if case["transA"] else (M, K)), ((N, K) if case["transB"] else (K, N))
    return (a, b) if nb == 1 else ((nb, *a), (nb, *b))


def prepare(case, seed):
    op, L, g = case["op"], case["L"], _gen(seed)
    if op in ("gemm", "gemm_vjp"):
        a, b = _gemm_shapes(case)
        s = dict(case=case, A=_rand(g, a, L), B=_rand(g, b, L))
        if op == "gemm_vjp":
            s["G"] = _rand(g, (case["M"], case["N"]), L)
        return s
    if op == "gram":
        return dict(case=case, P=[_rand(g, (case["rows"], case["N"]), L) for _ in range(case["chunks"])])
    if op == "chol":
        pairs = []
        for npad, ns in _sizes(case):
            if len(ns) == 1:                                                       # one block: its own size
                npad = ns[0]
            pairs.append((_spd(g, ns, npad, L), _rand(g, (len(ns), npad, case["nrhs"]), L)))
        return dict(case=case, pairs=pairs)
    if op in ("mul", "add"):
        return dict(case=case, A=_rand(g, (case["n"],), L), B=_rand(g, (case["n"],), L))
    if op in ("decode", "encode"):
        A = _rand(g, (case["n"],), L)
        nl = limbs_for_precision(case["precision"])
        return dict(case=case, nl=nl, **(dict(A=A) if op == "encode" else dict(buf=encode_bigfloats(A, nl))))
    blocks, N = ising_like_shapes(case["blocks"], case["N"], seed=case["blocks"])  # shapes: part of the case
    for bl in blocks:
        P = bl["K"] * bl["dim"] * (bl["dim"] + 1) // 2
        bl["Ve"], bl["Vo"] = damped_bases(bl["d"], bl["he"], bl["ho"])
        bl["c"], bl["B"] = _rand(g, (P, 1), L), _rand(g, (P, N), L)
    return dict(case=case, sdp=SDP(blocks, _rand(g, (N, 1), L), 0, L))


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "gemm":
        C = mpf.gemm(state["A"], state["B"], case["transA"], case["transB"])
        return C.m, C.e
    if op == "gemm_vjp":
        dA, dB = gemm_vjp(state["A"], state["B"], state["G"], case["transA"], case["transB"])
        return dA.m, dA.e, dB.m, dB.e
    if op == "gram":
        acc = mpf.GramAcc(case["N"], case["L"])
        for P in state["P"]:
            acc.add(P)
        Q = copy_lower_to_upper(acc.result())                                      # only the lower half is defined
        return Q.m, Q.e
    if op == "chol":
        return [t for X in mpf.chol_solve_many(state["pairs"]) for t in (X.m, X.e)]
    if op == "mul":
        C = mpf.mul(state["A"], state["B"])
        return C.m, C.e
    if op == "add":
        C = mpf.add(state["A"], state["B"], -1)
        return C.m, C.e
    if op == "decode":
        A, end = decode_bigfloats(state["buf"], 0, case["n"], state["nl"], case["L"])
        return A.m, A.e, end
    if op == "encode":
        return np.frombuffer(encode_bigfloats(state["A"], state["nl"]), dtype=np.uint8)
    sol = Solver(state["sdp"], case["L"])
    res = sol.run(max_iter=case["iters"])
    out = [sol.y.m, sol.y.e, float(res["primalObjective"]), float(res["dualObjective"])]
    for st in sol.st:
        x = st["xs"]["x"]
        out += [x.m, x.e]
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def _number(L):
    return 4 * L + 8                                                               # limbs and exponent


def _mac(L):
    """int8 operations of one exact multiply-add of L-limb numbers through 15-bit residues"""
    return 8 * math.ceil((64 * L + 17) / 15)


def work(case):
    op, L = case["op"], case["L"]
    w = _number(L)
    if op in ("gemm", "gemm_vjp"):
        M, K, N, nb = case["M"], case["K"], case["N"], case["nb"]
        if op == "gemm":
            return dict(bytes=nb * (M * K + K * N + M * N) * w, flops=nb * M * K * N * _mac(L))
        return dict(bytes=(2 * M * K + 2 * K * N + M * N) * w, flops=2 * M * K * N * _mac(L))
    if op == "gram":
        N, R = case["N"], case["rows"] * case["chunks"]
        return dict(bytes=(R * N + N * (N + 1) // 2) * w, flops=R * N * (N + 1) // 2 * _mac(L))
    if op == "chol":
        ns = [n for _, v in _sizes(case) for n in v]
        m = case["nrhs"]
        return dict(bytes=sum(n * (n + 1) // 2 + 2 * n * m for n in ns) * w,
                    flops=sum(n ** 3 / 6 + n * n * m for n in ns) * _mac(L))
    if op in ("mul", "add"):
        return dict(bytes=3 * case["n"] * w, flops=case["n"] * (2 * L * L if op == "mul" else 2 * L))
    if op in ("decode", "encode"):
        return dict(bytes=case["n"] * (w + 13 + 8 * limbs_for_precision(case["precision"])), flops=0)
    # per iteration: P = L^-1 B, its Gram matrix, the Schur complements' factors (blocks of about 31 points and
    # dimensions 1, 2, 3 in the ratio 6 : 3 : 1)
    N, b, it = case["N"], case["blocks"], case["iters"]
    P = [31.0] * (b * 6 // 10) + [93.0] * (b * 3 // 10)
    P += [186.0] * (b - len(P))
    macs = sum(p ** 3 / 6 + p * p * N / 2 + p * N * N / 2 for p in P) + N ** 3 / 6
    return dict(bytes=it * sum(p * N + p * p for p in P) * w, flops=it * macs * _mac(L))


def exact(case, seed):
    """every output is a whole number or a count of bytes (limbs, exponents) but the solver's objectives, which
    have no closed form"""
    return None
