// Schur-complement assembly of one chunk in one launch (sdpvibe/solver.py:634-652).
//
// From the pairings AXI = V^T X^-1 V and AY = V^T Y V of both parities ((2 nb, W, W), W = dim K) the
// reference composes S (nb, P, P), P = K dim (dim + 1) / 2, out of elementwise MPF products and sums over
// K x K sub-blocks.  Here one thread makes one lower entry (b, i, j) of S with the same operations in the
// same order:
//   dim 1:   S = AXI_0 AY_0 + AXI_1 AY_1                       (parities 0, 1: the fold)
//   dim > 1: row i in pair segment s_i = (c0, r0) at offset a, column j in s_j = (c1, r1) at offset bb
//            (segment s = c (c + 1) / 2 + r, pairs c >= r); per parity, with A = AXI, Y = AY and
//            [u, v] the entry (u K + a, v K + bb) of a pairing block:
//              el = ((A[c0,r1] Y[r0,c1] + A[r0,r1] Y[c0,c1]) + A[c0,c1] Y[r0,r1]) + A[r0,c1] Y[c0,r1]
//            then S = (el_0 + el_1) 2^-2
// each product and sum rounded as mpf_mul / mpf_add, so S is the composed result bit for bit; S is written
// at (i, j) and (j, i) (the reference copies its lower triangle up), and the diagonal entry of a padding
// row (xmask false) is set to one.
#include <cmath>

#include "common.cuh"
#include "mpcol.cuh"

namespace {
using namespace sdpv;

constexpr int kThreads = kColThreads;

__device__ __forceinline__ void seg_of(int s, int& c, int& r) {
  c = 0;
  while ((c + 1) * (c + 2) / 2 <= s) c++;
  r = s - c * (c + 1) / 2;
}

// words of the working columns (a product's operands, or a sum's), then three kept numbers of L words
__host__ __device__ inline int work_words(int L) { return 2 * ((L + 3) & ~3) > 2 * L + 2 ? 2 * ((L + 3) & ~3) : 2 * L + 2; }

__global__ void __launch_bounds__(kThreads)
    schur_kernel(int L, i64 nb, int P, int K, int dim, const int32_t* __restrict__ A, const i64* __restrict__ eA,
                 const int32_t* __restrict__ Y, const i64* __restrict__ eY, const uint8_t* __restrict__ xmask,
                 const int32_t* __restrict__ onem, i64 onee, int32_t* __restrict__ S, i64* __restrict__ eS) {
  extern __shared__ u32 cols[];
  const i64 ntri = (i64)P * (P + 1) / 2;
  const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nb * ntri) return;
  const i64 b = t / ntri;
  const int q = (int)(t - b * ntri);
  int i = (int)((sqrt(8.0 * q + 1.0) - 1.0) * 0.5);                // lower entry q -> (i, j), j <= i
  while ((i + 1) * (i + 2) / 2 <= q) i++;
  while (i * (i + 1) / 2 > q) i--;
  const int j = q - i * (i + 1) / 2;
  const int W = dim * K;
  const i64 plane = 2 * nb * (i64)W * W, splane = nb * (i64)P * P;
  u32* work = cols + threadIdx.x;
  u32* keep = work + (size_t)work_words(L) * T_;
  auto slot = [&](int s) { return keep + (size_t)s * L * T_; };
  const i64 o1 = (b * P + i) * (i64)P + j, o2 = (b * P + j) * (i64)P + i;
  i64 er;
  // kept number d = entry of AXI at ia times entry of AY at iy; returns its exponent
  auto product = [&](int d, i64 ia, i64 iy) -> i64 {
    i64 e;
    col_mpf_mul(work, A + ia, plane, __ldg(eA + ia), Y + iy, plane, __ldg(eY + iy), L, (int32_t*)slot(d), T_, &e);
    return e;
  };
  auto sum = [&](int x, i64 ex, int y, i64 ey, int32_t* out, i64 stride) -> i64 {
    i64 e;
    col_mpf_add(work, ColSrc{slot(x)}, ex, ColSrc{slot(y)}, ey, 1, L, out, stride, &e);
    return e;
  };
  if (i == j && !xmask[b * P + i]) {
    for (int k = 0; k < L; k++) S[(i64)k * splane + o1] = onem[k];
    er = onee;
  } else {
    i64 ee[2];
    if (dim == 1) {
      for (int p = 0; p < 2; p++) {
        const i64 idx = ((p * nb + b) * W + i) * W + j;
        ee[p] = product(p, idx, idx);
      }
    } else {
      const int si = i / K, a = i - si * K, sj = j / K, bb = j - sj * K;
      int c0, r0, c1, r1;
      seg_of(si, c0, r0);
      seg_of(sj, c1, r1);
      for (int p = 0; p < 2; p++) {
        const i64 base = (p * nb + b) * (i64)W;
        // A[u, v] Y[w, z]: entry (u K + a, v K + bb) of AXI times entry (w K + a, z K + bb) of AY
        auto term = [&](int d, int u, int v, int w, int z) {
          return product(d, (base + u * K + a) * W + v * K + bb, (base + w * K + a) * W + z * K + bb);
        };
        ee[p] = term(p, c0, r1, r0, c1);
        for (int x = 0; x < 3; x++) {
          const i64 et = x == 0 ? term(2, r0, r1, c0, c1) : (x == 1 ? term(2, c0, c1, r0, r1) : term(2, r0, c1, c0, r1));
          ee[p] = sum(p, ee[p], 2, et, (int32_t*)slot(p), T_);
        }
      }
    }
    er = sum(0, ee[0], 1, ee[1], S + o1, splane);
    if (dim > 1 && er != SDPV_EZ) er -= 2;
  }
  if (i != j)
    for (int k = 0; k < L; k++) S[(i64)k * splane + o2] = S[(i64)k * splane + o1];
  eS[o1] = er;
  eS[o2] = er;
}

}  // namespace

extern "C" int sdpv_schur_assemble(int L, int64_t nb, int P, int K, int dim, const int32_t* AXI, const int64_t* eAXI,
                                   const int32_t* AY, const int64_t* eAY, const uint8_t* xmask, const int32_t* one_m,
                                   int64_t one_e, int32_t* S, int64_t* eS, void* stream) {
  if (L < 1 || L > 64 || nb < 0 || K < 1 || dim < 1 || P != K * dim * (dim + 1) / 2) return SDPV_EINVAL;
  const i64 n = nb * (i64)P * (P + 1) / 2;
  if (n == 0) return SDPV_OK;
  const unsigned grid = (unsigned)((n + kThreads - 1) / kThreads);
  const size_t smem = (size_t)(work_words(L) + 3 * L) * kColThreads * 4, most = (size_t)(work_words(64) + 192) * kColThreads * 4;
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(schur_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return sdpv::set_cuda_error(e);
    set[dev & 63] = true;
  }
  schur_kernel<<<grid, kThreads, smem, sdpv::as_stream(stream)>>>(L, nb, P, K, dim, AXI, eAXI, AY, eAY, xmask, one_m, one_e,
                                                                  S, eS);
  return sdpv::launch_status();
}
