// Step-length eigenvalues on the GPU (FP64): batched symmetric eigenvalues by cyclic Jacobi.
//
// The step length needs lambda_min of M = L^-1 dM L^-T per block (sdpvibe/solver.py:1064-1093); the
// reference takes a float64 copy of M (scaled to O(1)) to the host and calls LAPACK.  Here the copy stays
// on the device: one CTA per block, the block in shared memory, rotations in the round-robin parallel
// order (n/2 disjoint (p, q) pairs per step: rows first, then columns, then the exact 2 x 2 update of the
// pivots), sweeps until the off-diagonal mass is below (eps ||A||_F)^2 / 4 or 40 sweeps.
//
// What bounds it: the latency of a step -- the rotations' square roots and divisions, then the update.  A thread
// takes the 2 x 2 sub-block of a row pair and a column pair and applies both rotations to it in registers (each
// entry is touched by exactly one such pair of rotations), so a step is one pass over the block and two barriers
// instead of two passes, a pivot pass and four; the same bits (the products and fused products of each rotation are
// written out as the two passes had them).  The sub-blocks are dealt to the threads one after the other, in CTAs of
// as many warps as there are sub-blocks: with many small blocks several CTAs share an SM, and warps that only reach
// the barriers, or run half empty, cost as much as working ones.  Against the two passes on 256 threads: six blocks of
// 64 rows 2.95 -> 0.75 ms, of 128 rows 23.8 -> 3.6 ms, 360 blocks of 21 rows 196 -> 162 us, of 41 rows 727 -> 591 us (on
// 512 threads with a warp per row pair those two were 327 and 1048 us).
//
// Error bound returned with each block: a rotation applied in float64 is an exact orthogonal similarity of
// a matrix perturbed by at most a few eps ||A||_F in each of the 2 (n - 1) rotations an entry takes per
// sweep, and the final off-diagonal part moves eigenvalues by at most its Frobenius norm (Weyl):
//   err = (6 n S + n + 2) eps ||A||_F + ||off(A_final)||_F   (S sweeps),
// a larger bound than LAPACK's (n + 2) eps ||A||_F; a block it does not resolve goes to the
// multiprecision refinement, as in the reference.
#include <cmath>

#include "common.cuh"

namespace {

constexpr int kThreads = 512;              // at most
constexpr int kSum = 256;                  // terms t, t + kSum, ... form partial sum t of a norm (the order is part of the result)
constexpr int kNmax = 128;                 // blocks up to 128 x 128 (even padded size <= 128)

// The sum of the squares a[e]^2, e < n, that `take` selects, over the CTA's threads: kSum partial sums as above, summed by
// butterflies of 32 and in ascending order of these.  red: kSum / 32 values of shared memory; the result is in thread 0.
template <class Take>
__device__ __forceinline__ double sum_squares(const double* a, int n, double* red, Take take) {
  const int lane = threadIdx.x & 31;
  for (int g = threadIdx.x >> 5; g < kSum / 32; g += blockDim.x >> 5) {
    double part = 0.0;
    if (32 * g >= n) break;                              // empty sums are left out: 0 + 0
    for (int e = 32 * g + lane; e < n; e += kSum)
      if (take(e)) part = fma(a[e], a[e], part);
    for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) red[g] = part;
  }
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < kSum / 32; k++) t += 32 * k < n ? red[k] : 0.0;
  return t;
}

template <bool ROWS>
__global__ void __launch_bounds__(kThreads) jacobi_kernel(const double* __restrict__ A, int n, double* __restrict__ w,
                                                          double* __restrict__ err, int* __restrict__ sweeps_out) {
  extern __shared__ __align__(16) double sa[];          // np x np, row-major
  __shared__ double red[kSum / 32];
  __shared__ double cs[kNmax / 2], sn[kNmax / 2], tt[kNmax / 2], dp[kNmax / 2], dq[kNmax / 2];
  __shared__ int pp[kNmax / 2], qq[kNmax / 2];
  __shared__ double s_norm, s_off;
  __shared__ int s_done;
  const int np = n + (n & 1);                            // an odd size gets an inert zero row / column
  const int tid = threadIdx.x, T = blockDim.x;
  const double* Ab = A + (size_t)blockIdx.x * n * n;
  for (int e = tid; e < np * np; e += T) {
    const int i = e / np, j = e % np;
    sa[e] = (i < n && j < n) ? Ab[(size_t)i * n + j] : 0.0;
  }
  __syncthreads();
  // ||A||_F
  const double sq = sum_squares(sa, np * np, red, [](int) { return true; });
  if (tid == 0) {
    s_norm = sqrt(sq);
    s_done = 0;
  }
  __syncthreads();
  const double eps = 2.220446049250313e-16;              // 2^-52
  const double tol = 0.25 * (eps * s_norm) * (eps * s_norm);
  const int half = np / 2;
  const int k0 = tid / half, l0 = tid - k0 * half, dk = T / half, dl = T - dk * half;
  int sweep = 0;
  for (; sweep < 40 && !s_done; sweep++) {
    for (int r = 0; r < np - 1; r++) {
      // round-robin pairs: position 0 fixed, positions 1..np-1 rotated by r
      if (tid < half) {
        const int a = tid, b = np - 1 - tid;
        const int p0 = a == 0 ? 0 : 1 + (a - 1 + r) % (np - 1);
        const int q0 = 1 + (b - 1 + r) % (np - 1);
        const int p = p0 < q0 ? p0 : q0, q = p0 < q0 ? q0 : p0;
        const double apq = sa[p * np + q], app = sa[p * np + p], aqq = sa[q * np + q];
        double c = 1.0, s = 0.0, t = 0.0;
        if (apq != 0.0) {
          const double theta = (aqq - app) / (2.0 * apq);
          t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(1.0 + theta * theta));
          c = 1.0 / sqrt(1.0 + t * t);
          s = t * c;
        }
        pp[tid] = p;
        qq[tid] = q;
        cs[tid] = c;
        sn[tid] = s;
        tt[tid] = t * apq;                               // the pivots move by -/+ t a_pq
        dp[tid] = app;
        dq[tid] = aqq;
      }
      __syncthreads();
      auto rotate = [&](int k, int l) {                  // rows p, q of pair k, columns u, v of pair l
        const int p = pp[k], q = qq[k], u = pp[l], v = qq[l];
        if (k == l && sn[k] != 0.0) {                    // the rotated 2 x 2 block exactly
          sa[p * np + p] = dp[k] - tt[k];
          sa[q * np + q] = dq[k] + tt[k];
          sa[p * np + q] = 0.0;
          sa[q * np + p] = 0.0;
          return;
        }
        double c = cs[k], s = sn[k];
        const double apu = sa[p * np + u], aqu = sa[q * np + u], apv = sa[p * np + v], aqv = sa[q * np + v];
        const double rpu = fma(c, apu, -(s * aqu)), rqu = fma(s, apu, c * aqu);
        const double rpv = fma(c, apv, -(s * aqv)), rqv = fma(s, apv, c * aqv);
        c = cs[l];
        s = sn[l];
        sa[p * np + u] = fma(c, rpu, -(s * rpv));
        sa[p * np + v] = fma(s, rpu, c * rpv);
        sa[q * np + u] = fma(c, rqu, -(s * rqv));
        sa[q * np + v] = fma(s, rqu, c * rqv);
      };
      if (ROWS) {                                        // a warp per row pair
        for (int k = tid >> 5; k < half; k += T >> 5)
          for (int l = tid & 31; l < half; l += 32) rotate(k, l);
      } else {                                           // sub-blocks tid, tid + T, ...
        int k = k0, l = l0;
        for (int e = tid; e < half * half; e += T) {
          rotate(k, l);
          k += dk;
          l += dl;
          if (l >= half) l -= half, k++;
        }
      }
      __syncthreads();
    }
    // off-diagonal mass
    const double off = sum_squares(sa, np * np, red, [&](int e) { return e / np != e % np; });
    if (tid == 0) {
      s_off = off;
      s_done = off <= tol;
    }
    __syncthreads();
  }
  // eigenvalues: the diagonal (without the inert padding entry), ascending by rank
  for (int i = tid; i < n; i += T) {
    const double v = sa[i * np + i];
    int rank = 0;
    for (int j = 0; j < n; j++) {
      const double u = sa[j * np + j];
      rank += (u < v) || (u == v && j < i);
    }
    w[(size_t)blockIdx.x * n + rank] = v;
  }
  if (tid == 0) {
    err[blockIdx.x] = (6.0 * n * sweep + n + 2) * eps * s_norm + sqrt(s_off);
    if (sweeps_out) sweeps_out[blockIdx.x] = sweep;
  }
}

}  // namespace

extern "C" int sdpv_eig_sym_f64(const double* A, int64_t nb, int n, double* w, double* err, int* sweeps, void* stream) {
  if (nb < 0 || n < 1 || n > kNmax || nb > 0x7fffffff) return SDPV_EINVAL;
  if (nb == 0) return SDPV_OK;
  const int np = n + (n & 1);
  const size_t smem = (size_t)np * np * sizeof(double);
  static bool attr[64] = {};
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!attr[dev & 63]) {
    const int most = (int)(kNmax * kNmax * sizeof(double));
    cudaError_t e = cudaFuncSetAttribute(jacobi_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(jacobi_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return sdpv::set_cuda_error(e);
    attr[dev & 63] = true;
  }
  // Warps for the sub-blocks in as few rounds as the threads allow: 512 (at 62 registers two such CTAs share an SM),
  // 256 where three or four blocks share one, 128 from five on.  A warp per row pair where that takes no more rounds (its
  // row's rotation is read once and without conflicts).
  const int64_t by_smem = 227 * 1024 / (smem + 6 * 1024), by_count = (nb + sms - 1) / sms;
  const int64_t per_sm = by_smem < by_count ? by_smem : by_count;
  const int half = np / 2, pairs = half * half, most = per_sm <= 2 ? kThreads : (per_sm <= 4 ? 256 : 128);
  const int rounds = (pairs + most - 1) / most;
  int threads = ((pairs + rounds - 1) / rounds + 31) / 32 * 32;
  if (threads < 64) threads = 64;
  const bool by_rows = ((half + most / 32 - 1) / (most / 32)) * ((half + 31) / 32) <= rounds;
  if (by_rows)
    jacobi_kernel<true><<<(unsigned)nb, most, smem, sdpv::as_stream(stream)>>>(A, n, w, err, sweeps);
  else
    jacobi_kernel<false><<<(unsigned)nb, threads, smem, sdpv::as_stream(stream)>>>(A, n, w, err, sweeps);
  return sdpv::launch_status();
}
