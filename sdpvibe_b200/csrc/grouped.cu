// Grouped Cholesky / triangular-solve support kernels: every launch works through a device descriptor table
// whose rows may belong to blocks of different sizes, so one launch serves all blocks of a wave.
//
// Storage (limb planes, plane stride = the arena's entry count):
//   factor arena   (L, T, 32, 32)  lower tiles (b, i, j), i >= j, of every block, fixed point at one exponent e;
//   inverse arena  (L, D, 32, 32)  the inverse X_j of every diagonal tile, exponent xe[d] per tile;
//   solve arena    (L, RT, 32, m)  32-row tiles of the right-hand sides / solutions, exponents Pe (RT, m) per
//                                  (row tile, column);
//   workspaces     (L, rows, KP)   operand rows gathered for one grouped residue product.
// The kernels: tile copies into workspaces (grp_copy, optional transpose, shared-memory staged), the rounding
// of CRT outputs to a fixed exponent combined into a destination (grp_finish_fixed), the solves' per-column
// exponents, rounding and aligned sums (grp_solve_round) and rescales (grp_merge), and the tile conversions
// around the base-case kernels (grp_tile_widen, grp_tile_narrow).  Roundings are the reference's:
// floor(x / 2^s + 1/2) on two's-complement words (sdpvibe/limbops.py:31-62), the aligned sum of two operands
// rounded independently to max(ea, eb) + 1 (sdpvibe/batched.py:55-79), per-column output exponents from the
// maximal bit length (sdpvibe/batched.py:200-231).
//
// What bounds them: with few blocks, the latency of an entry's dependent passes.  So an entry's words are copied into
// a shared-memory column at once (cp.async) and shifted from there, and the entries of a tile or group are spread
// over several CTAs.  Measured (B200, L = 26, one 274-row matrix, per launch): finish 20 -> 5.9 us, narrow 62 -> 11.6,
// widen 43 -> 8.3, solve_round 12.8 -> 6.9, merge 6.2 -> 4.0; 600 blocks of 8 ... 160 rows: finish 121 -> 58, narrow
// 111 -> 84, solve_round 31.5 -> 13.9.
#include "common.cuh"

namespace {

constexpr int kArenas = 4;
constexpr int kLMax = 128;                 // most limbs of a solve's right-hand sides (shared-memory columns of 128 threads)
constexpr int kMaxSrc = 7;                 // rounded products summed into one destination by grp_finish_fixed

struct Arenas {
  int32_t* p[kArenas];
  i64 plane[kArenas];
};

// Two's-complement words of one entry in a shared-memory column of stride T words (word k at c[k T], conflict
// free; T = the CTA's threads): words below 0 are zero, from n on the sign.
struct Col {
  const u32* c;
  int T, n;
  u32 ext;
  __device__ __forceinline__ u32 operator()(int i) const { return i < 0 ? 0u : (i >= n ? ext : c[i * T]); }
};
__device__ __forceinline__ Col make_col(const u32* c, int T, int n) {
  return Col{c, T, n, (c[(n - 1) * T] >> 31) ? 0xffffffffu : 0u};
}
// Shift amounts past these bounds give the same words: all sign above, all zero below.
__device__ __forceinline__ int clamp_shift(i64 s, int n, int nout) {
  const i64 hi = 32 * (i64)(n + 1), lo = -32 * (i64)(nout + 1);
  return (int)(s > hi ? hi : (s < lo ? lo : s));
}
// Streaming floor(x / 2^s + 1/2) of the words w: output word k in ascending order.
template <class Word>
struct Shr {
  Word w;
  int q, r;
  u32 lo, carry;
  __device__ __forceinline__ Shr(Word w_, int s) : w(w_), q(s >> 5), r(s & 31) {
    carry = s > 0 ? (w((s - 1) >> 5) >> ((s - 1) & 31)) & 1u : 0u;
    lo = w(q);
  }
  __device__ __forceinline__ u32 next(int k) {
    const u32 hi = w(q + k + 1);
    const u32 f = __funnelshift_r(lo, hi, r), v = f + carry;
    carry = v < f ? 1u : 0u;
    lo = hi;
    return v;
  }
};
template <class Word>
__device__ __forceinline__ Shr<Word> make_shr(Word w, int s) { return Shr<Word>(w, s); }

// Words [0, n) of an entry (plane stride `plane`) into a column; every copy in flight at once.
__device__ __forceinline__ void stage_col(u32* c, int T, const int32_t* src, i64 plane, int n) {
#pragma unroll 8
  for (int k = 0; k < n; k++, src += plane, c += T) cp_async4(c, src, 4u);
}

__device__ __forceinline__ int col_bits(const u32* c, int stride, int n) {
  const u32 ext = (c[(n - 1) * stride] >> 31) ? 0xffffffffu : 0u;
  for (int k = n - 1; k >= 0; k--) {
    const u32 v = c[k * stride] ^ ext;
    if (v) return 32 * k + 32 - __clz(v);
  }
  return 0;
}

// ---------------------------------------------------------------- tile copies into a workspace
// desc (8 int64): src arena, src base entry, src row stride, dst base entry, dst row stride, rows, cols (<= 32),
// transpose.  One CTA per descriptor and limb plane (grid y); dst[r][c] = src[r][c], or dst[c][r] = src[r][c]
// staged through shared memory so that both sides are read / written along rows.
__global__ void __launch_bounds__(256) grp_copy_kernel(Arenas src, int32_t* __restrict__ dst, i64 dplane, int L,
                                                       const i64* __restrict__ desc) {
  __shared__ int32_t t[32][33];
  const i64* d = desc + 8 * (i64)blockIdx.x;
  const int sid = (int)d[0], rows = (int)d[5], cols = (int)d[6], trans = (int)d[7];
  const i64 sbase = d[1], sld = d[2], dbase = d[3], dld = d[4];
  const int tid = threadIdx.x;
  for (int k = blockIdx.y; k < L; k += gridDim.y) {
    const int32_t* S = src.p[sid] + (i64)k * src.plane[sid] + sbase;
    int32_t* D = dst + (i64)k * dplane + dbase;
    if (!trans) {
      for (int idx = tid; idx < rows * 32; idx += 256) {
        const int r = idx >> 5, c = idx & 31;
        if (c < cols) D[r * dld + c] = S[r * sld + c];
      }
    } else {
      for (int idx = tid; idx < 1024; idx += 256) {
        const int r = idx >> 5, c = idx & 31;
        t[r][c] = (r < rows && c < cols) ? S[r * sld + c] : 0;
      }
      __syncthreads();
      for (int idx = tid; idx < 1024; idx += 256) {
        const int c = idx >> 5, r = idx & 31;          // destination row c, column r
        if (r < rows && c < cols) D[c * dld + r] = t[r][c];
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------- fixed-exponent rounding into a destination
// desc (40 int64): out arena, out base, out ld, base arena (-1: zero), base base, base ld, rows, cols, nsrc (<= 7),
// then per source: CRT entry base, sign (+1 / -1), shift constant, exponent index (-1: none).  Entry (r, c):
//   out = base + sum_i sign_i round(W_i[r][c] / 2^s_i) mod 2^(32 L),  s_i = cst_i - xe[idx_i]
// where W_i[r][c] is the CRT value (W words, planes Ntot apart) at entry crt_base_i + r * w + c.  Eight CTAs per
// descriptor (grid y), one entry per thread for a 32 x 32 block.  Only the L + 2 words that the rounding reads and the
// sign word are staged; the next source is in flight while one is added (the word-by-word loads of a plain loop had
// set the time: 20 us a launch of few tiles, with 32 of them per factorisation of 9 tile columns).
constexpr int kFinT = 128;
__global__ void __launch_bounds__(kFinT) grp_finish_fixed_kernel(const int32_t* __restrict__ Wd, int W, i64 Ntot, i64 w,
                                                                 Arenas ar, int L, const i64* __restrict__ xe,
                                                                 const i64* __restrict__ desc) {
  extern __shared__ u32 cols[];
  u32* sum = cols + threadIdx.x;                        // L words, then two source columns of L + 3 words
  u32* buf = sum + L * kFinT;
  const i64* d = desc + 40 * (i64)blockIdx.x;
  const int oid = (int)d[0], bid = (int)d[3], rows = (int)d[6], ncol = (int)d[7];
  const int ns = (int)d[8] < kMaxSrc ? (int)d[8] : kMaxSrc;
  const i64 obase = d[1], old_ = d[2], bbase = d[4], bld = d[5];
  for (int idx = blockIdx.y * kFinT + threadIdx.x; idx < rows * ncol; idx += gridDim.y * kFinT) {
    const int r = idx / ncol, c = idx - r * ncol;
    if (bid >= 0) stage_col(sum, kFinT, ar.p[bid] + bbase + (i64)r * bld + c, ar.plane[bid], L);
    else
      for (int k = 0; k < L; k++) sum[k * kFinT] = 0u;
    int32_t* op = ar.p[oid] + obase + (i64)r * old_ + c;
    const i64 oplane = ar.plane[oid];
    // words b0 .. of source i: those from the rounding bit's word up to word q + L, and the top (sign) word last
    auto issue = [&](int i, int& s, int& b0) {
      const i64* si = d + 9 + 4 * i;
      s = clamp_shift(si[2] - (si[3] >= 0 ? xe[si[3]] : 0), W, L);
      const int q = s >> 5;
      b0 = q - 1 > 0 ? (q - 1 < W - 1 ? q - 1 : W - 1) : 0;
      const int e = q + L + 1 < W ? (q + L + 1 > b0 ? q + L + 1 : b0) : W;    // [b0, e)
      const int32_t* src = Wd + si[0] + (i64)r * w + c;
      u32* dst = buf + (i & 1) * (L + 3) * kFinT;
      stage_col(dst, kFinT, src + (i64)b0 * Ntot, Ntot, e - b0);
      cp_async4(dst + (L + 2) * kFinT, src + (i64)(W - 1) * Ntot, 4u);
    };
    int s0 = 0, b0 = 0, s1 = 0, b1 = 0;
    if (ns > 0) issue(0, s0, b0);
    cp_async_commit();
    for (int i = 0; i < ns; i++) {
      if (i + 1 < ns) issue(i + 1, s1, b1);
      cp_async_commit();
      cp_async_wait<1>();
      const u32* col = buf + (i & 1) * (L + 3) * kFinT;
      const u32 ext = (col[(L + 2) * kFinT] >> 31) ? 0xffffffffu : 0u;
      auto st = make_shr([&](int j) { return j < 0 ? 0u : (j >= W ? ext : col[(j - b0) * kFinT]); }, s0);
      const bool last = i + 1 == ns;
      const u32 flip = d[9 + 4 * i + 1] < 0 ? 0xffffffffu : 0u;      // subtract: add the complement and one
      u32 carry = flip & 1u;
#pragma unroll 4
      for (int k = 0; k < L; k++) {
        const u32 v = st.next(k) ^ flip, x = sum[k * kFinT];
        const u32 t = x + v, u = t + carry;
        carry = (t < x ? 1u : 0u) | (u < t ? 1u : 0u);
        if (last) op[(i64)k * oplane] = (int32_t)u;
        else sum[k * kFinT] = u;
      }
      s0 = s1;
      b0 = b1;
    }
    if (ns == 0) {
      cp_async_wait<0>();
      for (int k = 0; k < L; k++) op[(i64)k * oplane] = (int32_t)sum[k * kFinT];
    }
  }
}

// ---------------------------------------------------------------- triangular solves: fused 'col' rounding
// desc (10 int64): CRT row0, rows (32 nrt), column c0, ncols (<= 32), eA constant, eA index (-1 none, else +
// xe[idx]), B row tile (its column exponents), mode, base row tile 0, destination row tile 0.  For each column c,
// mx = max over the group's rows of the CRT bit length, s = mx - (32 L - 32), e_in = eA + Pe[B row tile][c],
// eU = e_in + s ('col' rounding, sdpvibe/batched.py:200-231); then every entry u = round(U / 2^s) goes to the
// destination row tiles dst0 .. dst0 + nrt - 1: mode 0 stores it (exponent eU), modes 1 / 2 form the aligned
// difference / sum with the base row tiles base0 .. (exponent eb): e2 = max(eb, eU) + 1, round(b / 2^(e2 - eb))
// -/+ round(u / 2^(e2 - eU)) (sdpvibe/batched.py:82-92).
// Columns are independent, so a group's columns are shared out over CTAs (grid y, kColSet = 8 each: one 32-byte
// sector per row and limb), which then hold one or two entries per thread for a few row tiles; an entry's words
// are staged in shared-memory columns.
constexpr int kColSet = 8;
__global__ void __launch_bounds__(256) grp_solve_round_kernel(const int32_t* __restrict__ Wd, const i64* __restrict__ bl,
                                                              int W, i64 Ntot, i64 w, int32_t* __restrict__ P,
                                                              i64 Pplane, i64* __restrict__ Pe, i64 m, int L,
                                                              const i64* __restrict__ xe,
                                                              const i64* __restrict__ desc) {
  extern __shared__ u32 cols[];
  __shared__ i64 s_part[32][kColSet];
  __shared__ i64 s_su[kColSet], s_eu[kColSet];
  const i64* d = desc + 10 * (i64)blockIdx.x;
  const int cfirst = blockIdx.y * kColSet;
  if (cfirst >= (int)d[3]) return;
  const i64 row0 = d[0], rows = d[1], c0 = d[2] + cfirst, brt0 = d[8], drt0 = d[9];
  const int ncols = (int)d[3] - cfirst < kColSet ? (int)d[3] - cfirst : kColSet, mode = (int)d[7];
  const int T = blockDim.x, tid = threadIdx.x, c = tid % kColSet, rg = tid / kColSet, nrg = T / kColSet;
  i64 mx = 0;
  if (c < ncols)
    for (i64 r = rg; r < rows; r += nrg) {
      const i64 v = bl[(row0 + r) * w + c0 + c];
      mx = v > mx ? v : mx;
    }
  s_part[rg][c] = mx;
  __syncthreads();
  if (tid < ncols) {
    i64 v = s_part[0][tid];
    for (int q = 1; q < nrg; q++) v = s_part[q][tid] > v ? s_part[q][tid] : v;
    const i64 s = v - (32 * (i64)L - 32);
    const i64 eA = d[4] + (d[5] >= 0 ? xe[d[5]] : 0);
    s_su[tid] = s;
    s_eu[tid] = eA + Pe[d[6] * m + c0 + tid] + s;
  }
  __syncthreads();
  const i64 nrt = rows / 32;
  u32* cu = cols + tid;                                  // L + 3 words of U, then L of b
  u32* cb = cu + (L + 3) * T;
  for (i64 idx = tid; idx < rows * ncols; idx += T) {
    const int cc = (int)(idx % ncols);
    const i64 rr = idx / ncols, t = rr / 32, r = rr % 32;
    const int32_t* u = Wd + (row0 + rr) * w + c0 + cc;
    int32_t* dst = P + (drt0 + t) * 32 * m + r * m + c0 + cc;
    const int su = clamp_shift(s_su[cc], W, L), q = su >> 5;
    const int b0 = q - 1 > 0 ? (q - 1 < W - 1 ? q - 1 : W - 1) : 0;
    const int e = q + L + 1 < W ? (q + L + 1 > b0 ? q + L + 1 : b0) : W;
    stage_col(cu, T, u + (i64)b0 * Ntot, Ntot, e - b0);
    cp_async4(cu + (L + 2) * T, u + (i64)(W - 1) * Ntot, 4u);
    if (mode) stage_col(cb, T, P + (brt0 + t) * 32 * m + r * m + c0 + cc, Pplane, L);
    cp_async_commit();
    const i64 eb = mode ? Pe[(brt0 + t) * m + c0 + cc] : 0, eu = s_eu[cc];
    cp_async_wait<0>();
    const u32 ext = (cu[(L + 2) * T] >> 31) ? 0xffffffffu : 0u;
    auto st = make_shr([&](int j) { return j < 0 ? 0u : (j >= W ? ext : cu[(j - b0) * T]); }, su);
    if (mode == 0) {
#pragma unroll 4
      for (int k = 0; k < L; k++) dst[(i64)k * Pplane] = (int32_t)st.next(k);
      continue;
    }
    // u in place of U: for su >= 0 word k is written after index q + k + 1 - b0 > k was read (b0 is q - 1, 0 below);
    // a left shift (nothing to round) reads at or below k, so it runs downward
    if (su >= 0) {
#pragma unroll 4
      for (int k = 0; k < L; k++) {
        const u32 v = st.next(k);
        cu[k * T] = v;
      }
    } else {
      for (int k = L - 1; k >= 0; k--) {
        const u32 v = __funnelshift_r(st.w(q + k), st.w(q + k + 1), su & 31);
        cu[k * T] = v;
      }
    }
    const i64 e2 = (eb > eu ? eb : eu) + 1;
    auto sb = make_shr(make_col(cb, T, L), clamp_shift(e2 - eb, L, L));
    auto sv = make_shr(make_col(cu, T, L), clamp_shift(e2 - eu, L, L));
    const u32 flip = mode == 1 ? 0xffffffffu : 0u;
    u32 carry = flip & 1u;
#pragma unroll 4
    for (int k = 0; k < L; k++) {
      const u32 x = sb.next(k), y = sv.next(k) ^ flip;
      const u32 a = x + y, o = a + carry;
      carry = (a < x ? 1u : 0u) | (o < a ? 1u : 0u);
      dst[(i64)k * Pplane] = (int32_t)o;
    }
  }
  __syncthreads();
  if (tid < ncols) {
    for (i64 t = 0; t < nrt; t++) {
      i64 e = s_eu[tid];
      if (mode) {
        const i64 eb = Pe[(brt0 + t) * m + c0 + tid];
        e = (eb > e ? eb : e) + 1;
      }
      Pe[(drt0 + t) * m + c0 + tid] = e;
    }
  }
}

// ---------------------------------------------------------------- triangular solves: common column exponents
// desc (4 int64): first row tile, row tiles, column c0, ncols (<= 32).  ee[c] = max over the row tiles of
// Pe[rt][c]; every entry is re-rounded to it (sdpvibe/batched.py:45-52) and Pe set to ee.  Columns shared out over
// CTAs as in grp_solve_round.
__global__ void __launch_bounds__(256) grp_merge_kernel(int32_t* __restrict__ P, i64 Pplane, i64* __restrict__ Pe,
                                                        i64 m, int L, const i64* __restrict__ desc) {
  extern __shared__ u32 cols[];
  __shared__ i64 s_ee[kColSet];
  const i64* d = desc + 4 * (i64)blockIdx.x;
  const int cfirst = blockIdx.y * kColSet;
  if (cfirst >= (int)d[3]) return;
  const i64 rt0 = d[0], nrt = d[1], c0 = d[2] + cfirst;
  const int ncols = (int)d[3] - cfirst < kColSet ? (int)d[3] - cfirst : kColSet;
  const int T = blockDim.x, tid = threadIdx.x;
  if (tid < ncols) {
    i64 ee = Pe[rt0 * m + c0 + tid];
    for (i64 t = 1; t < nrt; t++) {
      const i64 v = Pe[(rt0 + t) * m + c0 + tid];
      ee = v > ee ? v : ee;
    }
    s_ee[tid] = ee;
  }
  __syncthreads();
  u32* col = cols + tid;
  const i64 n = nrt * 32 * ncols;
  for (i64 idx = tid; idx < n; idx += T) {
    const int c = (int)(idx % ncols);
    const i64 rr = idx / ncols, t = rr / 32, r = rr % 32;
    const i64 s = s_ee[c] - Pe[(rt0 + t) * m + c0 + c];
    if (s == 0) continue;
    int32_t* x = P + (rt0 + t) * 32 * m + r * m + c0 + c;
    stage_col(col, T, x, Pplane, L);
    cp_async_commit();
    cp_async_wait<0>();
    auto st = make_shr(make_col(col, T, L), clamp_shift(s, L, L));
#pragma unroll 4
    for (int k = 0; k < L; k++) x[(i64)k * Pplane] = (int32_t)st.next(k);
  }
  __syncthreads();
  if (tid < ncols)
    for (i64 t = 0; t < nrt; t++) Pe[(rt0 + t) * m + c0 + tid] = s_ee[tid];
}

// ---------------------------------------------------------------- base-tile conversions
// Both work on 128 entries (4 rows) per CTA, eight CTAs per tile (grid y), with the wide, entry-major numbers passing
// through shared memory (an odd row length WL | 1: conflict free by entry) so that global memory sees whole runs.
constexpr int kTileT = 128;

// Diagonal tile (factor arena entry base fbase[t], exponent e) -> wide fixed point (WL words, exponent -F):
// the exact shift by e + F; entries above the diagonal are zero.  Out entry-major (tiles, 32, 32, WL).
__global__ void __launch_bounds__(kTileT) grp_tile_widen_kernel(const int32_t* __restrict__ Fa, i64 Fplane, int L,
                                                                i64 e, int WL, int LF, const i64* __restrict__ fbase,
                                                                u32* __restrict__ out) {
  extern __shared__ u32 cols[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, WP = WL | 1;
  const int idx = blockIdx.y * kTileT + tid, r = idx >> 5, c = idx & 31;
  u32* col = cols + tid;                               // L words; then the wide entries
  u32* wide = cols + L * kTileT;
  const i64 s = -32 * (i64)LF - e;
  u32* mine = wide + tid * WP;
  if (c <= r) {
    stage_col(col, kTileT, Fa + fbase[blockIdx.x] + idx, Fplane, L);
    cp_async_commit();
    cp_async_wait<0>();
    auto st = make_shr(make_col(col, kTileT, L), clamp_shift(s, L, WL));
#pragma unroll 4
    for (int k = 0; k < WL; k++) mine[k] = st.next(k);
  } else {
    for (int k = 0; k < WL; k++) mine[k] = 0u;
  }
  __syncthreads();
  u32* o = out + ((i64)blockIdx.x * 1024 + blockIdx.y * kTileT) * WL;
  for (int n = warp; n < kTileT; n += kTileT / 32)
    for (int k = lane; k < WL; k += 32) o[(i64)n * WL + k] = wide[n * WP + k];
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Factored tile (wide, exponent -F) -> the factor arena at exponent e (L limbs, zero above the diagonal);
// its inverse (wide) -> the inverse arena at xe = max bit length - F - (32 L - 32) over the tile (one exponent
// per tile, sdpvibe/batched.py:243-262): the eight CTAs of a tile form a cluster and exchange their maxima.
__global__ void __cluster_dims__(1, 8, 1) __launch_bounds__(kTileT)
    grp_tile_narrow_kernel(const u32* __restrict__ Lw, const u32* __restrict__ Xw, int WL, int LF,
                           int32_t* __restrict__ Fa, i64 Fplane, int L, i64 e, const i64* __restrict__ fbase,
                           int32_t* __restrict__ Xa, i64 Xplane, const i64* __restrict__ xidx, i64* __restrict__ xe) {
  extern __shared__ u32 cols[];
  __shared__ int s_max[kTileT / 32], s_all;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, WP = WL | 1;
  const int idx = blockIdx.y * kTileT + tid, r = idx >> 5, c = idx & 31;
  const i64 F = 32 * (i64)LF, first = ((i64)blockIdx.x * 1024 + blockIdx.y * kTileT) * WL;
  const i64 base = fbase[blockIdx.x], xi = xidx[blockIdx.x];
  u32 *wl = cols, *wx = cols + kTileT * WP;
  for (int n = warp; n < kTileT; n += kTileT / 32)
    for (int k = lane; k < WL; k += 32) {
      cp_async4(wx + n * WP + k, Xw + first + (i64)n * WL + k, 4u);
      cp_async4(wl + n * WP + k, Lw + first + (i64)n * WL + k, 4u);
    }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const u32 *myl = wl + tid * WP, *myx = wx + tid * WP;
  int mx = col_bits(myx, 1, WL);
  for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) s_max[warp] = mx;
  __syncthreads();
  if (tid == 0) s_all = max(max(s_max[0], s_max[1]), max(s_max[2], s_max[3]));
  cluster_sync();
  int tile_max = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    u32 addr;
    int v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&s_all)), "r"(k));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr));
    tile_max = max(tile_max, v);
  }
  cluster_sync();
  int32_t* fo = Fa + base + idx;
  if (c > r) {
    for (int k = 0; k < L; k++) fo[(i64)k * Fplane] = 0;
  } else {
    auto st = make_shr(make_col(myl, 1, WL), clamp_shift(e + F, WL, L));
#pragma unroll 4
    for (int k = 0; k < L; k++) fo[(i64)k * Fplane] = (int32_t)st.next(k);
  }
  const i64 ex = (i64)tile_max - F - (32 * (i64)L - 32);
  auto sx = make_shr(make_col(myx, 1, WL), clamp_shift(ex + F, WL, L));
  int32_t* xo = Xa + xi * 1024 + idx;
#pragma unroll 4
  for (int k = 0; k < L; k++) xo[(i64)k * Xplane] = (int32_t)sx.next(k);
  if (tid == 0 && blockIdx.y == 0) xe[xi] = ex;
}

// Dynamic shared memory of `bytes`, the kernel's limit raised to the most a CTA can have, once per device.
template <class Kernel>
int grp_smem(Kernel kernel, size_t bytes, bool (&set)[64]) {
  if (bytes > 220 * 1024) return SDPV_EINVAL;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return sdpv::set_cuda_error(e);
    set[dev & 63] = true;
  }
  return SDPV_OK;
}

Arenas make_arenas(int32_t* const* ptrs, const int64_t* planes, int n) {
  Arenas a{};
  for (int i = 0; i < kArenas; i++) {
    a.p[i] = i < n ? ptrs[i] : nullptr;
    a.plane[i] = i < n ? planes[i] : 0;
  }
  return a;
}

}  // namespace

extern "C" int sdpv_grp_copy(int32_t* const* src_host, const int64_t* src_planes_host, int nsrc, int32_t* dst,
                             int64_t dst_plane, int L, const int64_t* desc, int64_t ndesc, void* stream) {
  if (nsrc < 1 || nsrc > kArenas || !src_host || !src_planes_host || !dst || L < 1 || ndesc < 0 ||
      ndesc > 0x7fffffff || (ndesc && !desc))
    return SDPV_EINVAL;
  if (ndesc == 0) return SDPV_OK;
  const dim3 grid((unsigned)ndesc, (unsigned)(L < 65535 ? L : 65535));
  grp_copy_kernel<<<grid, 256, 0, sdpv::as_stream(stream)>>>(make_arenas(src_host, src_planes_host, nsrc), dst,
                                                              dst_plane, L, desc);
  return sdpv::launch_status();
}

extern "C" int sdpv_grp_finish_fixed(const int32_t* Wd, int W, int64_t Ntot, int64_t w, int32_t* const* ar_host,
                                     const int64_t* planes_host, int nar, int L, const int64_t* xe, const int64_t* desc,
                                     int64_t ndesc, void* stream) {
  if (!Wd || W < 1 || nar < 1 || nar > kArenas || !ar_host || !planes_host || L < 1 || ndesc < 0 ||
      ndesc > 0x7fffffff || (ndesc && !desc))
    return SDPV_EINVAL;
  if (ndesc == 0) return SDPV_OK;
  static bool set[64] = {};
  const size_t smem = (size_t)(L + 2 * (L + 3)) * kFinT * 4;
  const int rc = grp_smem(grp_finish_fixed_kernel, smem, set);
  if (rc != SDPV_OK) return rc;
  grp_finish_fixed_kernel<<<dim3((unsigned)ndesc, 8), kFinT, smem, sdpv::as_stream(stream)>>>(
      Wd, W, Ntot, w, make_arenas(ar_host, planes_host, nar), L, xe, desc);
  return sdpv::launch_status();
}

extern "C" int sdpv_grp_solve_round(const int32_t* Wd, const int64_t* bl, int W, int64_t Ntot, int64_t w, int32_t* P,
                                    int64_t Pplane, int64_t* Pe, int64_t m, int L, const int64_t* xe, const int64_t* desc,
                                    int64_t ndesc, void* stream) {
  if (!Wd || !bl || W < 1 || !P || !Pe || m < 1 || L < 1 || L > kLMax || ndesc < 0 || ndesc > 0x7fffffff ||
      (ndesc && !desc))
    return SDPV_EINVAL;
  if (ndesc == 0) return SDPV_OK;
  static bool set[64] = {};
  const int T = L <= 64 ? 256 : 128;
  const size_t smem = (size_t)(2 * L + 3) * T * 4;
  const int rc = grp_smem(grp_solve_round_kernel, smem, set);
  if (rc != SDPV_OK) return rc;
  const unsigned sets = (unsigned)(((m < 32 ? m : 32) + kColSet - 1) / kColSet);
  grp_solve_round_kernel<<<dim3((unsigned)ndesc, sets), T, smem, sdpv::as_stream(stream)>>>(Wd, bl, W, Ntot, w, P, Pplane,
                                                                                          Pe, m, L, xe, desc);
  return sdpv::launch_status();
}

extern "C" int sdpv_grp_merge(int32_t* P, int64_t Pplane, int64_t* Pe, int64_t m, int L, const int64_t* desc,
                              int64_t ndesc, void* stream) {
  if (!P || !Pe || m < 1 || L < 1 || ndesc < 0 || ndesc > 0x7fffffff || (ndesc && !desc)) return SDPV_EINVAL;
  if (ndesc == 0) return SDPV_OK;
  static bool set[64] = {};
  const int T = L <= 128 ? 256 : 128;
  const size_t smem = (size_t)L * T * 4;
  const int rc = grp_smem(grp_merge_kernel, smem, set);
  if (rc != SDPV_OK) return rc;
  const unsigned sets = (unsigned)(((m < 32 ? m : 32) + kColSet - 1) / kColSet);
  grp_merge_kernel<<<dim3((unsigned)ndesc, sets), T, smem, sdpv::as_stream(stream)>>>(P, Pplane, Pe, m, L, desc);
  return sdpv::launch_status();
}

extern "C" int sdpv_grp_tile_widen(const int32_t* Fa, int64_t Fplane, int L, int64_t e, int WL, int LF,
                                   const int64_t* fbase, int64_t ntiles, uint32_t* out, void* stream) {
  if (!Fa || !fbase || !out || L < 1 || WL <= L || LF < 2 || ntiles < 0 || ntiles > 0x7fffffff) return SDPV_EINVAL;
  if (ntiles == 0) return SDPV_OK;
  static bool set[64] = {};
  const size_t smem = (size_t)(L + (WL | 1)) * kTileT * 4;
  const int rc = grp_smem(grp_tile_widen_kernel, smem, set);
  if (rc != SDPV_OK) return rc;
  grp_tile_widen_kernel<<<dim3((unsigned)ntiles, 8), kTileT, smem, sdpv::as_stream(stream)>>>(Fa, Fplane, L, e, WL, LF,
                                                                                             fbase, out);
  return sdpv::launch_status();
}

extern "C" int sdpv_grp_tile_narrow(const uint32_t* Lw, const uint32_t* Xw, int WL, int LF, int32_t* Fa, int64_t Fplane,
                                    int L, int64_t e, const int64_t* fbase, int32_t* Xa, int64_t Xplane,
                                    const int64_t* xidx, int64_t* xe, int64_t ntiles, void* stream) {
  if (!Lw || !Xw || !Fa || !fbase || !Xa || !xidx || !xe || L < 1 || WL <= L || LF < 2 || ntiles < 0 ||
      ntiles > 0x7fffffff)
    return SDPV_EINVAL;
  if (ntiles == 0) return SDPV_OK;
  static bool set[64] = {};
  const size_t smem = (size_t)2 * (WL | 1) * kTileT * 4;
  const int rc = grp_smem(grp_tile_narrow_kernel, smem, set);
  if (rc != SDPV_OK) return rc;
  grp_tile_narrow_kernel<<<dim3((unsigned)ntiles, 8), kTileT, smem, sdpv::as_stream(stream)>>>(
      Lw, Xw, WL, LF, Fa, Fplane, L, e, fbase, Xa, Xplane, xidx, xe);
  return sdpv::launch_status();
}
