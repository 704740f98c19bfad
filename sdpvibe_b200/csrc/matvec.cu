// C = A^T B for a long, wide A (K, M) and a few columns B (K, N): the residual products of the solver (B^T x).
//
// A residue product decomposes every entry of A into 2 n residue bytes to use each once: 637 of 1500 us for 7380 x
// 1000 by one column at L = 26, against 127 us that reading A takes.  Here A's entries meet the column directly on
// the tensor cores.  With numbers as signed base-256 digits (a + 0x8080..80 per byte, then each byte less 128),
//   c_i = sum_k a_ik x_k = sum_t 256^t sum_k sum_j a_ik[j] x_k[t - j],
// i.e. for every k a product of the 128 x 4L matrix of a block's digits with the Toeplitz matrix of x_k's digits.
// Both are int8 operands of tcgen05.mma, summed over k in int32 (|digits| <= 128: exact for 32000 / L values of k).
//   * mv_prep: Toeplitz operands.  Ordered by descending t, the 8-row x 16-byte core matrix at (row group 2h + p,
//     chunk c) depends on p and c + h only, so the operand is two runs of core matrices read with equal strides
//     in both directions (no swizzle): 5.4 KB per k at L = 26 instead of 28 KB, and nothing is expanded in shared
//     memory.
//   * mv_main: a CTA takes 128 columns of A and a range of k; three groups of 128 threads round rows k in turn to
//     their columns' exponents (one thread per entry, its limbs by cp.async) and write the operand tile, one thread
//     streams the Toeplitz operands (bulk copies) and issues the products; the int32 sums of the range go to
//     the workspace.
//   * mv_finish: sums over the ranges, carries, renormalisation (mpcol.cuh).
// The sums are exact, so the result is that of the residue product bit for bit.  7380 x 1000 by one column: 1503-1530 ->
// 376-426 us on several boxes (mv_main 319), by two (A rounded once for both) 494.  What bounds mv_main: the rounding's
// instructions and waits (251 us without it) over about 105 KB of shared-memory traffic per k (820 cycles).  Three groups
// of aligners with three rows of A staged each: two groups 381 us, four with two rows 321 (shared memory holds no more).
#include <cstring>

#include "common.cuh"
#include "mpcol.cuh"

namespace {
using namespace sdpv;

constexpr int kGroups = 3;                   // aligner groups of 128 threads, an operand tile each
constexpr int kRaw = 3;                      // rows of A staged per group: one rounded, the others in flight
constexpr int kFSlots = 8;                   // Toeplitz operands in flight, at most
constexpr int kRows = 128;                   // columns of A (rows of the product) per CTA
constexpr int kThreads = kGroups * 128 + 64; // aligners, a warp for the products, one for the Toeplitz operands
constexpr int kLmax = 32;                    // 4 L digits in one 128-byte operand row

struct MvShape {
  int ks, nh, nc;                            // K steps of 32 digits, row groups per parity, core matrices per run
};
__host__ __device__ inline MvShape mv_shape(int L) {
  MvShape s;
  s.ks = (4 * L + 31) / 32;
  s.nh = 2 * ((L + 3) / 4);                  // 16 nh >= 8 L digit sums, 8 nh a multiple of 16 (the MMA's N)
  s.nc = 2 * s.ks + s.nh - 1;
  return s;
}
__host__ __device__ inline i64 mv_image(int L) { return 2ll * mv_shape(L).nc * 128; }   // Toeplitz bytes per k

// v += c over four words (c: carry in and out)
__device__ __forceinline__ void add_carry4(u32 (&v)[4], u32& c) {
  asm("add.cc.u32 %0, %0, %4;\n\t"
      "addc.cc.u32 %1, %1, 0;\n\t"
      "addc.cc.u32 %2, %2, 0;\n\t"
      "addc.cc.u32 %3, %3, 0;\n\t"
      "addc.u32 %4, 0, 0;"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(c));
}
// v += 0x80808080 per word + c
__device__ __forceinline__ void add_bias4(u32 (&v)[4], u32& c) {
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %4, 0xffffffff;\n\t"
      "addc.cc.u32 %0, %0, 0x80808080;\n\t"
      "addc.cc.u32 %1, %1, 0x80808080;\n\t"
      "addc.cc.u32 %2, %2, 0x80808080;\n\t"
      "addc.cc.u32 %3, %3, 0x80808080;\n\t"
      "addc.u32 %4, 0, 0;\n\t}"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(c));
}

// Words of one entry rounded to shift s (half up, ties toward +infinity) as signed digits: words 4 c .. 4 c + 3 of
// (value + 0x80...80) ^ 0x80...80 (zeros past L) in ascending order; sets the overflow bit if the value does not fit.
// The entry's words at col[i stride], i < L; word L of the column is written with the sign extension, so that a
// right shift (the usual case: the reference exponent is at or above the entry's) reads it unconditionally.
template <class Out>
__device__ __forceinline__ void align_digits(u32* col, int stride, int L, i64 s64, Out out, unsigned* err) {
  const u32 ext = (col[(L - 1) * stride] >> 31) ? 0xffffffffu : 0u;
  col[L * stride] = ext;
  const i64 hi = 32 * (i64)(L + 1), lo = -32 * (i64)(L + 1);
  const int s = (int)(s64 > hi ? hi : (s64 < lo ? lo : s64));       // further shifts give the same words
  const int q = s >> 5, r = s & 31;
  u32 c1, c2 = 0, last = 0, a, top;
  auto block = [&](int k0, u32 (&v)[4]) {                            // four shifted words -> digits
    add_carry4(v, c1);
    const int rest = L - k0;
    last = rest >= 4 ? v[3] : (rest == 3 ? v[2] : (rest == 2 ? v[1] : v[0]));
    if (rest < 4) top = v[rest > 0 ? rest : 0];                      // the word above the result
    add_bias4(v, c2);
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = k0 + u < L ? v[u] ^ 0x80808080u : 0u;
    out(k0 >> 2, make_uint4(v[0], v[1], v[2], v[3]));
  };
  top = 0;
  if (s >= 0) {
    c1 = s > 0 ? (col[min((s - 1) >> 5, L) * stride] >> ((s - 1) & 31)) & 1u : 0u;
    a = col[min(q, L) * stride];
    for (int k0 = 0; k0 < L; k0 += 4) {
      u32 v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const u32 b = col[min(q + k0 + u + 1, L) * stride];
        v[u] = __funnelshift_r(a, b, r);
        a = b;
      }
      block(k0, v);
    }
    if ((L & 3) == 0) top = __funnelshift_r(a, col[min(q + L + 1, L) * stride], r) + c1;
  } else {                                                           // left shift: exact
    auto w = [&](int i) { return i < 0 ? 0u : col[min(i, L) * stride]; };
    c1 = 0;
    for (int k0 = 0; k0 < L; k0 += 4) {
      u32 v[4];
      for (int u = 0; u < 4; u++) v[u] = __funnelshift_r(w(q + k0 + u), w(q + k0 + u + 1), r);
      block(k0, v);
    }
    if ((L & 3) == 0) top = __funnelshift_r(w(q + L), w(q + L + 1), r);
  }
  if (top != ((last >> 31) ? 0xffffffffu : 0u)) atomicOr(err, SDPV_ERRBIT_OVERFLOW);
}

// ---------------------------------------------------------------- Toeplitz operands
// Image of (column n, k): core matrices [p][m], m < nc, of 8 rows r x 16 bytes b: digit (16 nh - 1) - 8 p - r - b - 16 m
// of the aligned entry (zero outside its 4 L digits).  32 entries per CTA.
constexpr int kPrep = 32, kZPad = 160;       // zero bytes around an entry's digits: indices -159 .. 16 nh - 1
__global__ void __launch_bounds__(128) mv_prep_kernel(const int32_t* __restrict__ B, const i64* __restrict__ eB, int L,
                                                      i64 K, i64 N, i64 ks, i64 ns, i64 n0,
                                                      const i64* __restrict__ Eb, uint8_t* __restrict__ F,
                                                      unsigned* err) {
  // entry (k, n) at k ks + n ns; plane stride K N; columns n0 + blockIdx.y
  extern __shared__ __align__(16) u32 sm[];
  const MvShape sh = mv_shape(L);
  const int tid = threadIdx.x;
  const i64 n = n0 + blockIdx.y, k0 = (i64)blockIdx.x * kPrep;
  const int zw = (2 * kZPad + 16 * sh.nh + 15) / 16 * 4 + 1;         // words per entry (odd pitch)
  u32* raw = sm;                                                     // [L + 1][32]
  u32* z = sm + (L + 1) * kPrep;                                           // [32][zw], digit d at byte kZPad + d
  for (int i = tid; i < kPrep * zw; i += 128) z[i] = 0u;
  __syncthreads();
  if (tid < kPrep && k0 + tid < K) {
    const i64 idx = (k0 + tid) * ks + n * ns;
    for (int l = 0; l < L; l++) cp_async4(raw + l * kPrep + tid, B + (i64)l * K * N + idx, 4u);
    cp_async_commit();
    const i64 ev = eB[idx];
    cp_async_wait<0>();
    u32* zo = z + tid * zw + kZPad / 4;
    align_digits(raw + tid, kPrep, L, ev == SDPV_EZ ? (1ll << 30) : Eb[n] - ev,
                 [&](int c4, uint4 v) {
                   zo[4 * c4] = v.x;
                   zo[4 * c4 + 1] = v.y;
                   zo[4 * c4 + 2] = v.z;
                   zo[4 * c4 + 3] = v.w;
                 },
                 err);
  }
  __syncthreads();
  const int per = 2 * sh.nc * 8;                                     // 16-byte rows of an image
  const i64 left = K - k0 < kPrep ? K - k0 : kPrep;
  uint4* out = reinterpret_cast<uint4*>(F + (blockIdx.y * K + k0) * mv_image(L));
  for (int i = tid; i < (int)left * per; i += 128) {
    const int e = i / per, j = i - e * per, r = j & 7, m = (j >> 3) % sh.nc, p = (j >> 3) / sh.nc;
    const int o = kZPad + 16 * sh.nh - 1 - 8 * p - r - 16 * m - 15;  // the 16 bytes o .. o + 15, reversed
    const u32* zs = z + e * zw + (o >> 2);
    const int sft = 8 * (o & 3);
    u32 w[4];
#pragma unroll
    for (int t = 0; t < 4; t++) w[t] = __byte_perm(__funnelshift_r(zs[t], zs[t + 1], sft), 0u, 0x0123);
    out[i] = make_uint4(w[3], w[2], w[1], w[0]);
  }
}

// ---------------------------------------------------------------- the products
struct MvSmem {
  uint8_t a[kGroups][kRows * 128];           // operand tiles (128-byte swizzle), 1024-aligned
  u64 full[kGroups], empty[kGroups], raw_full[kGroups][kRaw], ffull[kFSlots], fempty[kFSlots], done;
  u32 tmem_slot;
  volatile int abort;
};

// No-swizzle K-major descriptor: core matrices 128 bytes apart along K and along the rows.
__device__ __forceinline__ u64 sdesc_core128(u32 addr) {
  return (u64)((addr & 0x3FFFF) >> 4) | ((u64)(128 >> 4) << 16) | ((u64)(128 >> 4) << 32) | ((u64)1 << 46);
}

// A raw stage: L limb rows of 128 words, a row for the sign extension, 128 exponents.
__host__ __device__ inline int stage_words(int L) { return (L + 3) * 128; }

// The OR of pred over an aligner group (named barrier 1 + g): abort decisions are the group's.
__device__ __forceinline__ bool group_any(int g, bool pred) {
  u32 r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((u32)pred), "r"(1 + g)
      : "memory");
  return r != 0;
}

// NC columns of op(B) at once (1 or 2): A is rounded once for both.
// Dynamic shared memory: MvSmem, then [nf][NC] images, then per aligner group [kRaw] raw stages.  tma: the stages are filled
// by tensor copies of map_m (M, K, L) and map_e (2 M words, K): no thread has loads of its own outstanding when it
// fences its tile (with cp.async stages the fence waited for them: 406 us per column at 7380 x 1000).
template <int NC>
__global__ void __launch_bounds__(kThreads, 1)
    mv_main_kernel(const __grid_constant__ CUtensorMap map_m, const __grid_constant__ CUtensorMap map_e, int tma,
                   const int32_t* __restrict__ A, const i64* __restrict__ eA, int L, i64 K, i64 M,
                   const i64* __restrict__ Ea, const uint8_t* __restrict__ F, i64 kper, i64 Mp, int nf,
                   int32_t* __restrict__ part, i64 part_col, unsigned* err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  MvSmem& S = *reinterpret_cast<MvSmem*>((uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023));
  const MvShape sh = mv_shape(L);
  const u32 fbytes = (u32)mv_image(L);
  uint8_t* fsm = reinterpret_cast<uint8_t*>(&S) + ((sizeof(MvSmem) + 127) & ~(size_t)127);
  u32* raw = reinterpret_cast<u32*>(fsm + nf * NC * fbytes);
  const int tid = threadIdx.x, warp = tid >> 5;
  const i64 i0 = (i64)blockIdx.x * kRows, k0 = (i64)blockIdx.y * kper;
  const int steps = (int)(K - k0 < kper ? K - k0 : kper);

  if (tid == 0) {
    for (int s = 0; s < kGroups; s++) {
      mbar_init(&S.full[s], 128);
      mbar_init(&S.empty[s], 1);
      for (int r = 0; r < kRaw; r++) mbar_init(&S.raw_full[s][r], 1);
    }
    for (int s = 0; s < kFSlots; s++) {
      mbar_init(&S.ffull[s], 1);
      mbar_init(&S.fempty[s], 1);
    }
    mbar_init(&S.done, 1);
    S.abort = 0;
    mbar_fence_init();
  }
  if (warp == 4 * kGroups) {
    tmem_alloc(&S.tmem_slot, 256 * NC);
    tmem_relinquish();
  }
  for (int i = tid; i < kGroups * kRows * 128 / 16; i += kThreads)         // digits past 4 L stay zero
    reinterpret_cast<uint4*>(&S.a[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
  __syncthreads();
  tc_fence_after();
  const u32 tmem = S.tmem_slot;
  const int nn = 8 * sh.nh;                                          // columns per parity
  int loaded = 0;                                                    // the loading thread: images issued

  if (warp < 4 * kGroups) {
    // aligners: group g takes steps g, g + kGroups, ...; thread = row (column i of A)
    const int g = tid >> 7, row = tid & 127;
    const i64 i = i0 + row, plane = K * M;
    const bool in = i < M;
    const i64 target = in ? Ea[i] : 0;
    u32* stage = raw + (size_t)g * kRaw * stage_words(L);
    auto issue = [&](int n, int st) {                                // step n of the CTA into raw stage st
      if (n >= steps) {
        cp_async_commit();
        return;
      }
      u32* dst = stage + (size_t)st * stage_words(L);
      if (tma) {
        if (row == 0) {
          mbar_expect_tx(&S.raw_full[g][st], (u32)L * 512 + 1024);
          tma_load_3d(dst, &map_m, &S.raw_full[g][st], (int)i0, (int)(k0 + n), 0);
          tma_load_2d(dst + (L + 1) * 128, &map_e, &S.raw_full[g][st], (int)(2 * i0), (int)(k0 + n));
        }
        return;
      }
      const i64 idx = (k0 + n) * M + (in ? i : 0);
      const int32_t* src = A + idx;
      u32* d1 = dst + row;
      const u32 nb = in ? 4u : 0u;
#pragma unroll 8
      for (int l = 0; l < L; l++, src += plane, d1 += 128) cp_async4(d1, src, nb);
      const u32* es = reinterpret_cast<const u32*>(eA + idx);
      cp_async4(dst + (L + 1) * 128 + 2 * row, es, nb);
      cp_async4(dst + (L + 1) * 128 + 2 * row + 1, es + 1, nb);
      cp_async_commit();
    };
#pragma unroll
    for (int r = 0; r < kRaw - 1; r++) issue(g + r * kGroups, r);
    bool ok = true;
    int it = 0;
    for (int n = g; n < steps; n += kGroups, it++) {
      // this stage has landed; the one before it is no longer read by any thread
      const int st = it % kRaw;
      if (tma) ok = mbar_wait(&S.raw_full[g][st], (it / kRaw) & 1, err);
      else cp_async_wait<kRaw - 2>();
      if (group_any(g, !ok)) {
        S.abort = 1;
        break;
      }
      issue(n + (kRaw - 1) * kGroups, (it + kRaw - 1) % kRaw);
      u32* w = stage + (size_t)st * stage_words(L);
      const i64 e = in ? *reinterpret_cast<const i64*>(w + (L + 1) * 128 + 2 * row) : SDPV_EZ;
      // the products of this tile's previous step have read it
      if (it > 0) ok = mbar_wait(&S.empty[g], (it - 1) & 1, err);
      if (group_any(g, !ok || S.abort)) {
        S.abort = 1;
        break;
      }
      uint8_t* dst = &S.a[g][0];
      align_digits(w + row, 128, L, e == SDPV_EZ ? (1ll << 30) : target - e,
                   [&](int c4, uint4 v) { *reinterpret_cast<uint4*>(dst + sw128_off(row, c4)) = v; }, err);
      fence_proxy_async_smem();
      mbar_arrive(&S.full[g]);
    }
    cp_async_wait<0>();
    if (tma && row == 0 && S.abort)                                  // let copies in flight land (bounded)
      for (int r = it; r < it + kRaw && g + r * kGroups < steps; r++)
        mbar_wait(&S.raw_full[g][r % kRaw], (r / kRaw) & 1, err);
  } else if (tid == 128 * kGroups + 32) {
    // Toeplitz operands: image n into slot n mod nf once the products of step n - nf have read it
    const uint8_t* src = F + k0 * (i64)fbytes;
    int fs = 0, round = 0;
    for (int n = 0; n < steps && !S.abort; n++) {
      if (round > 0 && !mbar_wait(&S.fempty[fs], (round - 1) & 1, err)) {
        S.abort = 1;
        break;
      }
      mbar_expect_tx(&S.ffull[fs], NC * fbytes);
#pragma unroll
      for (int c = 0; c < NC; c++)                                   // column c's images follow K images later
        bulk_load(fsm + (fs * NC + c) * fbytes, src + ((i64)c * K + n) * fbytes, fbytes, &S.ffull[fs]);
      loaded = n + 1;
      if (++fs == nf) fs = 0, round++;
    }
  } else if (tid == 128 * kGroups) {
    // products: one thread, its instructions are the step's serial part (with the loads and their waits in the same
    // thread, and slots counted by divisions, it set the time: 480 us per column at 7380 x 1000)
    const u32 idesc = idesc_i8(kRows, nn);
    const u64 f0 = sdesc_core128(smem_u32(fsm)), fstep = (NC * fbytes) >> 4, fcol = fbytes >> 4;
    const u64 a0 = sdesc_sw128(smem_u32(&S.a[0][0]));
    const u64 par = (u64)sh.nc * 8;                                  // parity 1's core matrices, in 16-byte units
    int fs = 0, g = 0;
    u32 fphase = 0, aphase = 0;
    for (int n = 0; n < steps && !S.abort; n++) {
      if (!mbar_wait(&S.ffull[fs], fphase, err) || !mbar_wait(&S.full[g], aphase, err)) {
        S.abort = 1;
        break;
      }
      tc_fence_after();
      const u64 ad = a0 + (u64)g * (kRows * 128 / 16), bd = f0 + (u64)fs * fstep;
#pragma unroll
      for (int s = 0; s < 4; s++) {
        if (s >= sh.ks) break;
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
          for (int p = 0; p < 2; p++)
            mma_i8(tmem + c * 256 + p * nn, ad + 2 * s, bd + c * fcol + p * par + 16 * s, idesc, (n | s) ? 1u : 0u);
      }
      mma_commit(&S.empty[g]);
      mma_commit(&S.fempty[fs]);
      if (++fs == nf) fs = 0, fphase ^= 1;
      if (++g == kGroups) g = 0, aphase ^= 1;
    }
    mma_commit(&S.done);
    if (!mbar_wait(&S.done, 0, err)) S.abort = 1;
  }
  __syncthreads();
  // a wait gave up, perhaps after the last image was issued: let the images land before the CTA ends (bounded)
  if (S.abort)
    for (int j = loaded > nf ? loaded - nf : 0; j < loaded; j++) mbar_wait(&S.ffull[j % nf], (j / nf) & 1, err);
  tc_fence_after();
  if (warp < 4 && !S.abort && __all_sync(0xffffffffu, mbar_wait(&S.done, 0, err))) {
    tc_fence_after();
    // TMEM column p nn + 8 h + r = digit sum t = 16 nh - 1 - 16 h - 8 p - r; plane t of the range's sums, lanes = i
    for (int c = 0; c < NC; c++) {
      int32_t* out = part + c * part_col + (i64)blockIdx.y * 16 * sh.nh * Mp + i0 + (tid & 127);
      for (int c0 = 0; c0 < 2 * nn; c0 += 16) {
        u32 v[16];
        tmem_ld16(tmem + ((u32)(warp * 32) << 16) + c * 256 + c0, v);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 16; u++) {
          const int cc = c0 + u, p = cc >= nn ? 1 : 0, hr = cc - p * nn;
          const int t = 16 * sh.nh - 1 - 16 * (hr >> 3) - 8 * p - (hr & 7);
          out[(i64)t * Mp] = (int32_t)v[u];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4 * kGroups) tmem_dealloc(tmem, 256 * NC);
}

// ---------------------------------------------------------------- sums of the ranges, carries, renormalisation
// 8 entries of one column per CTA (grid y: columns): 128 threads per entry sum the ranges (a sector of 8 entries
// per plane), one carries and normalises.  part: [column][range][t][Mp].
constexpr int kFin = 8;
__global__ void __launch_bounds__(1024) mv_finish_kernel(const int32_t* __restrict__ part, i64 part_col, i64 Mp,
                                                         int nrange, int L, i64 M, i64 N, i64 n0,
                                                         const i64* __restrict__ Ea, const i64* __restrict__ Eb,
                                                         int32_t* __restrict__ O, i64* __restrict__ eO) {
  extern __shared__ i64 sums[];                                      // [T][kFin], then the word columns
  const int T = 16 * mv_shape(L).nh, e = threadIdx.x % kFin;
  const i64 i = (i64)blockIdx.x * kFin + e, n = n0 + blockIdx.y;
  part += blockIdx.y * part_col;
  for (int t = threadIdx.x / kFin; t < T; t += 1024 / kFin) {
    const int32_t* p = part + (i64)t * Mp + i;                       // (rows up to Mp >= M rounded to 128 exist)
    i64 s = 0;
#pragma unroll 16
    for (int q = 0; q < nrange; q++) s += (i64)__ldg(p + (i64)q * T * Mp);
    sums[t * kFin + e] = s;
  }
  __syncthreads();
  if (threadIdx.x >= kFin || i >= M) return;
  u32* col = reinterpret_cast<u32*>(sums + T * kFin) + e;            // words at stride kColThreads
  const int W = T / 4 + 2;
  i64 carry = 0;
#pragma unroll 4
  for (int w = 0; w < W; w++) {
    i64 v = carry;                                                   // |sums| < 2^38: no overflow
    if (4 * w < T)
#pragma unroll
      for (int u = 0; u < 4; u++) v += sums[(4 * w + u) * kFin + e] * (1ll << (8 * u));
    col[w * kColThreads] = (u32)v;
    carry = v >> 32;
  }
  const i64 o = i * N + n;
  col_mpf_norm(col, W, Ea[i] + Eb[n], L, O + o, M * N, eO + o);
}

i64 round_up(i64 a, i64 b) { return (a + b - 1) / b * b; }

// Ranges of k per block of columns, for nc columns at once.  A CTA fills an SM, so blocks * nrange CTAs run in rounds of
// one per SM; the time of a round's steps against that of a range's digit sums, written and read back, decides (us,
// fitted to 1 .. 296 ranges of twelve sizes at L = 6, 16, 26, 32).  One range per block left SMs idle from 75 blocks of
// columns on: 10000 x 1000 at L = 26 835 -> 604 us (5 ranges), four columns 2145 -> 1620.  No more values of k than int32
// sums hold.
void mv_split(int L, i64 K, i64 M, int nc, i64& kper, int& nrange) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const i64 blocks = (M + kRows - 1) / kRows, least = (K + 32000 / L - 1) / (32000 / L), most = (K + 15) / 16;
  const double step = 0.38 + 0.0155 * L + (nc - 1) * 0.012 * L, start = 3.0;
  const double sums = nc * (double)(blocks * kRows) * (9e-5 * mv_shape(L).nh + 2.3e-4);
  double best = 1e300;
  kper = K;
  nrange = 1;
  for (int rounds = 0; rounds <= 8; rounds++) {                      // the most ranges in so many rounds
    i64 r = rounds * (i64)sms / blocks;
    r = r > most ? most : r;
    r = r < least ? least : r;
    const i64 k = (K + r - 1) / r, n = (K + k - 1) / k;
    const double cost = (double)((blocks * n + sms - 1) / sms) * ((double)k * step + start) + sums * (double)n;
    if (cost < best) best = cost, kper = k, nrange = (int)n;
  }
}

// Columns whose Toeplitz images the workspace holds: all N where they take at most a quarter of A's bytes, else the two that
// are worked at once (5.4 KB per value of k and column at L = 26: four columns of 65536 x 128 would take more than A).
i64 image_columns(int L, i64 M, i64 N) { return N <= 2 || 4 * N * mv_image(L) <= M * (4 * L + 8) ? N : 2; }

}  // namespace

// Bytes of workspace of sdpv_gemm_tall (0: the shape is not taken).
extern "C" int sdpv_gemm_tall_workspace(int L, int64_t M, int64_t K, int64_t N, int64_t* bytes) {
  if (!bytes) return SDPV_EINVAL;
  *bytes = 0;
  if (L < 1 || L > kLmax || M < 1 || K < 1 || K > 65536 || N < 1 || N > 4) return SDPV_OK;
  i64 kper;
  int nrange;
  const int nc = N > 1 ? 2 : 1;                                        // columns worked at once
  mv_split(L, K, M, nc, kper, nrange);
  *bytes = round_up(image_columns(L, M, N) * K * mv_image(L), 256) + nc * (i64)nrange * 16 * mv_shape(L).nh * round_up(M, kRows) * 4;
  return SDPV_OK;
}

extern "C" int sdpv_gemm_tall(const int32_t* Am, const int64_t* Ae, const int32_t* Bm, const int64_t* Be, int L, int64_t M,
                              int64_t K, int64_t N, int transB, const int64_t* Ea, const int64_t* Eb, void* ws,
                              int64_t ws_bytes, int32_t* O, int64_t* eO, void* stream) {
  int64_t need = 0;
  sdpv_gemm_tall_workspace(L, M, K, N, &need);
  if (!need || ws_bytes < need || !ws || ((uintptr_t)ws & 255)) return SDPV_EINVAL;
  cudaStream_t st = sdpv::as_stream(stream);
  unsigned* err = sdpv::device_error_word();
  const MvShape sh = mv_shape(L);
  uint8_t* F = static_cast<uint8_t*>(ws);
  const i64 images = image_columns(L, M, N);
  int32_t* part = reinterpret_cast<int32_t*>(F + round_up(images * K * mv_image(L), 256));
  i64 kper;
  int nrange;
  mv_split(L, K, M, N > 1 ? 2 : 1, kper, nrange);
  const i64 Mp = round_up(M, kRows);
  const int zw = (2 * kZPad + 16 * sh.nh + 15) / 16 * 4 + 1;
  const size_t sm_prep = (size_t)(L + 1 + zw) * kPrep * 4;
  const size_t fixed = 1024 + ((sizeof(MvSmem) + 127) & ~(size_t)127) + (size_t)kGroups * kRaw * stage_words(L) * 4;
  auto slots = [&](int nc) {
    const i64 fit = (i64)(227 * 1024 - fixed) / (nc * mv_image(L));
    return (int)(fit < kFSlots ? fit : kFSlots);
  };
  auto sm_main = [&](int nc) { return fixed + (size_t)slots(nc) * nc * mv_image(L); };
  const size_t sm_fin = (size_t)16 * sh.nh * kFin * 8 + (size_t)(16 * sh.nh / 4 + 2) * kColThreads * 4;
  // tensor copies need 16-byte rows: M a multiple of 4 (and of 2 for the exponents)
  int tma = M % 4 == 0 && M < (1ll << 30) && (((uintptr_t)Am | (uintptr_t)Ae) & 15) == 0;
  CUtensorMap mm, me;
  memset(&mm, 0, sizeof(mm));
  memset(&me, 0, sizeof(me));
  if (tma) {
    sdpv::EncodeTiledFn fn = sdpv::encode_tiled_fn();
    cuuint64_t dm[3] = {(cuuint64_t)M, (cuuint64_t)K, (cuuint64_t)L}, sm_[2] = {(cuuint64_t)M * 4, (cuuint64_t)(K * M) * 4};
    cuuint32_t bm[3] = {128, 1, (cuuint32_t)L}, one[3] = {1, 1, 1};
    cuuint64_t de[2] = {(cuuint64_t)M * 2, (cuuint64_t)K}, se[1] = {(cuuint64_t)M * 8};
    cuuint32_t be[2] = {256, 1};
    tma = fn &&
          fn(&mm, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<int32_t*>(Am), dm, sm_, bm, one,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
          fn(&me, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<int64_t*>(Ae), de, se, be, one,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  const i64 part_col = (i64)nrange * 16 * sh.nh * Mp;
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(mv_main_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mv_main_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mv_finish_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e != cudaSuccess) return sdpv::set_cuda_error(e);
    set[dev & 63] = true;
  }
  const dim3 grid((unsigned)(Mp / kRows), (unsigned)nrange);
  for (i64 n = 0; n < N;) {
    const int nc = n + 1 < N ? 2 : 1;                                  // two columns at once
    if (n % images == 0)
      mv_prep_kernel<<<dim3((unsigned)((K + kPrep - 1) / kPrep), (unsigned)(images < N - n ? images : N - n)), 128, sm_prep,
                       st>>>(Bm, Be, L, K, N, transB ? 1 : N, transB ? K : 1, n, Eb, F, err);
    const uint8_t* Fn = F + n % images * K * mv_image(L);
    if (nc == 2)
      mv_main_kernel<2><<<grid, kThreads, sm_main(2), st>>>(mm, me, tma, Am, Ae, L, K, M, Ea, Fn, kper, Mp, slots(2), part,
                                                        part_col, err);
    else
      mv_main_kernel<1><<<grid, kThreads, sm_main(1), st>>>(mm, me, tma, Am, Ae, L, K, M, Ea, Fn, kper, Mp, slots(1), part,
                                                        part_col, err);
    mv_finish_kernel<<<dim3((unsigned)((M + kFin - 1) / kFin), (unsigned)nc), 1024, sm_fin, st>>>(
        part, part_col, Mp, nrange, L, M, N, n, Ea, Eb, O, eO);
    n += nc;
  }
  return sdpv::launch_status();
}
