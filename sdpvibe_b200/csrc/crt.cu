// CRT reconstruction fused with rounding.
//
// For an entry with residues a_i (n moduli m_i, M = prod m_i, |value| < M/4):
//   y_i = a_i (M/m_i)^-1 mod m_i in [0, m_i),  k = round(sum y_i / m_i),
//   value = sum_i y_i (M/m_i) - k M  (sdpvibe/rns.py:140-159, 227-245; sdpvibe/limbops.py:85-152).
// One CTA of 128 threads per tile of 128 entries (persistent over tiles):
//   * pre-pass (one thread per entry): y_i from the int16 accumulator, its digits y = 128 yh + yl as two
//     K-major byte rows in shared memory;
//   * digit contraction on the tensor cores: Z = [Yh Yl] C^T (tcgen05.mma kind::i8 on unsigned bytes, M = 128
//     entries, N = 128 digit rows per chunk, K = both digits of every modulus), C = the base-256 digits of 128
//     M/m_i and M/m_i, preceded by four rows that give sum y_i round(2^29 / m_i), i.e. k (ctx.cu).  All chunks
//     are issued back to back into TMEM (one column per digit) and waited for once;
//   * epilogue (the same thread, TMEM lane = entry): a word is z0 + 2^8 z1 + 2^16 z2 + 2^24 z3 + k N_w + carry
//     with N = 2^(32W) - M, all of it off the carry chain but one 64-bit add;
//   * crt_block streams the words out; crt_norm puts them in the thread's column of the tile that held Y (the
//     products are done with it) and renormalises from there (mpcol.cuh).
// No intermediate leaves the SM; one launch replaces crt_pre + digit GEMM + crt_carry + normalize.
//
// What bounds it: latency.  A one-tile CTA's four warps go through its phases one after the other (issue active in 21 %
// of the cycles with 235 tiles); four tiles on an SM wait for the residues' loads (49 %), the pre-pass's instructions
// (about 11 per residue) being the larger part of what is issued.  Both digits of y in one contraction halve the TMEM columns and take the
// digit recombination and k Md out of the epilogue.  Measured (B200, against two signed digit products in four
// waited-for chunks with the words in local memory): 1000 entries at 116 moduli 37 -> 15 us, crt_block of 1024 entries
// 22 -> 15 us; over 128 moduli, whose table passes through the SM once per tile, 160000 entries at L = 34 349 -> 144 us
// and at 58 603 -> 232.  Calls of at most two tiles per SM run as CTAs of one tile (two per SM up to 128 moduli, 102 KB
// each at 116); larger ones with at most 128 moduli take crt4_kernel below.
#include "common.cuh"
#include "crt_reduce.h"
#include "mpcol.cuh"

namespace {
using namespace sdpv;

constexpr int kThreads = kColThreads;       // = entries of a tile
constexpr int kDig = 128;                   // digit rows per chunk (N)
constexpr u32 kSlice = 128 * 128;
constexpr int kNmax = 256;                  // moduli: two 128-byte K tiles per digit plane
constexpr int kWmax = 128;                  // words
constexpr int kSlots = 4;                   // digit chunks (512 TMEM columns), and table slots, at most
constexpr size_t kHead = 6144;              // barriers, CrtMod[kNmax], N[kWmax]

struct CrtHead {
  u64 full[kSlots], empty[kSlots], done;
  u32 tmem_slot;
  int abort;
};

// Four digit columns as one word's contribution.  WIDE: z0 + 2^8 z1 may exceed 32 bits (z <= n 381 255, and
// 257 n 381 255 >= 2^32 from n = 173 on; taken from 169 on).
template <bool WIDE>
__device__ __forceinline__ u64 digit_word(const u32* z) {
  if (WIDE) return ((u64)z[0] + ((u64)z[1] << 8)) + ((((u64)z[2]) + ((u64)z[3] << 8)) << 16);
  return (u64)(z[1] * 256u + z[0]) + (u64)(z[3] * 256u + z[2]) * 65536ull;
}

// Residues v[q] of moduli gb + q -> y = residue inv mod m in [0, m), its digits into the entry's rows of Y.
__device__ __forceinline__ void store_digits(const CrtMod* TB, int gb, const int (&v)[32], int row, uint8_t* Yh,
                                             uint8_t* Yl) {
#pragma unroll
  for (int h = 0; h < 2; h++) {                        // 16 moduli per 16-byte chunk
    u32 ph[4], pl[4];
#pragma unroll
    for (int q4 = 0; q4 < 4; q4++) {
      u32 y[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int a = v[16 * h + 4 * q4 + u];
        const int4 c = *reinterpret_cast<const int4*>(&TB[gb + 16 * h + 4 * q4 + u]);
        // q = round(a inv / m) from the float product (off by less than 0.002)
        const float fa = __int_as_float(0x4B008000 + a) - 8421376.0f;
        const int qb = __float_as_int(fmaf(fa, __int_as_float(c.z), 12582912.0f));
        y[u] = crt_reduce((u32)a, (u32)c.y, (u32)c.x, (u32)c.w, (u32)qb);
      }
      const u32 p01 = y[0] + (y[1] << 16), p23 = y[2] + (y[3] << 16);
      ph[q4] = __byte_perm(p01 >> 7, p23 >> 7, 0x6420);
      pl[q4] = __byte_perm(p01, p23, 0x6420) & 0x7F7F7F7Fu;
    }
    const int g16 = gb + 16 * h, kt = g16 >> 7, chunk = (g16 & 127) >> 4;
    *reinterpret_cast<uint4*>(Yh + kt * kSlice + sw128_off(row, chunk)) = make_uint4(ph[0], ph[1], ph[2], ph[3]);
    *reinterpret_cast<uint4*>(Yl + kt * kSlice + sw128_off(row, chunk)) = make_uint4(pl[0], pl[1], pl[2], pl[3]);
  }
}

// Dynamic shared memory: [head] [Y: 2 ktc slices] [nslot chunk slots of 2 ktc slices].  The whole table stays
// resident where it fits (n <= 128); else its chunks pass through the slots, from L2, once per tile.
template <int MODE, bool WIDE>
__global__ void __launch_bounds__(kThreads, 2)
    crt_kernel(const int16_t* __restrict__ acc, i64 ldg, i64 N, i64 j0, i64 w, i64 rows, i64 rows_per_block,
               const int64_t* __restrict__ rowexp, const int64_t* __restrict__ colexp, int L, int n, int W, int ktc,
               int nchunk, int nslot, u32 tcols, const CrtMod* __restrict__ mods, const u32* __restrict__ negm,
               const uint8_t* __restrict__ ct, int32_t* __restrict__ out, int64_t* __restrict__ out2,
               const int32_t* __restrict__ pred, unsigned* __restrict__ err) {
  if (pred && *pred == 0) return;                      // predicated launch: nothing to do this time
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  CrtHead& H = *reinterpret_cast<CrtHead*>(base);
  CrtMod* TB = reinterpret_cast<CrtMod*>(base + 1024);
  u32* NM = reinterpret_cast<u32*>(base + 1024 + sizeof(CrtMod) * kNmax);
  const int tid = threadIdx.x, warp = tid >> 5;
  uint8_t* Yh = base + kHead;
  uint8_t* Yl = Yh + (size_t)ktc * kSlice;
  u32* col = reinterpret_cast<u32*>(Yh) + tid;         // this entry's word column, once Y is free
  const u32 cbytes = 2u * ktc * kSlice;                // one chunk of the table
  uint8_t* slots = Yh + cbytes;
  const i64 B = rows * w;
  const i64 ntiles = (B + 127) / 128;
  const bool resident = nslot >= nchunk;

  i64 tile = blockIdx.x;
  i64 e = tile * 128 + tid;
  bool valid = e < B;
  i64 r = valid ? e / w : 0, jj = valid ? e - r * w : 0;
  const int16_t* ap = acc + r * N + j0 + jj;
  // 32 residues at a time, the next 32 in flight while these are used (the first before any set-up)
  auto load = [&](int gb, int (&v)[32]) {
#pragma unroll
    for (int q = 0; q < 32; q++) v[q] = (valid && gb + q < n) ? (int)__ldcs(ap + (i64)(gb + q) * ldg) : 0;
  };
  int va[32], vb[32];
  load(0, va);

  if (tid == 0) {
    for (int s = 0; s < kSlots; s++) {
      mbar_init(&H.full[s], 1);
      mbar_init(&H.empty[s], 1);
    }
    mbar_init(&H.done, 1);
    H.abort = 0;
    mbar_fence_init();
    for (int s = 0; s < nslot; s++) {                  // nslot <= nchunk
      mbar_expect_tx(&H.full[s], cbytes);
      for (u32 o = 0; o < cbytes; o += kSlice) bulk_load(slots + s * cbytes + o, ct + (size_t)s * cbytes + o, kSlice, &H.full[s]);
    }
  }
  if (warp == 0) {
    tmem_alloc(&H.tmem_slot, tcols);
    tmem_relinquish();
  }
  for (int g = tid; g < 128 * ktc && g < kNmax; g += kThreads) TB[g] = mods[g];
  for (int k = tid; k < W; k += kThreads) NM[k] = negm[k];
  __syncthreads();
  tc_fence_after();
  const u32 tmem = H.tmem_slot;
  const u32 lane0 = (u32)(warp * 32) << 16;
  const u32 idesc = idesc_u8(128, kDig);
  const int ksteps = (n + 31) / 32;
  u32 seq = 0, phase = 0;                              // chunks used so far, parity of `done`
  u32 loads = nslot;                                   // thread 32: table copies issued

  while (true) {
    // ---- pre-pass: the digits of y_i
    auto digits = [&](int gb, const int (&v)[32]) { store_digits(TB, gb, v, tid, Yh, Yl); };
    for (int gb = 0; gb < n; gb += 64) {
      if (gb + 32 < n) load(gb + 32, vb);
      digits(gb, va);
      if (gb + 32 >= n) break;
      if (gb + 64 < n) load(gb + 64, va);
      digits(gb + 32, vb);
    }
    fence_proxy_async_smem();
    __syncthreads();

    // ---- digit products, carried into words
    u32 kq = 0, carry = 0;
    int hz = -1, ho = -1;                              // crt_block: highest word != 0, != 0xffffffff
    u32 hzv = 0, hov = 0, wtop = 0;
    if (tid == 0) {
      tc_fence_after();
      for (int c = 0; c < nchunk; c++, seq++) {
        const u32 s = resident ? (u32)c : seq % nslot;
        if (!mbar_wait(&H.full[s], resident ? 0u : (seq / nslot) & 1u, err)) {
          H.abort = 1;
          break;
        }
        const u32 tb = smem_u32(slots) + s * cbytes;
        for (int h = 0; h < 2; h++)
          for (int ks = 0; ks < ksteps; ks++) {
            const u32 o = (u32)(h * ktc + (ks >> 2)) * kSlice + (u32)(ks & 3) * 32;
            mma_i8(tmem + c * kDig, sdesc_sw128(smem_u32(Yh) + o), sdesc_sw128(tb + o), idesc, (h | ks) ? 1u : 0u);
          }
        if (!resident) mma_commit(&H.empty[s]);
      }
      mma_commit(&H.done);
    } else if (tid == 32 && !resident) {
      // refill each slot with the chunk nslot further in the sequence (it wraps over the tiles)
      for (int c = 0; c < nchunk; c++, seq++) {
        const u32 s = seq % nslot;
        if (!mbar_wait(&H.empty[s], (seq / nslot) & 1u, err)) {
          H.abort = 1;
          break;
        }
        const bool last = tile + gridDim.x >= ntiles;
        const u32 nx = (u32)c + nslot;        // < 2 nchunk
        if (nx >= (u32)nchunk && last) continue;
        loads = seq + nslot + 1;
        mbar_expect_tx(&H.full[s], cbytes);
        const uint8_t* src = ct + (size_t)(nx % nchunk) * cbytes;
        for (u32 o = 0; o < cbytes; o += kSlice) bulk_load(slots + s * cbytes + o, src + o, kSlice, &H.full[s]);
      }
    }
    __syncwarp();
    if (!mbar_wait(&H.done, phase, err)) H.abort = 1;
    phase ^= 1;
    tc_fence_after();
    const int ncol = 4 * (W + 1);
    u32 za[32], zb[32];
    auto words8 = [&](int c0, const u32 (&z)[32]) {  // digit columns c0 .. c0 + 31
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int wd = c0 / 4 + j - 1;
        if (wd >= W) break;
        u64 v = digit_word<WIDE>(z + 4 * j);
        if (j == 0 && wd < 0) {
          kq = (u32)((v + (1u << 28)) >> 29);
          continue;
        }
        v += (u64)kq * NM[wd];
        v += carry;
        const u32 wv = (u32)v;
        carry = (u32)(v >> 32);
        if (MODE == 0) {
          if (valid) out[(i64)wd * B + e] = (int32_t)wv;
          if (wv != 0u) hz = wd, hzv = wv;
          if (wv != 0xffffffffu) ho = wd, hov = wv;
          wtop = wv;
        } else {
          col[wd * kThreads] = wv;
        }
      }
    };
    tmem_ld32(tmem + lane0, za);
    for (int c0 = 0; c0 < ncol; c0 += 64) {          // the next 32 columns are read while these are carried
      tmem_ld_wait();
      if (c0 + 32 < ncol) tmem_ld32(tmem + lane0 + c0 + 32, zb);
      words8(c0, za);
      tmem_ld_wait();
      if (c0 + 32 >= ncol) break;
      if (c0 + 64 < ncol) tmem_ld32(tmem + lane0 + c0 + 64, za);
      words8(c0 + 32, zb);
    }
    tc_fence_before();

    // ---- outputs
    if (valid) {
      if (MODE == 0) {
        // bit length of v (v >= 0) or of ~v (v < 0): the highest word differing from the extension
        const bool ng = (wtop >> 31) != 0;
        const int k = ng ? ho : hz;
        const u32 x = ng ? ~hov : hzv;
        out2[e] = k < 0 ? 0 : 32 * (i64)k + 32 - __clz(x);
      } else {
        col_mpf_norm(col, W, rowexp[r] + colexp[(r / rows_per_block) * N + j0 + jj], L, out + e, B, out2 + e);
      }
    }
    tile += gridDim.x;
    if (tile >= ntiles) break;
    e = tile * 128 + tid;
    valid = e < B;
    r = valid ? e / w : 0;
    jj = valid ? e - r * w : 0;
    ap = acc + r * N + j0 + jj;
    load(0, va);
    __syncthreads();                                   // everyone is done with the columns over Y and with TMEM
    if (H.abort) break;
  }
  __syncthreads();
  if (H.abort && tid == 0) mbar_wait(&H.done, phase ^ 1u, err);   // a wait gave up: let products and copies drain (bounded)
  if (H.abort && tid == 32)
    for (int s = 0; s < nslot; s++) {
      const int p = last_load_parity(loads, nslot, s);
      if (p >= 0) mbar_wait(&H.full[s], (u32)p, err);
    }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, tcols);
}

// The same for calls of many tiles with n <= 128 (one or two digit chunks): kWide tiles at a time on an SM, each worked
// by its own four warps, which share one copy of the table.  TMEM then holds one chunk per tile, so the chunks run
// one after the other, the first one's words waiting in registers while the second's product still reads Y.
// Measured against two one-tile CTAs per SM (8 warps, latency-bound): 158760 entries at 116 moduli 68 -> 54 us
// (130 before the one contraction), 65536 at 104 30 -> 22, the 34 calls of a 600-block Cholesky and solve 5.8 -> 4.1 ms.
constexpr int kWide = 4;
struct Crt4Head {
  u64 full, done[kWide];
  u32 tmem_slot;
};
__device__ __forceinline__ void tile_sync(int grp) { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); }
// tile_sync with the OR of pred over the tile's threads: they give up together
__device__ __forceinline__ bool tile_sync_or(int grp, bool pred) {
  u32 r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((u32)pred), "r"(1 + grp)
      : "memory");
  return r != 0;
}

// Waits once more where the bounded wait gives up (the error bit is set): copies and products get that time to land before
// the CTA goes on or ends.  Inlined in MODE 0 and a call in MODE 1: the kernel uses all 128 registers, and the other way
// round the loop's schedule suffers (400000 entries at 116 moduli: 143 instead of 123 us, 112 instead of 110).
__device__ __noinline__ bool mbar_again(u64* bar, u32 phase, unsigned* err) { return mbar_wait(bar, phase, err); }
template <int MODE>
__device__ __forceinline__ bool mbar_drain(u64* bar, u32 phase, unsigned* err) {
  return mbar_wait(bar, phase, err) || (MODE == 0 ? mbar_wait(bar, phase, err) : mbar_again(bar, phase, err));
}

template <int MODE>
__global__ void __launch_bounds__(kThreads * kWide, 1)
    crt4_kernel(const int16_t* __restrict__ acc, i64 ldg, i64 N, i64 j0, i64 w, i64 rows, i64 rows_per_block,
                const int64_t* __restrict__ rowexp, const int64_t* __restrict__ colexp, int L, int n, int W, int nchunk,
                const CrtMod* __restrict__ mods, const u32* __restrict__ negm, const uint8_t* __restrict__ ct,
                int32_t* __restrict__ out, int64_t* __restrict__ out2, const int32_t* __restrict__ pred,
                unsigned* __restrict__ err) {
  if (pred && *pred == 0) return;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Crt4Head& H = *reinterpret_cast<Crt4Head*>(base);
  CrtMod* TB = reinterpret_cast<CrtMod*>(base + 1024);
  u32* NM = reinterpret_cast<u32*>(base + 1024 + sizeof(CrtMod) * kNmax);
  const int tid = threadIdx.x, warp = tid >> 5, grp = tid >> 7, lt = tid & 127;
  uint8_t* Yh = base + kHead + (size_t)grp * 2 * kSlice;
  uint8_t* Yl = Yh + kSlice;
  uint8_t* table = base + kHead + (size_t)kWide * 2 * kSlice;
  u32* col = reinterpret_cast<u32*>(Yh) + lt;
  const i64 B = rows * w, ntiles = (B + 127) / 128;

  if (tid == 0) {
    mbar_init(&H.full, 1);
    for (int g = 0; g < kWide; g++) mbar_init(&H.done[g], 1);
    mbar_fence_init();
    mbar_expect_tx(&H.full, (u32)nchunk * 2 * kSlice);
    for (u32 o = 0; o < (u32)nchunk * 2 * kSlice; o += kSlice) bulk_load(table + o, ct + o, kSlice, &H.full);
  }
  if (warp == 0) {
    tmem_alloc(&H.tmem_slot, 512);
    tmem_relinquish();
  }
  if (tid < 128) TB[tid] = mods[tid];
  for (int k = tid; k < W; k += kThreads * kWide) NM[k] = negm[k];
  __syncthreads();
  tc_fence_after();
  const u32 tmem = H.tmem_slot + (u32)grp * kDig;
  const u32 taddr = tmem + ((u32)((warp & 3) * 32) << 16);
  const u32 idesc = idesc_u8(128, kDig);
  const int ksteps = (n + 31) / 32;
  u32 phase = 0;
  bool ok = mbar_drain<MODE>(&H.full, 0, err);

  // tiles go round the CTAs first, so that a last partial round spreads over the SMs
  for (i64 tile = (i64)grp * gridDim.x + blockIdx.x; tile < ntiles; tile += (i64)kWide * gridDim.x) {
    const i64 e = tile * 128 + lt;
    const bool valid = e < B;
    const i64 r = valid ? e / w : 0, jj = valid ? e - r * w : 0;
    const int16_t* ap = acc + r * N + j0 + jj;
    for (int gb = 0; gb < n; gb += 32) {
      int v[32];
#pragma unroll
      for (int q = 0; q < 32; q++) v[q] = (valid && gb + q < n) ? (int)__ldcs(ap + (i64)(gb + q) * ldg) : 0;
      store_digits(TB, gb, v, lt, Yh, Yl);
    }
    fence_proxy_async_smem();
    tile_sync(grp);
    u32 kq = 0, carry = 0, hold[32];
    int hz = -1, ho = -1;
    u32 hzv = 0, hov = 0, wtop = 0;
    // word of four digit columns at word index wd (-1: the rows that give k); put(wd, word)
    auto word = [&](const u32* z, int wd, auto put) {
      u64 v = digit_word<false>(z);
      if (wd < 0) {
        kq = (u32)((v + (1u << 28)) >> 29);
        return;
      }
      v += (u64)kq * NM[wd];
      v += carry;
      carry = (u32)(v >> 32);
      put((u32)v);
    };
#pragma unroll
    for (int c = 0; c < 2; c++) {
      if (c >= nchunk) break;
      if (lt == 0) {
        tc_fence_after();
        const u32 tb = smem_u32(table) + (u32)c * 2 * kSlice, yb = smem_u32(Yh);
        for (int h = 0; h < 2; h++)
          for (int ks = 0; ks < ksteps; ks++) {
            const u32 o = (u32)h * kSlice + (u32)ks * 32;
            mma_i8(tmem, sdesc_sw128(yb + o), sdesc_sw128(tb + o), idesc, (h | ks) ? 1u : 0u);
          }
        mma_commit(&H.done[grp]);
      }
      __syncwarp();
      ok = mbar_drain<MODE>(&H.done[grp], phase, err) && ok;
      phase ^= 1;
      tc_fence_after();
      const bool last = c + 1 == nchunk;
      if (MODE == 1 && c == 1) {
#pragma unroll
        for (int k = 0; k < 31; k++) col[k * kThreads] = hold[k + 1];
      }
#pragma unroll
      for (int c0 = 0; c0 < kDig; c0 += 32) {
        if (c * kDig + c0 < 4 * (W + 1)) {
          u32 z[32];
          tmem_ld32(taddr + c0, z);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int wd = (c * kDig + c0) / 4 + j - 1;
            if (wd < W)
              word(z + 4 * j, wd, [&](u32 wv) {
                if (MODE == 0) {
                  if (valid) out[(i64)wd * B + e] = (int32_t)wv;
                  if (wv != 0u) hz = wd, hzv = wv;
                  if (wv != 0xffffffffu) ho = wd, hov = wv;
                  wtop = wv;
                } else if (last) {
                  col[wd * kThreads] = wv;
                } else {
                  hold[c0 / 4 + j] = wv;
                }
              });
          }
        }
      }
      tc_fence_before();
      if (!last) tile_sync(grp);                       // the next chunk's product overwrites the columns
    }
    if (valid) {
      if (MODE == 0) {
        const bool ng = (wtop >> 31) != 0;
        const int k = ng ? ho : hz;
        const u32 x = ng ? ~hov : hzv;
        out2[e] = k < 0 ? 0 : 32 * (i64)k + 32 - __clz(x);
      } else {
        col_mpf_norm(col, W, rowexp[r] + colexp[(r / rows_per_block) * N + j0 + jj], L, out + e, B, out2 + e);
      }
    }
    if (tile_sync_or(grp, !ok)) break;                 // (else) the columns over Y and TMEM are free again
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(H.tmem_slot, 512);
}

template <int MODE>
int launch_crt4(const sdpv_ctx* c, const int16_t* acc, i64 ldg, i64 N, i64 j0, i64 w, i64 rows, i64 rpb,
                const int64_t* rowexp, const int64_t* colexp, int L, int32_t* out, int64_t* out2, cudaStream_t st,
                const int32_t* pred, int sms) {
  const CtxDev& d = c->d;
  const int nchunk = d.Epad / kDig;
  const size_t smem = 1024 + kHead + (size_t)(kWide + nchunk) * 2 * kSlice;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(crt4_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return set_cuda_error(e);
    attr_set[dev & 63] = true;
  }
  crt4_kernel<MODE><<<(unsigned)sms, kThreads * kWide, smem, st>>>(acc, ldg, N, j0, w, rows, rpb, rowexp, colexp, L, d.n,
                                                                  d.W, nchunk, d.crtmod, d.negm, d.ct, out, out2, pred,
                                                                  device_error_word());
  return launch_status();
}

template <int MODE, bool WIDE>
int launch_crt_t(const sdpv_ctx* c, const int16_t* acc, i64 ldg, i64 N, i64 j0, i64 w, i64 rows, i64 rpb,
                 const int64_t* rowexp, const int64_t* colexp, int L, int32_t* out, int64_t* out2, cudaStream_t st,
                 const int32_t* pred) {
  const CtxDev& d = c->d;
  const int nchunk = d.Epad / kDig;
  const size_t chunk = (size_t)2 * d.ktc * kSlice, fixed = 1024 + kHead + chunk;      // Y is as large as a chunk
  int nslot = (int)((227 * 1024 - fixed) / chunk);      // 2 slots of 64 KB for ktc = 2
  if (nslot > nchunk) nslot = nchunk;
  u32 tcols = 128;
  while ((int)tcols < kDig * nchunk) tcols *= 2;
  // CTAs per SM: what shared memory holds (three with one digit chunk, two with two, one with two K tiles: never more
  // than TMEM's 512 columns serve), at most the tuned count.  With one K tile the calls have at most two tiles per SM.
  const size_t smem = fixed + nslot * chunk;
  int per_sm = (int)((228 * 1024) / (smem + 1024));
  const int tuned = sdpv::tune(SDPV_TUNE_CRT_CTAS);
  if (per_sm > tuned) per_sm = tuned;
  if (per_sm < 1) per_sm = 1;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(crt_kernel<MODE, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         227 * 1024);
    if (e != cudaSuccess) return set_cuda_error(e);
    attr_set[dev & 63] = true;
  }
  const i64 ntiles = (rows * w + 127) / 128;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  i64 gx = (i64)per_sm * sms;
  if (gx > ntiles) gx = ntiles;
  crt_kernel<MODE, WIDE><<<(unsigned)gx, kThreads, smem, st>>>(
      acc, ldg, N, j0, w, rows, rpb, rowexp, colexp, L, d.n, d.W, d.ktc, nchunk, nslot, tcols, d.crtmod, d.negm, d.ct,
      out, out2, pred, device_error_word());
  return launch_status();
}

template <int MODE>
int launch_crt(const sdpv_ctx* c, const int16_t* acc, i64 ldg, i64 N, i64 j0, i64 w, i64 rows, i64 rpb,
               const int64_t* rowexp, const int64_t* colexp, int L, int32_t* out, int64_t* out2, cudaStream_t st,
               const int32_t* pred = nullptr) {
  const CtxDev& d = c->d;
  // at most 256 moduli (L <= 59); there 4 + E <= 512 and a word column fits the 64 ktc words of an entry in Y
  if (d.n > kNmax || d.Epad > kSlots * kDig || d.W > kWmax || d.W > 64 * d.ktc) return SDPV_EINVAL;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // more tiles than one round of two per SM: four per SM on a shared table (where it fits: n <= 128)
  if (d.ktc == 1 && d.Epad <= 2 * kDig && d.W <= 64 && (rows * w + 127) / 128 > 2 * sms)
    return launch_crt4<MODE>(c, acc, ldg, N, j0, w, rows, rpb, rowexp, colexp, L, out, out2, st, pred, sms);
  if (d.n > 168)
    return launch_crt_t<MODE, true>(c, acc, ldg, N, j0, w, rows, rpb, rowexp, colexp, L, out, out2, st, pred);
  return launch_crt_t<MODE, false>(c, acc, ldg, N, j0, w, rows, rpb, rowexp, colexp, L, out, out2, st, pred);
}

}  // namespace

extern "C" int sdpv_crt_block(const sdpv_ctx* c, const int16_t* acc, int64_t ldg, int64_t N, int64_t j0, int64_t w,
                              int64_t rows, int32_t* words, int64_t* bitlen, void* stream) {
  if (!c || N < 0 || j0 < 0 || w < 0 || j0 + w > N || rows < 0 || c->d.W > 160) return SDPV_EINVAL;
  if (rows == 0 || w == 0) return SDPV_OK;
  return launch_crt<0>(c, acc, ldg, N, j0, w, rows, rows, nullptr, nullptr, c->d.L, words, bitlen,
                       sdpv::as_stream(stream));
}

extern "C" int sdpv_crt_norm(const sdpv_ctx* c, const int16_t* acc, int64_t ldg, int64_t N, int64_t j0, int64_t w,
                             int64_t rows, int64_t rows_per_block, const int64_t* rowexp, const int64_t* colexp, int L,
                             int32_t* O, int64_t* eO, void* stream) {
  if (!c || N < 0 || j0 < 0 || w < 0 || j0 + w > N || rows < 0 || rows_per_block < 1 || L < 1 || L > 160 ||
      c->d.W > 160)
    return SDPV_EINVAL;
  if (rows == 0 || w == 0) return SDPV_OK;
  return launch_crt<1>(c, acc, ldg, N, j0, w, rows, rows_per_block, rowexp, colexp, L, O, eO,
                       sdpv::as_stream(stream));
}

extern "C" int sdpv_crt_norm_if(const sdpv_ctx* c, const int16_t* acc, int64_t ldg, int64_t N, int64_t j0, int64_t w,
                                int64_t rows, int64_t rows_per_block, const int64_t* rowexp, const int64_t* colexp,
                                int L, int32_t* O, int64_t* eO, const int32_t* pred, void* stream) {
  if (!c || !pred || N < 0 || j0 < 0 || w < 0 || j0 + w > N || rows < 0 || rows_per_block < 1 || L < 1 || L > 160 ||
      c->d.W > 160)
    return SDPV_EINVAL;
  if (rows == 0 || w == 0) return SDPV_OK;
  return launch_crt<1>(c, acc, ldg, N, j0, w, rows, rows_per_block, rowexp, colexp, L, O, eO,
                       sdpv::as_stream(stream), pred);
}
