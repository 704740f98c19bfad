// Entrywise multiprecision arithmetic on shared-memory columns.
//
// A thread keeps its entry's words in a column of shared memory (word k at c[k * kColThreads]: a warp's
// accesses at one k are 32 consecutive words, so any word offset is conflict free).  The words are brought in
// by 4-byte cp.async straight from the limb planes -- every load of the entry in flight at once -- and the
// result words leave in ascending order through one streaming pass (shift, rounding carry, sign).  Dynamic
// word offsets therefore cost one shared-memory access instead of a local-memory array.  Measured (B200), against
// the same operations on u32 arrays of the entry in local memory: product of 605160 entries at L = 26 291 -> 84
// us (2.4 TB/s of operands and result; the short product's multiply-adds and its 8 shared-memory reads per 16 of
// them are the larger part), sum of 150001 at L = 50 142 -> 37 us (2.5 TB/s; the passes of one CTA are in
// sequence and shared memory holds four CTAs of 128 such entries).  Wider numbers leave fewer CTAs per SM (one of
// products at 128 and 160 limbs) and still gain: 200000 entries at L = 64 / 100 / 160 products 611 -> 119, 2070 -> 280,
// 6941 -> 780 us, sums 326 -> 62, 594 -> 114, 1024 -> 229.
#pragma once
#include "common.cuh"

namespace sdpv {

constexpr int kColThreads = 128;
constexpr int T_ = kColThreads;

// Words [0, n) of one entry (plane stride `plane`) into the column; cp_async_wait afterwards.
__device__ __forceinline__ void col_stage(u32* c, const int32_t* __restrict__ src, i64 plane, int n) {
#pragma unroll 8
  for (int k = 0; k < n; k++, src += plane, c += T_) cp_async4(c, src, 4u);
}

// x - 1 in place (x != 0): with it |x| = ~(x - 1) for a negative x, so a column is read as a magnitude by
// XOR with the sign mask.  Usually one word.
__device__ __forceinline__ void col_dec(u32* c, int n) {
  for (int k = 0; k < n; k++, c += T_) {
    const u32 v = *c;
    *c = v - 1u;
    if (v) break;
  }
}

__device__ __forceinline__ bool col_is_zero(const u32* c, int n) {
  for (int k = n - 1; k >= 0; k--)
    if (c[k * T_]) return false;
  return true;
}

// bit length of the magnitude c ^ mask
__device__ __forceinline__ int col_bitlen(const u32* c, int n, u32 mask) {
  for (int k = n - 1; k >= 0; k--) {
    const u32 x = c[k * T_] ^ mask;
    if (x) return 32 * k + 32 - __clz(x);
  }
  return 0;
}

// Streaming output of round_half_up(mag / 2^s) (exact left shift for s <= 0), L words, negated if neg: the
// carries of the rounding and of the negation run along with the words (sdpvibe/mpf.py:36-56).
// w(i): magnitude word i, 0 outside the magnitude.
template <class Word>
__device__ __forceinline__ void col_emit(Word w, int s, int L, bool neg, int32_t* __restrict__ out, i64 plane) {
  const int q = s >> 5, r = s & 31;
  u32 c1 = s > 0 ? (w((s - 1) >> 5) >> ((s - 1) & 31)) & 1u : 0u;
  const u32 m = neg ? 0xffffffffu : 0u;
  u32 c2 = neg ? 1u : 0u;
  u32 lo = w(q);
#pragma unroll 4
  for (int k = 0; k < L; k++, out += plane) {
    const u32 hi = w(q + k + 1);
    const u32 f = __funnelshift_r(lo, hi, r);
    const u32 v = f + c1;
    c1 = v < f ? 1u : 0u;
    const u32 u = (v ^ m) + c2;
    c2 = u < c2 ? 1u : 0u;
    lo = hi;
    *out = (int32_t)u;
  }
}

__device__ __forceinline__ void put_zero(int32_t* __restrict__ out, i64 plane, i64* __restrict__ eo, int L) {
  for (int k = 0; k < L; k++) out[(i64)k * plane] = 0;
  *eo = SDPV_EZ;
}

// ---------------------------------------------------------------- product
// s += a b on a 96-bit column sum
__device__ __forceinline__ void mac96(u32 (&s)[3], u32 a, u32 b) {
  asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32 %2, %2, 0;"
      : "+r"(s[0]), "+r"(s[1]), "+r"(s[2])
      : "r"(a), "r"(b));
}
// carry a finished column (words 1, 2) into the next one
__device__ __forceinline__ void carry96(u32 (&s)[3], const u32 (&from)[3]) {
  asm("add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %2, %2, 0;"
      : "+r"(s[0]), "+r"(s[1]), "+r"(s[2])
      : "r"(from[1]), "r"(from[2]));
}

// Product of two magnitudes of 4 nb words (columns a, b) by output blocks of four words, kb = kstart ..
// 2 nb - 1: emit(kb, w) gets words 4 kb .. 4 kb + 3 in ascending order.  Blocks below kstart are left out, so
// the words come out low by less than kstart + 1 units of word 4 kstart + 4.
template <class Emit>
__device__ __forceinline__ void col_product(const u32* a, const u32* b, int nb, int kstart, Emit emit) {
  u32 s[7][3];
#pragma unroll
  for (int t = 0; t < 7; t++) s[t][0] = s[t][1] = s[t][2] = 0u;
  for (int kb = kstart; kb < 2 * nb; kb++) {
    const int i0 = kb - nb + 1 > 0 ? kb - nb + 1 : 0, i1 = kb < nb - 1 ? kb : nb - 1;
    const u32* pa = a + 4 * i0 * T_;
    const u32* pb = b + 4 * (kb - i0) * T_;
    for (int i = i0; i <= i1; i++, pa += 4 * T_, pb -= 4 * T_) {
      u32 x[4], y[4];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        x[t] = pa[t * T_];
        y[t] = pb[t * T_];
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) mac96(s[u + v], x[u], y[v]);
    }
    u32 w[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      w[t] = s[t][0];
      carry96(s[t + 1], s[t]);
    }
#pragma unroll
    for (int t = 0; t < 3; t++)
#pragma unroll
      for (int h = 0; h < 3; h++) s[t][h] = s[t + 4][h];
#pragma unroll
    for (int t = 3; t < 7; t++) s[t][0] = s[t][1] = s[t][2] = 0u;
    emit(kb, w);
  }
}

// the sign's magnitude form in place: padded column of n words (low pad words zero)
__device__ __forceinline__ void col_magnitude(u32* c, int n, bool neg) {
  if (!neg) return;
  col_dec(c, n);
#pragma unroll 4
  for (int k = 0; k < n; k++) c[k * T_] ^= 0xffffffffu;
}

// Any product (operands not normalised, or the short product's guard word undecided): the whole product
// twice, first for its bit length, then shifted, rounded and written as its words appear; nothing is stored.
// Rare, so it is kept out of line.
static __device__ __noinline__ int col_mul_general(const u32* a, const u32* b, int nb, int L, bool neg, int32_t* out,
                                            i64 plane) {
  int top = 0;
  col_product(a, b, nb, 0, [&](int kb, const u32 (&w)[4]) {
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (w[t]) top = 32 * (4 * kb + t) + 32 - __clz(w[t]);
  });
  const int s = top - (32 * L - 2), q = s >> 5, r = s & 31;
  const u32 m = neg ? 0xffffffffu : 0u;
  u32 c1 = 0, c2 = neg ? 1u : 0u, p1 = 0, p2 = 0;           // the last two words
  int k = 0;
  auto word = [&](u32 lo, u32 hi) {
    const u32 f = __funnelshift_r(lo, hi, r);
    const u32 v = f + c1;
    c1 = v < f ? 1u : 0u;
    const u32 u = (v ^ m) + c2;
    c2 = u < c2 ? 1u : 0u;
    if (k < L) out[(i64)k * plane] = (int32_t)u;
    k++;
  };
  for (int z = 0; z < -q - 1; z++) word(0u, 0u);            // left shifts by whole words
  auto next = [&](int i, u32 w) {                           // word i of the product
    if (i == q + 1 && s > 0) c1 = r ? (p1 >> (r - 1)) & 1u : p2 >> 31;
    if (i >= q + 1) word(p1, w);
    p2 = p1;
    p1 = w;
  };
  col_product(a, b, nb, 0, [&](int kb, const u32 (&w)[4]) {
#pragma unroll
    for (int t = 0; t < 4; t++) next(4 * kb + t, w[t]);
  });
  next(8 * nb, 0u);                                         // (L = 1: the result's only word is the top one)
  while (k < L) word(0u, 0u);
  return s;
}

// Operand of a sum already in shared memory (a column of the same thread): copied instead of staged.
struct ColSrc {
  const u32* c;
  __device__ __forceinline__ void operator()(u32* dst, int L) const {
    for (int k = 0; k < L; k++) dst[k * T_] = c[k * T_];
  }
};
// Operand in limb planes.
struct PlaneSrc {
  const int32_t* p;
  i64 plane;
  __device__ __forceinline__ void operator()(u32* dst, int L) const { col_stage(dst, p, plane, L); }
};

// r = a b of the entry whose operand words lie at A + k pa and B + k pb, written at O + k po -- limb planes, or a
// column of the thread with po = T_ -- (magnitude rounded half up to NB = 32L - 2 bits, zero -> EZ:
// sdpvibe/mpf.py:58-89).  col: 2 ceil4(L) words.
//
// Normalised operands (both magnitudes of exactly NB bits) take a short product: the result needs the product
// from its word LM + pad - 1 up (LM = ceil4(L), the operands shifted up by pad = LM - L words), so the 4 x 4
// word blocks below kstart are left out and word g = 4 kstart + 4 guards the rounding -- unless it lies within
// the bound of what was left out below 2^32, no carry can come out of it (28 of 49 blocks at L = 26).
__device__ __forceinline__ void col_mpf_mul(u32* col, const int32_t* __restrict__ A, i64 pa, i64 ea,
                                            const int32_t* __restrict__ B, i64 pb, i64 eb, int L,
                                            int32_t* __restrict__ O, i64 po, i64* __restrict__ eO) {
  const int LM = (L + 3) & ~3, pad = LM - L, nb = LM >> 2;
  u32 *ca = col, *cb = col + LM * T_;
  bool na, nbg;
  auto load = [&]() {
    for (int k = 0; k < pad; k++) ca[k * T_] = cb[k * T_] = 0u;
    col_stage(ca + pad * T_, A, pa, L);
    col_stage(cb + pad * T_, B, pb, L);
    cp_async_commit();
    cp_async_wait<0>();
    na = ca[(LM - 1) * T_] >> 31;
    nbg = cb[(LM - 1) * T_] >> 31;
    col_magnitude(ca, LM, na);
    col_magnitude(cb, LM, nbg);
  };
  load();
  const u32 ta = ca[(LM - 1) * T_], tb = cb[(LM - 1) * T_];
  if ((!ta && col_is_zero(ca, LM)) || (!tb && col_is_zero(cb, LM))) {
    put_zero(O, po, eO, L);
    return;
  }
  int s;
  bool done = false;
  if ((ta >> 29) == 1u && (tb >> 29) == 1u) {
    const int ks = (LM + pad - 10 >= 0) ? ((LM + pad - 10) >> 2) + 1 : 0;
    const int base = 4 * (nb - 1);                         // product word p is kept at column index p - base:
    col_product(ca, cb, nb, ks, [&](int kb, const u32 (&w)[4]) {   // block kb - (nb - 1) of a is no longer needed
      if (kb >= nb - 1) {
#pragma unroll
        for (int t = 0; t < 4; t++) ca[(4 * kb - base + t) * T_] = w[t];
      }
    });
    if (ks == 0 || ca[(4 * ks + 4 - base) * T_] < 0xffffff00u) {
      s = 64 * LM - __clz(ca[(2 * LM - 1 - base) * T_]) - (32 * L - 2);
      col_emit([&](int i) { return i < 2 * LM ? ca[(i - base) * T_] : 0u; }, s, L, na != nbg, O, po);
      done = true;
    } else {
      load();
    }
  }
  if (!done) s = col_mul_general(ca, cb, nb, L, na != nbg, O, po);
  *eO = ea + eb + (s - 64 * pad);
}

// ---------------------------------------------------------------- sum
// r = a + sgn b (operands aligned at max exponent - 32 in L + 2 words, each rounded half up, then the sum
// renormalised with its magnitude rounded half up: sdpvibe/mpf.py:92-124).  The two aligned operands are
// formed, signed and added word by word in one pass; the sum replaces a in its column.  col: 2 L + 2 words.
template <class SrcA, class SrcB>
__device__ __forceinline__ void col_mpf_add(u32* col, SrcA A, i64 ea, SrcB B, i64 eb, int sgn, int L, int32_t* O, i64 po,
                                            i64* eO) {
  u32 *ca = col, *cb = col + (L + 2) * T_;
  A(ca, L);
  B(cb, L);
  cp_async_commit();
  cp_async_wait<0>();
  const u32 ta = ca[(L - 1) * T_], tb = cb[(L - 1) * T_];
  const u32 ma = (ta >> 31) ? 0xffffffffu : 0u, mb = (tb >> 31) ? 0xffffffffu : 0u;
  const bool zb = (!tb && col_is_zero(cb, L)) || eb == SDPV_EZ;
  const bool za = (!ta && col_is_zero(ca, L)) || ea == SDPV_EZ;
  if (za && zb) {
    put_zero(O, po, eO, L);
    return;
  }
  if (za) ea = SDPV_EZ;
  if (zb) eb = SDPV_EZ;
  if (ma) col_dec(ca, L);
  if (mb) col_dec(cb, L);
  const int far = 32 * (L + 3);
  const i64 t = (ea > eb ? ea : eb) - 32;
  const i64 da = ea - t, db = eb - t;
  const int sa = (da < -(i64)far) ? far : (int)(-da);
  const int sb = (db < -(i64)far) ? far : (int)(-db);
  // an operand that counts as zero contributes zero words (nothing is read for it)
  const int la = za ? 0 : L, lb = zb ? 0 : L;
  auto wa = [&](int i) { return (unsigned)i < (unsigned)la ? ca[i * T_] ^ ma : 0u; };
  auto wb = [&](int i) { return (unsigned)i < (unsigned)lb ? cb[i * T_] ^ mb : 0u; };
  const int qa = sa >> 5, ra = sa & 31, qb = sb >> 5, rb = sb & 31;
  u32 c1a = sa > 0 ? (wa((sa - 1) >> 5) >> ((sa - 1) & 31)) & 1u : 0u;
  u32 c1b = sb > 0 ? (wb((sb - 1) >> 5) >> ((sb - 1) & 31)) & 1u : 0u;
  const u32 fb = sgn < 0 ? ~mb : mb;                        // sign of sgn b
  u32 c2a = ma & 1u, c2b = fb & 1u, c = 0;
  u32 alo = wa(qa), blo = wb(qb);
  u32 v = 0;
#pragma unroll 4
  for (int k = 0; k < L + 2; k++) {                         // the words read lie at or above k: a's q is >= -1
    const u32 ahi = wa(qa + k + 1), bhi = wb(qb + k + 1);
    const u32 fa = __funnelshift_r(alo, ahi, ra), va = fa + c1a;
    c1a = va < fa ? 1u : 0u;
    const u32 ua = (va ^ ma) + c2a;
    c2a = ua < c2a ? 1u : 0u;
    const u32 fbw = __funnelshift_r(blo, bhi, rb), vb = fbw + c1b;
    c1b = vb < fbw ? 1u : 0u;
    const u32 ub = (vb ^ fb) + c2b;
    c2b = ub < c2b ? 1u : 0u;
    alo = ahi;
    blo = bhi;
    const u32 sab = ua + ub;
    v = sab + c;
    c = (sab < ua ? 1u : 0u) | (v < sab ? 1u : 0u);
    ca[k * T_] = v;
  }
  const bool ns = v >> 31;
  const u32 ms = ns ? 0xffffffffu : 0u;
  if (ns) col_dec(ca, L + 2);
  const int bl = col_bitlen(ca, L + 2, ms);
  if (!bl) {
    put_zero(O, po, eO, L);
    return;
  }
  const int s = bl - (32 * L - 2);
  col_emit([&](int i) { return (unsigned)i < (unsigned)(L + 2) ? ca[i * T_] ^ ms : 0u; }, s, L, ns, O, po);
  *eO = t + s;
}

// ---------------------------------------------------------------- renormalisation
// LI words (in the column, two's complement) at exponent ei -> MPF of L words (sdpvibe/mpf.py:307-313).
__device__ __forceinline__ void col_mpf_norm(u32* col, int LI, i64 ei, int L, int32_t* __restrict__ O, i64 po,
                                             i64* __restrict__ eO) {
  const bool ng = col[(LI - 1) * T_] >> 31;
  const u32 m = ng ? 0xffffffffu : 0u;
  if (ng) col_dec(col, LI);
  const int bl = col_bitlen(col, LI, m);
  if (!bl) {
    put_zero(O, po, eO, L);
    return;
  }
  const int s = bl - (32 * L - 2);
  col_emit([&](int i) { return (unsigned)i < (unsigned)LI ? col[i * T_] ^ m : 0u; }, s, L, ng, O, po);
  *eO = ei + s;
}

}  // namespace sdpv
