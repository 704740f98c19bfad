// Arithmetic of the CRT kernels in plain C++ (the host compiles it too).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SDPV_HD __host__ __device__ __forceinline__
#else
#define SDPV_HD inline
#endif

namespace sdpv {

// y = a inv mod m in [0, m) for the rounded quotient q of a inv / m, |a inv - q m| <= 0.502 m, given as the bits qb of
// the float 1.5 2^23 + q; cm = (bits of 1.5 2^23) m mod 2^32.  The products are taken modulo 2^32, hence unsigned: qb m
// is about 2^45.  One correction gives y in [0, m) (an arithmetic shift and a mask: as 0 - (x >> 31) the CRT of 400000 entries
// at 116 moduli took 128.5 instead of 125.8 us).
SDPV_HD uint32_t crt_reduce(uint32_t a, uint32_t inv, uint32_t m, uint32_t cm, uint32_t qb) {
  const uint32_t x = a * inv + cm - qb * m;
  return x + ((uint32_t)((int32_t)x >> 31) & m);
}

// Copies go round nslot slots in order, `loads` of them so far: the parity of the phase that the last copy into slot s
// completes, -1 if there was none.
SDPV_HD int last_load_parity(uint32_t loads, uint32_t nslot, uint32_t s) {
  return loads <= s ? -1 : (int)(((loads - 1 - s) / nslot) & 1u);
}

}  // namespace sdpv
