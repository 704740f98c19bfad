// Reduction of the CRT pre-pass, in plain C++ (the host compiles it too).
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
// is about 2^45.  One correction gives y in [0, m).
SDPV_HD uint32_t crt_reduce(uint32_t a, uint32_t inv, uint32_t m, uint32_t cm, uint32_t qb) {
  const uint32_t x = a * inv + cm - qb * m;
  return x + ((0u - (x >> 31)) & m);
}

}  // namespace sdpv
