// The bits of the double a value widens to, in integer arithmetic, and what is hashed from them.
//
// GB300's FP64 pipe takes conversions at a small fraction of the integer rate, so kernels that only need a
// value's double to hash it or to take it apart build its bits with shifts.
#pragma once

#include "cql_internal.cuh"

// the double bits of a 32-bit float (exact: subnormals normalized, infinities and NaN kept)
__device__ __forceinline__ unsigned long long cql_f32_bits(uint32_t b)
{
  unsigned long long sign = (unsigned long long)(b >> 31) << 63;
  uint32_t e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
  if (e == 0xffu) return sign | 0x7ff0000000000000ull | ((unsigned long long)m << 29);
  if (e == 0)
  {
    if (m == 0) return sign;
    uint32_t shift = __clz(m) - 8;   // bring the leading one to bit 23
    m = (m << shift) & 0x7fffffu;
    return sign | ((unsigned long long)(1023 - 126 - shift) << 52) | ((unsigned long long)m << 29);
  }
  return sign | ((unsigned long long)(e - 127 + 1023) << 52) | ((unsigned long long)m << 29);
}

// the double bits of a whole number below 2^53 in magnitude (exact)
__device__ __forceinline__ unsigned long long cql_int_bits(long long v)
{
  if (v == 0) return 0;
  unsigned long long sign = v < 0 ? 0x8000000000000000ull : 0ull, a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  int p = 63 - __clzll(a);
  return sign | ((unsigned long long)(1023 + p) << 52) | ((a << (52 - p)) & 0xfffffffffffffull);
}

__device__ __forceinline__ uint32_t hash_u32(uint32_t x)
{
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// Where a value's HyperLogLog update lands (aggregate_reduce.comp:66-92): the register of its hash's top p
// bits, and rho, the place of the leading one in the rest.
__device__ __forceinline__ void cql_hll_place(unsigned long long bits, uint32_t p, uint32_t* bucket, uint32_t* rho)
{
  uint32_t h = hash_u32((uint32_t)bits ^ hash_u32((uint32_t)(bits >> 32)));
  uint32_t rest_bits = 32u - p;
  *bucket = h >> rest_bits;
  uint32_t rest = h & ((1u << rest_bits) - 1u);
  // findMSB: the index of the highest set bit, -1 for zero
  int msb = rest ? 31 - __clz(rest) : -1;
  *rho = msb < 0 ? rest_bits + 1u : rest_bits - (uint32_t)msb;
}
