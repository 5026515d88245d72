// 64-bit LCG of HPL's matrix generator, shared by matgen and the fused
// residual.  X(n+1) = a X(n) + c mod 2^64 with a = 6364136223846793005,
// c = 1 (include/hpl_pmatgen.hpp:35-36).
#pragma once
#include <cstdint>

namespace hplb {

constexpr uint64_t kLcgMult = 6364136223846793005ull;
constexpr uint64_t kLcgAdd  = 1ull;

// Affine jump X -> a X + c.
struct Jump {
  uint64_t a, c;
};

// Apply x, then y.
__host__ __device__ inline Jump compose(Jump x, Jump y) {
  return Jump{y.a * x.a, y.a * x.c + y.c};
}

// Jump by k steps, by repeated squaring (the reference's HPL_xjumpm,
// src/matgen/HPL_xjumpm.cpp:81-91, loops k times; the constants are equal).
__host__ __device__ inline Jump jump_by(uint64_t k) {
  Jump acc{1, 0}, p{kLcgMult, kLcgAdd};
  while(k) {
    if(k & 1) acc = compose(acc, p);
    p = compose(p, p);
    k >>= 1;
  }
  return acc;
}

__host__ __device__ inline uint64_t apply(Jump j, uint64_t x) { return j.a * x + j.c; }

// Matrix entry from a state.  The reference adds the four 16-bit parts with
// power-of-two scales (src/matgen/HPL_pdrandmat_device.cpp:65-73); of its steps
// only two round: t = RN(hi + lo 2^-32) of the state's 32-bit halves (the sums
// before it have at most 48 bits) and RN(0.5 - t 2^-32).  Two fused multiply-
// adds round at the same places.  The halves become doubles by their bits
// (2^52 + v) - 2^52 instead of four integer conversions (hplb_matgen at
// N = 16384: 620 -> 533 us).
__device__ __forceinline__ double lcg_value(uint64_t r) {
  const double hi = __hiloint2double(0x43300000, (int)(uint32_t)(r >> 32)) - 0x1p52;
  const double lo = __hiloint2double(0x43300000, (int)(uint32_t)r) - 0x1p52;
  return __fma_rn(__fma_rn(lo, 0x1p-32, hi), -0x1p-32, 0.5);
}

}  // namespace hplb
