// Balanced (centered) base-b limbs of a coefficient, in 32-bit arithmetic
// (decompose_coeff_balanced / centered_mod, labrador/src/main_protocol/mod.rs:258-323).
//
// The canonical coefficient is centered into (-q/2, q/2]; its limbs are those of its
// magnitude a < 2^31 with the sign put back: with u = a mod b, the limb is u and the
// carry a / b where u <= b / 2, else u - b with the carry one larger. That equals the
// reference's truncating remainder rule, which is odd in its argument. (In 64-bit
// divisions, four limbs of the LaBRADOR round's Gram took 10.6 us by themselves.)
#pragma once
#include <stdint.h>

#include "grid_field.cuh"

namespace grid {

// Limbs of polynomials of d coefficients to out [poly][limb][d]; out null: none.
struct LimbSpec {
  uint32_t* out = nullptr;
  uint64_t base = 2;  // 2 .. 2^32
  uint32_t shift = 0; // log2(base) of a power of two, else 0
  int limbs = 0;
};

inline LimbSpec limb_spec(uint32_t* out, uint64_t base, size_t limbs) {
  LimbSpec l;
  l.out = out;
  l.base = base;
  l.limbs = (int)limbs;
  if ((base & (base - 1)) == 0)
    while ((1ull << l.shift) < base) ++l.shift;
  return l;
}

// One limb of magnitude a (sign `neg`) as a Montgomery word; a becomes the carry.
__device__ __forceinline__ uint32_t next_limb(uint32_t& a, bool neg, const LimbSpec& l,
                                              const FieldParams& f) {
  const uint32_t half = (uint32_t)(l.base >> 1);
  uint32_t u, carry;
  if (l.shift) {
    carry = l.shift < 32 ? a >> l.shift : 0u;
    u = l.shift < 32 ? a & ((1u << l.shift) - 1u) : a;
  } else {
    carry = a / (uint32_t)l.base;
    u = a - carry * (uint32_t)l.base;
  }
  if (u > half) {
    u = (uint32_t)l.base - u;
    ++carry;
    neg = !neg;
  }
  a = carry;
  const uint32_t w = mont_mul(u, f.r2, f.q, f.qinv);  // u < 2^32: u mod q in Montgomery form
  return neg && w ? f.q - w : w;
}

// The limbs of coefficients i .. i + 3 of a polynomial (Montgomery words x); dst: the
// polynomial's first limb at coefficient i, 16-byte aligned.
__device__ __forceinline__ void store_limbs4(uint4 x, uint32_t* dst, int d, const LimbSpec& l,
                                             const FieldParams& f) {
  uint32_t a[4] = {from_mont(x.x, f), from_mont(x.y, f), from_mont(x.z, f), from_mont(x.w, f)};
  bool neg[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    neg[j] = a[j] > f.q / 2;
    if (neg[j]) a[j] = f.q - a[j];
  }
  for (int k = 0; k < l.limbs; ++k, dst += d) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = next_limb(a[j], neg[j], l, f);
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace grid
