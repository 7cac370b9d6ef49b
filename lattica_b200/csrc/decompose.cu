// Digit decompositions of R_q coefficients.
//
// Balanced (centered) base-b limbs: decompose_coeff_balanced / centered_mod /
// decompose_poly_balanced / decompose_polys
// (labrador/src/main_protocol/mod.rs:258-323, 731-747): the canonical
// coefficient is centered into (-q/2, q/2], then limb = centered_mod(carry, b)
// in [-b/2, b/2] and carry = (carry - limb) / b, num_limbs times (a carry left
// after the last limb is dropped, as in the reference). Limb v is stored as the
// Montgomery word of v mod q. Output layout [poly][limb][coeff].
//
// Unsigned gadget digits: gadget_decompose / GadgetRing::decompose_element
// (algebra/src/poly/decomposition.rs:47-61, commit/src/gadget/mod.rs:151-162):
// digit = value % base, value /= base, k = #digits(q - 1) times.
#include <cuda_runtime.h>

#include "balanced.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"

namespace grid {
namespace {

// kVec: four coefficients per thread (16-byte aligned buffers, d a multiple of 4).
template <bool kVec>
__global__ void balanced_kernel(const uint32_t* __restrict__ in, size_t npolys, uint32_t d,
                                LimbSpec l, FieldParams f) {
  constexpr int W = kVec ? 4 : 1;
  const size_t total = npolys * (size_t)d / W;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const uint32_t per_poly = d / W;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    const size_t poly = idx / per_poly;
    const uint32_t i = (uint32_t)(idx % per_poly) * W;
    uint32_t* dst = l.out + poly * (size_t)l.limbs * d + i;
    if constexpr (kVec) {
      store_limbs4(reinterpret_cast<const uint4*>(in)[idx], dst, (int)d, l, f);
    } else {
      uint32_t a = from_mont(in[idx], f);
      const bool neg = a > f.q / 2;
      if (neg) a = f.q - a;
      for (int k = 0; k < l.limbs; ++k, dst += d) *dst = next_limb(a, neg, l, f);
    }
  }
}

// digit_major = 1: out[digit][len] (gadget_decompose); 0: out[poly][digit][coeff]
// (decompose_element per polynomial, concatenated).
__global__ void gadget_kernel(const uint32_t* __restrict__ in, size_t len, int d,
                              unsigned long long base, int digits, int digit_major,
                              uint32_t* __restrict__ out, FieldParams f) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < len; idx += stride) {
    unsigned long long v = from_mont(in[idx], f);
    for (int k = 0; k < digits; ++k) {
      const uint32_t digit = (uint32_t)((v % base) % f.q);
      v /= base;
      const size_t o = digit_major ? (size_t)k * len + idx
                                   : ((idx / d) * (size_t)digits + k) * d + (idx % d);
      out[o] = to_mont(digit, f);
    }
  }
}

unsigned blocks_for(size_t n, int num_sms) {
  size_t b = (n + 255) / 256;
  const size_t cap = (size_t)num_sms * 16;
  if (b > cap) b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace

bool limbs_ok(uint64_t base, size_t num_limbs) {
  return base >= 2 && base <= (1ull << 32) && num_limbs > 0 && num_limbs <= 64;
}

int launch_decompose_balanced(const grid_gpu_plan* p, const uint32_t* polys, size_t npolys,
                              uint64_t base, size_t num_limbs, uint32_t* out, cudaStream_t s) {
  if (!limbs_ok(base, num_limbs)) return GRID_ERR_INVALID_PARAMETERS;
  if (npolys == 0) return GRID_OK;
  const LimbSpec l = limb_spec(out, base, num_limbs);
  const size_t words = npolys * p->d;
  if (((reinterpret_cast<uintptr_t>(polys) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0 &&
      p->d % 4 == 0)
    balanced_kernel<true><<<blocks_for(words / 4, p->num_sms), 256, 0, s>>>(polys, npolys, p->d, l,
                                                                            p->f);
  else
    balanced_kernel<false><<<blocks_for(words, p->num_sms), 256, 0, s>>>(polys, npolys, p->d, l,
                                                                         p->f);
  return cuda_status(cudaGetLastError());
}

int launch_gadget_decompose(const grid_gpu_plan* p, const uint32_t* x, size_t len, uint64_t base,
                            size_t digits, int digit_major, uint32_t* out, cudaStream_t s) {
  if (base < 2 || digits == 0) return GRID_ERR_INVALID_PARAMETERS;
  if (len == 0) return GRID_OK;
  gadget_kernel<<<blocks_for(len, p->num_sms), 256, 0, s>>>(x, len, (int)p->d, base, (int)digits,
                                                             digit_major, out, p->f);
  return cuda_status(cudaGetLastError());
}

size_t gadget_digit_count(uint64_t q, uint64_t base) {
  uint64_t m = q - 1;
  size_t digits = 0;
  while (m > 0) {
    ++digits;
    m /= base;
  }
  return digits ? digits : 1;
}

}  // namespace grid
