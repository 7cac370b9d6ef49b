// ChaCha20 block function (RFC 8439) for device code: the JL keystream
// (IETF ChaCha20, nonce = part index) and the CRS sampler's ChaCha20Rng
// (64-bit block counter in words 12-13, stream 0 in words 14-15, which is the
// same block with the counter's high word in the nonce slot).
#pragma once
#include <stdint.h>

namespace grid {
namespace chacha {

// The key, and the state words 2, 6, 10, 14 and 3, 7, 11, 15 after the first round's
// quarter rounds on them: both streams keep words 14 and 15 zero, so those two of a
// block's 80 quarter rounds depend on the key alone.
struct ChachaKey {
  uint32_t k[8];
  uint32_t col2[4], col3[4];
};

inline ChachaKey make_key(const uint8_t seed[32]) {
  ChachaKey key;
  for (int i = 0; i < 8; ++i)
    key.k[i] = (uint32_t)seed[4 * i] | ((uint32_t)seed[4 * i + 1] << 8) |
               ((uint32_t)seed[4 * i + 2] << 16) | ((uint32_t)seed[4 * i + 3] << 24);
  auto rot = [](uint32_t x, int r) { return (x << r) | (x >> (32 - r)); };
  auto column = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t (&out)[4]) {
    uint32_t d = 0;
    a += b; d = rot(d ^ a, 16);
    c += d; b = rot(b ^ c, 12);
    a += b; d = rot(d ^ a, 8);
    c += d; b = rot(b ^ c, 7);
    out[0] = a; out[1] = b; out[2] = c; out[3] = d;
  };
  column(0x79622d32u, key.k[2], key.k[6], key.col2);
  column(0x6b206574u, key.k[3], key.k[7], key.col3);
  return key;
}

__device__ __forceinline__ uint32_t rotl(uint32_t x, int r) { return __funnelshift_l(x, x, r); }

__device__ __forceinline__ void quarter_round(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  a += b;
  d ^= a;
  d = rotl(d, 16);
  c += d;
  b ^= c;
  b = rotl(b, 12);
  a += b;
  d ^= a;
  d = rotl(d, 8);
  c += d;
  b ^= c;
  b = rotl(b, 7);
}

// RFC 8439 block function: out[16] = keystream words of block `counter`, nonce
// words (nonce0, 0, 0).
__device__ __forceinline__ void chacha20_block(const ChachaKey& key, uint32_t counter,
                                               uint32_t nonce0, uint32_t (&out)[16]) {
  uint32_t x0 = 0x61707865u, x1 = 0x3320646eu, x2 = key.col2[0], x3 = key.col3[0];
  uint32_t x4 = key.k[0], x5 = key.k[1], x6 = key.col2[1], x7 = key.col3[1];
  uint32_t x8 = key.k[4], x9 = key.k[5], x10 = key.col2[2], x11 = key.col3[2];
  uint32_t x12 = counter, x13 = nonce0, x14 = key.col2[3], x15 = key.col3[3];
  quarter_round(x0, x4, x8, x12);
  quarter_round(x1, x5, x9, x13);
  // second round of a pair, first round of the next; unrolled (a loop of one pair
  // measured 1360 cycles a block against 1280)
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    quarter_round(x0, x5, x10, x15);
    quarter_round(x1, x6, x11, x12);
    quarter_round(x2, x7, x8, x13);
    quarter_round(x3, x4, x9, x14);
    quarter_round(x0, x4, x8, x12);
    quarter_round(x1, x5, x9, x13);
    quarter_round(x2, x6, x10, x14);
    quarter_round(x3, x7, x11, x15);
  }
  quarter_round(x0, x5, x10, x15);
  quarter_round(x1, x6, x11, x12);
  quarter_round(x2, x7, x8, x13);
  quarter_round(x3, x4, x9, x14);
  out[0] = x0 + 0x61707865u; out[1] = x1 + 0x3320646eu;
  out[2] = x2 + 0x79622d32u; out[3] = x3 + 0x6b206574u;
  out[4] = x4 + key.k[0]; out[5] = x5 + key.k[1]; out[6] = x6 + key.k[2]; out[7] = x7 + key.k[3];
  out[8] = x8 + key.k[4]; out[9] = x9 + key.k[5]; out[10] = x10 + key.k[6];
  out[11] = x11 + key.k[7];
  out[12] = x12 + counter; out[13] = x13 + nonce0; out[14] = x14; out[15] = x15;
}

}  // namespace chacha
}  // namespace grid
