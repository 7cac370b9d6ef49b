// Uniform ring elements on the device, in the order and with the values of
// the reference's seeded commitment-key expansion.
//
// Reference path replaced: CommitKey::from_seed / generate_from_params /
// sample_uniform_mat (labrador/src/crs.rs:136-198, 308-326): the matrices A, B,
// C, D are ring elements drawn one after another from ChaCha20Rng(seed)
// (rand_chacha 0.10.0, Cargo.lock), every coefficient by PrimeField::rand
// (algebra/src/arith/prime.rs:730-743): a u64 sample s is accepted when
// s <= u64::MAX - ((u64::MAX % q + 1) % q) and maps to from_u64(s % q).
// The generator's u64 stream is the ChaCha20 keystream (64-bit block counter
// from 0, stream 0) read as consecutive little-endian word pairs, low word
// first (rand_core 0.10.1 block RNG).
//
// The sequence is sequential only through its rare rejections (probability
// below 2^-32 per sample for q < 2^32), so the device runs it as a compaction:
// every candidate is generated in parallel (one ChaCha20 block = 8 candidates
// per thread, 2048 per 256-thread segment). Pass 1 writes every candidate as if
// none before it had been rejected and counts each segment's rejections, pass 2 scans
// them, and pass 3 regenerates the segments that a rejection shifts (usually none) and
// writes accepted sample k to position k - (rejections before k). Candidates beyond
// the requested count are a margin for rejections; running out of it is
// reported (GRID_ERR_SAMPLE_EXHAUSTED through the plan's error word).
//
// The bound is the ALU pipe: 1280 cycles of a sub-partition per warp and block for
// ChaCha20, about 1400 with the reductions; 364544 polys of 64 coefficients are
// 0.11 ms of it. Measured there: 0.290 ms with a counting pass and a writing pass that
// both generated the keystream (and a scan of one segment word per thread and step),
// 0.134 ms now.
#include <cuda_runtime.h>

#include "grid_async.cuh"
#include "grid_chacha.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"

namespace grid {
namespace {

constexpr int kSegThreads = 256;
constexpr int kSegCands = kSegThreads * 8;  // candidates per segment

__device__ __forceinline__ void rng_block(const chacha::ChachaKey& key, unsigned long long blk,
                                          uint32_t (&w)[16]) {
  chacha::chacha20_block(key, (uint32_t)blk, (uint32_t)(blk >> 32), w);
}

__device__ __forceinline__ unsigned long long cand(const uint32_t (&w)[16], int c) {
  return (unsigned long long)w[2 * c] | ((unsigned long long)w[2 * c + 1] << 32);
}

// Exclusive prefix sum of v over the 256 threads of the CTA; *total gets the sum.
__device__ __forceinline__ unsigned cta_exclusive_scan(unsigned v, unsigned* total) {
  __shared__ unsigned warp_sums[kSegThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  unsigned before = 0, all = 0;
#pragma unroll
  for (int i = 0; i < kSegThreads / 32; ++i) {
    if (i < warp) before += warp_sums[i];
    all += warp_sums[i];
  }
  __syncthreads();  // warp_sums is reused by the next call
  *total = all;
  return before + x - v;
}

// from_u64(s % q) in Montgomery form, s = hi * 2^32 + lo: v = hi * (2^32 mod q) + lo is
// below q * 2^32, one reduction gives v * 2^-32 and one product by 2^96 * 2^-32 the word
// s * 2^32 mod q. r3 = 2^96 mod q with its companion r3 * q^-1 mod 2^32.
__device__ __forceinline__ uint32_t sample_word(uint32_t lo, uint32_t hi, const FieldParams& f,
                                                uint32_t r3, uint32_t r3q) {
  const uint64_t v = (uint64_t)hi * f.r1 + lo;
  const uint32_t m = (uint32_t)v * f.qinv;
  return mont_c(sub_lazy((uint32_t)(v >> 32), __umulhi(m, f.q), f.q), r3, r3q, f.q);
}

__global__ void __launch_bounds__(kSegThreads) crs_write_kernel(
    chacha::ChachaKey key, unsigned long long nseg, unsigned long long upper,
    unsigned long long count, uint32_t* __restrict__ out, FieldParams f, uint32_t r3, uint32_t r3q,
    unsigned* __restrict__ seg_rej, bool vec) {
  const uint32_t upper_hi = (uint32_t)(upper >> 32);
  const bool odd = threadIdx.x & 1;
  for (unsigned long long seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
    const unsigned long long blk = seg * kSegThreads + threadIdx.x;
    uint32_t w[16];
    rng_block(key, blk, w);
    bool rare = false;  // a candidate that may lie above the threshold
#pragma unroll
    for (int c = 0; c < 8; ++c) rare |= w[2 * c + 1] >= upper_hi;
    uint32_t x[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = sample_word(w[2 * c], w[2 * c + 1], f, r3, r3q);
    if (vec && (seg + 1) * kSegCands <= count) {
      // lanes of a pair write the even lane's 8 words, then the odd lane's: whole
      // sectors per store
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? x[i] : x[4 + i], 1);
        if (odd)
          x[i] = got;
        else
          x[4 + i] = got;
      }
      uint4* o = reinterpret_cast<uint4*>(out + (blk & ~1ull) * 8) + (odd ? 1 : 0);
      o[0] = make_uint4(x[0], x[1], x[2], x[3]);
      o[2] = make_uint4(x[4], x[5], x[6], x[7]);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (blk * 8 + c < count) out[blk * 8 + c] = x[c];
    }
    unsigned total = 0;
    if (__syncthreads_or(rare)) {
      unsigned rej = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) rej += cand(w, c) > upper ? 1u : 0u;
      cta_exclusive_scan(rej, &total);
    }
    if (threadIdx.x == 0) seg_rej[seg] = total;
  }
}

// One CTA: seg_off[s] = rejections in segments before s for s > 0, seg_off[0] = all of
// them (nothing precedes segment 0); short = whether the accepted candidates fall below
// `count`. Every thread takes a run of consecutive segments, so the loads of one
// step are independent.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) crs_scan_kernel(
    const unsigned* __restrict__ seg_rej, unsigned long long nseg, unsigned long long count,
    unsigned long long* __restrict__ seg_off, int* __restrict__ err) {
  __shared__ unsigned long long warp_sums[kScanThreads / 32];
  const unsigned long long per = (nseg + kScanThreads - 1) / kScanThreads;
  const unsigned long long beg = min(nseg, threadIdx.x * per), end = min(nseg, beg + per);
  unsigned long long own = 0;
#pragma unroll 8
  for (unsigned long long i = beg; i < end; ++i) own += seg_rej[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long x = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  unsigned long long before = 0, all = 0;
  for (int i = 0; i < kScanThreads / 32; ++i) {
    if (i < warp) before += warp_sums[i];
    all += warp_sums[i];
  }
  if (threadIdx.x == 0) {
    seg_off[0] = all;
    if (nseg * kSegCands - all < count) atomicExch(err, GRID_DEV_SAMPLE_SHORT);
  }
  if (all == 0) return;  // the shift pass reads no other offset
  unsigned long long run = before + x - own;
  for (unsigned long long i = beg; i < end; ++i) {
    if (i > 0) seg_off[i] = run;
    run += seg_rej[i];
  }
}

__global__ void __launch_bounds__(kSegThreads) crs_shift_kernel(
    chacha::ChachaKey key, unsigned long long nseg, unsigned long long upper,
    const unsigned* __restrict__ seg_rej, const unsigned long long* __restrict__ seg_off,
    unsigned long long count, uint32_t* __restrict__ out, FieldParams f, uint32_t r3,
    uint32_t r3q) {
  if (seg_off[0] == 0) return;  // no rejection at all
  for (unsigned long long seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
    const unsigned long long base = seg ? seg_off[seg] : 0;
    if (base == 0 && seg_rej[seg] == 0) continue;  // written in place already
    const unsigned long long blk = seg * kSegThreads + threadIdx.x;
    uint32_t w[16];
    rng_block(key, blk, w);
    unsigned rej = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) rej += cand(w, c) > upper ? 1u : 0u;
    unsigned total;
    unsigned long long before = base + cta_exclusive_scan(rej, &total);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (cand(w, c) > upper) {
        ++before;
        continue;
      }
      const unsigned long long dest = blk * 8 + c - before;
      if (dest < count) out[dest] = sample_word(w[2 * c], w[2 * c + 1], f, r3, r3q);
    }
  }
}

struct SampleGeometry {
  unsigned long long upper, nseg;
};

SampleGeometry sample_geometry(uint32_t q, unsigned long long count, unsigned long long accept_max) {
  SampleGeometry g;
  const unsigned long long reject = (~0ull % q + 1ull) % q;
  g.upper = accept_max ? accept_max : ~0ull - reject;
  // one spare segment covers the reference threshold's rejections (below 2^-32
  // per sample); a caller-chosen threshold gets a quarter more besides
  const unsigned long long cands = count + kSegCands + (accept_max ? count / 4 : 0);
  g.nseg = (cands + kSegCands - 1) / kSegCands;
  return g;
}

}  // namespace

size_t sample_uniform_workspace_bytes(uint32_t q, unsigned long long count,
                                      unsigned long long accept_max) {
  const SampleGeometry g = sample_geometry(q, count, accept_max);
  return ((g.nseg * 4 + 255) / 256) * 256 + g.nseg * 8;
}

int launch_sample_uniform(const grid_gpu_plan* p, const uint8_t seed[32], unsigned long long count,
                          unsigned long long accept_max, uint32_t* out, void* ws, size_t ws_bytes,
                          cudaStream_t s) {
  if (count == 0) return GRID_OK;
  const SampleGeometry g = sample_geometry(p->f.q, count, accept_max);
  if (ws_bytes < sample_uniform_workspace_bytes(p->f.q, count, accept_max))
    return GRID_ERR_INVALID_PARAMETERS;
  unsigned* seg_rej = static_cast<unsigned*>(ws);
  unsigned long long* seg_off = reinterpret_cast<unsigned long long*>(
      static_cast<char*>(ws) + ((g.nseg * 4 + 255) / 256) * 256);
  const chacha::ChachaKey key = chacha::make_key(seed);
  const uint32_t r3 = (uint32_t)(((unsigned __int128)1 << 96) % p->f.q);
  const uint32_t r3q = r3 * p->f.qinv;
  // one CTA per segment: the hardware balances them (a fixed share of segments per
  // CTA left a second, half-empty wave)
  const unsigned grid = (unsigned)(g.nseg < 0x7fffffffull ? g.nseg : 0x7fffffffull);
  const bool vec = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  crs_write_kernel<<<grid, kSegThreads, 0, s>>>(key, g.nseg, g.upper, count, out, p->f, r3, r3q,
                                                seg_rej, vec);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e);
  crs_scan_kernel<<<1, kScanThreads, 0, s>>>(seg_rej, g.nseg, count, seg_off, p->d_err);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  const unsigned long long cap = (unsigned long long)p->num_sms * 4;
  crs_shift_kernel<<<(unsigned)(g.nseg < cap ? g.nseg : cap), kSegThreads, 0, s>>>(
      key, g.nseg, g.upper, seg_rej, seg_off, count, out, p->f, r3, r3q);
  return cuda_status(cudaGetLastError());
}

}  // namespace grid
