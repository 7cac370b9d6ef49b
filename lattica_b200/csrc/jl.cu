// Johnson-Lindenstrauss projection of the LaBRADOR prover on the GPU.
//
// Reference path replaced: JLMatrix::project_and_extract_jl_rows /
// project_and_extract_seq (labrador/src/jl.rs:267-303, 388-508). Part i of the
// witness uses the IETF ChaCha20 keystream (RFC 8439; the reference uses the
// chacha20 0.10 crate) with key = seed, nonce = (u32 i, little endian) || 0^8,
// block counter from 0. Column `col` consumes packed_len = ceil(rows/4) bytes
// at keystream offset col*packed_len; row r reads bits 2*(r%4) of byte r/4:
// 00 -> +1, 01 -> -1, 1x -> 0. p[row] = sum over parts and columns of
// entry * coeff (mod q), accumulated on Montgomery words (the map to
// Montgomery form is additive, so this is the reference's field sum).
//
// The keystream is regenerated on the fly (the reference materialises the
// whole [rows][parts][d][n] i8 matrix, 2 GiB at the LaBRADOR round size);
// the i8 extraction is a separate, optional kernel.
#include <cuda_runtime.h>

#include <algorithm>

#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_chacha.cuh"
#include "grid_tc.cuh"
#include "jl_units.h"

namespace grid {
namespace {

using chacha::ChachaKey;
using chacha::chacha20_block;

constexpr int kJlWarps = 8;  // jl_flat_kernel
constexpr int kJlThreads = kJlWarps * 32;

// Keystream bytes [off, off + 64) of stream (key, nonce0) as 16 words
// (unused tail bytes are whatever the next block holds; callers mask rows).
__device__ __forceinline__ void keystream64(const ChachaKey& key, uint32_t nonce0, uint64_t off,
                                            uint32_t (&w)[16]) {
  const uint32_t blk = (uint32_t)(off >> 6);
  const uint32_t sh = (uint32_t)(off & 63);
  chacha20_block(key, blk, nonce0, w);
  if (sh != 0) {
    uint32_t nx[16];
    chacha20_block(key, blk + 1, nonce0, nx);
    // byte-shift the 128-byte window (w ++ nx) left by sh bytes
    const uint32_t ws = sh >> 2, bs = (sh & 3) * 8;
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t j = i + ws;
      const uint32_t lo = j < 16 ? w[j] : nx[j - 16];
      const uint32_t j2 = j + 1;
      const uint32_t hi = j2 < 16 ? w[j2] : (j2 < 32 ? nx[j2 - 16] : 0u);
      r[i] = bs ? __funnelshift_r(lo, hi, bs) : lo;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = r[i];
  }
}

// Keystream bytes [off, off + len), len <= 64, in a loop over one or two blocks, the second
// only where the bytes reach into it. With both written out, always, the projection of
// 64 x 65536 columns took 524 us for 128 rows and 656 for 200, 228 and 382 so, and
// 16 x 32768 columns of 4 rows 85 us (79 with more CTAs per SM), 40 so. In jl_flat_kernel
// the stores lose more than the keystream gains (64 x 153600 columns of 200 rows 2.5 ms
// there, 3.6 so): it keeps keystream64.
__device__ __forceinline__ void keystream_bytes(const ChachaKey& key, uint32_t nonce0,
                                                uint64_t off, int len, uint32_t (&w)[16]) {
  const uint32_t blk = (uint32_t)(off >> 6);
  const uint32_t sh = (uint32_t)(off & 63);
  const int blocks = sh + (uint32_t)len > 64 ? 2 : 1;
  uint32_t buf[32] = {};  // in local memory: shifted by a variable number of bytes
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    uint32_t o[16];
    chacha20_block(key, blk + b, nonce0, o);
#pragma unroll
    for (int i = 0; i < 16; ++i) buf[16 * b + i] = o[i];
  }
  const uint32_t ws = sh >> 2, bs = (sh & 3) * 8;
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = __funnelshift_r(buf[i + ws], buf[i + ws + 1], bs);
}

// ---------------------------------------------------------------------------
// Tensor-core projection. A producer warp takes a unit of 32 columns of one
// part: lane l computes the keystream of its column and writes the column's 256
// entries, shifted to M' = M + 1 in {0, 1, 2}, into an MN-major u8 A tile (rows
// contiguous), and the column's word as a zero-padded 16-byte column of an
// MN-major u8 B tile (bytes = N). Two u8 MMAs (128-row halves, K = 32) per unit
// accumulate D[r][i] = sum_c M'[r][c] * byte_i(x_c) in tensor memory across all
// of the CTA's units; then p_r = sum_i 2^(8i) (D[r][i] - sum_c byte_i(x_c)).
//
// The bound is the ALU pipe: a ChaCha20 block is 80 quarter rounds of 8 XORs
// and rotations, 1280 cycles of one sub-partition per warp (its additions run
// beside them: measured 1279-1301 cycles with none, half or all of them on the
// FMA pipe), so 0.29 ms for the LaBRADOR round's 8.4 M columns. Everything else
// is kept small against that:
//  * Entries are unpacked without a table. Bit by bit M' is (h, ~h & ~l) for a
//    code (h, l), a shift and two logic operations for the 16 entries of a word;
//    three masks then leave entry 4j + s of byte j in place, scaled by 4^s, and
//    the packed word itself serves for s = 0 (it holds e_0 + 4 e_1 + 16 e_2 +
//    64 e_3 per byte: the other three sums, subtracted at the end, leave e_0's).
//    A tile row 16 g + 4 s + j is therefore matrix row 16 g + 4 j + s, 4^s times
//    its entry. (Table lookups: 64 a column, each conflicting over the 32 lanes.)
//  * Every producer warp owns its A and B tile and hands it to the MMA warp
//    through two mbarriers, so no barrier holds the CTA's warps together: one
//    CTA of 20 producer warps per SM, where three CTAs of 8 met at two CTA
//    barriers per chunk of 256 columns.
// Measured at 64 x 131072 columns: 0.51 ms before, 0.42 ms now; with the int8 entries
// 1.21 ms before, 0.90 ms now.
// ---------------------------------------------------------------------------
constexpr uint32_t kUnitA = 256u * kUnitCols;           // A tile: 256 rows x 32 columns
constexpr uint32_t kPjB = 16u * kUnitCols;              // B tile: 16 bytes x 32 columns
constexpr int kGroup = 4;                               // warps per hand-over (mma_loop)
// The plain projection runs 20 producer warps (0.416 ms at 64 x 131072 columns with 16
// or 20, 0.421 with 24, 0.438 with 12). With the int8 entries it runs 12: the scattered
// 32-byte sector stores of more warps get in each other's way (0.90 ms with 12, 0.95
// with 8, 1.2 with 16, 1.6 with 20).
template <bool kFlat>
struct PjShape {
  static constexpr int WARPS = kFlat ? 12 : 20;         // producer warps
  static constexpr int THREADS = (WARPS + 1) * 32;      // + the MMA warp
  static constexpr uint32_t OFF_B = WARPS * kUnitA;
  static constexpr uint32_t OFF_BAR = OFF_B + WARPS * kPjB;
  static constexpr uint32_t SMEM =
      OFF_BAR + (2 * WARPS / kGroup + 1) * 8 + 32 + 128;  // + alignment slack
  static_assert(SMEM <= 232448 && WARPS % kGroup == 0, "shape");
};

// Row m, column k of a unit's A tile: 16-row x 8-column core matrices.
__device__ __forceinline__ uint32_t unit_a_off(uint32_t m, uint32_t k) {
  return (k >> 3) * 2048u + (m >> 4) * 128u + (k & 7u) * 16u + (m & 15u);
}

// The 16 entries of a keystream word as M' = M + 1, two bits each: 00 -> 2, 01 -> 0,
// 1x -> 1, i.e. low bit = h, high bit = ~h & ~l.
__device__ __forceinline__ uint32_t packed_entries(uint32_t w) {
  const uint32_t high = ~(w | (w + w)) & 0xAAAAAAAAu;
  return ((w >> 1) & 0x55555555u) | high;
}

// One column's entries into the A tile (dst = its column's first 16 rows).
__device__ __forceinline__ void store_entries(unsigned char* dst, const uint32_t (&w)[16]) {
#pragma unroll
  for (int g = 0; g < 16; ++g) {
    const uint32_t m = packed_entries(w[g]);
    *reinterpret_cast<uint4*>(dst + 128 * g) =
        make_uint4(m, m & 0x0C0C0C0Cu, m & 0x30303030u, m & 0xC0C0C0C0u);
  }
}

// Matrix row of tile row m, and the sum of a tile row's true entries from the
// accumulators of the warp's 32 tile rows (lane = m % 32; all lanes take part).
__device__ __forceinline__ int tile_row_to_row(int m) {
  return (m & ~15) | ((m & 3) << 2) | ((m >> 2) & 3);
}
__device__ __forceinline__ uint32_t unscale(uint32_t d, int lane) {
  const int s = (lane >> 2) & 3;
  uint32_t rest = __shfl_down_sync(0xffffffffu, d, 4);
  rest += __shfl_down_sync(0xffffffffu, d, 8);
  rest += __shfl_down_sync(0xffffffffu, d, 12);
  return s == 0 ? d - rest : d >> (2 * s);
}

// sum_i 2^(8i) (d_i - corr_i), exact in 64 bits.
__device__ __forceinline__ long long weigh(const uint32_t* d, const uint32_t* corr) {
  long long v = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) v += ((long long)d[i] - (long long)corr[i]) << (8 * i);
  return v;
}

// v mod q in [0, q).
__device__ __forceinline__ uint32_t residue(long long v, uint32_t q) {
  const long long r = v % (long long)q;
  return (uint32_t)(r < 0 ? r + q : r);
}

// The MMA warp's loop (one lane): warp w's units are first(w), first(w) + stride, ...
// below nunits, first() ascending; issue(w, accumulate) issues one unit's MMAs. A group
// of kGroup warps is handed over through one barrier and released by one commit, and the
// full rounds are unrolled, every descriptor one addition away from a constant: the
// MMA warp shares its sub-partition with six warps that saturate the ALU pipe, so each
// of its instructions costs 10 to 15 cycles, and a tcgen05 instruction 44 on an idle SM.
// (One barrier and commit per unit, descriptors built in the loop: 600 cycles a unit,
// where the units come every 380.)
// Ends when every unit is issued (or a wait gave up) and all MMAs are done.
template <int WARPS, typename First, typename Issue>
__device__ __forceinline__ void mma_loop(uint64_t* full, uint64_t* empty, uint64_t* done,
                                         uint32_t nunits, uint32_t stride, First first,
                                         Issue issue, int* err) {
  static_assert(WARPS % kGroup == 0, "whole groups");
  bool ok = true;
  uint32_t acc = 0;
  // nunits + stride stays below 2^32
  for (uint32_t base = 0, it = 0; ok && first(0) + base < nunits; base += stride, ++it) {
    if (acc && first(WARPS - 1) + base < nunits) {
#pragma unroll
      for (int g = 0; g < WARPS / kGroup; ++g) {
        ok = ok && mbar_wait(&full[g], it & 1, err);
        if (ok) {
          tc::fence_after_sync();
#pragma unroll
          for (int i = 0; i < kGroup; ++i) issue(kGroup * g + i, 1u);
          tc::mma_commit(&empty[g]);
        }
      }
      continue;
    }
#pragma unroll 1
    for (int g = 0; g < WARPS / kGroup && first(kGroup * g) + base < nunits; ++g) {
      if (!(ok = mbar_wait(&full[g], it & 1, err))) break;
      tc::fence_after_sync();
#pragma unroll 1
      for (int w = kGroup * g; w < kGroup * (g + 1) && first(w) + base < nunits; ++w) {
        issue(w, acc);
        acc = 1;
      }
      tc::mma_commit(&empty[g]);
    }
  }
  tc::mma_commit(done);  // completes once every MMA issued above has (at once if none was)
  mbar_wait_sleep(done, 0, err);
}

// The producers' wait for their tiles: asleep in the barrier, since polling warps
// hold up the MMA warp's own waits.
__device__ __forceinline__ bool tiles_free(uint64_t* bar, uint32_t it, int lane, int* err) {
  bool ok = true;
  if (it > 0) {
    if (lane == 0) ok = mbar_wait_sleep(bar, (it - 1) & 1, err);
    __syncwarp();
    ok = __shfl_sync(0xffffffffu, ok, 0);
  }
  return ok;
}

// kFlat (whole blocks, d % 8 == 0, n % 32 == 0): the kernel also writes the
// int8 entries flat[row][part][k][j] (col = j d + k), so the keystream is generated
// once. A unit is then 32 consecutive polynomials of one coefficient index: lane l
// takes polynomial 32 jg + l. For each word of 4 rows the four lanes of a quad
// swap bytes (a 4 x 4 transpose: two shuffles, two byte permutes) so that lane
// 4 g + r holds one row of polynomials 4 g .. 4 g + 3, and the warp's stores fill
// whole 32-byte sectors of four rows.
// kMany: parts from part0 on, one of several launches (an instance of its own: with the
// offset in every projection 64 x 131072 columns took 418 us for 413).
template <bool kWholeBlocks, bool kFlat = false, bool kMany = false>
__global__ void __launch_bounds__(PjShape<kFlat>::THREADS, 1) jl_tc_kernel(
    const uint32_t* __restrict__ parts, unsigned long long cols, int rows, int packed_len,
    ChachaKey key, uint32_t nunits, uint32_t per_part, uint32_t d, unsigned long long plane,
    int8_t* __restrict__ flat, unsigned long long* __restrict__ gsum, uint32_t q, bool fold,
    int* __restrict__ err, uint32_t part0) {
  using S = PjShape<kFlat>;
  constexpr int WARPS = S::WARPS;
  extern __shared__ __align__(128) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 127u) & ~127u) - raw);
  const uint32_t s0 = smem_addr(sm);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + S::OFF_BAR);
  uint64_t* empty = full + WARPS / kGroup;
  uint64_t* done = empty + WARPS / kGroup;
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(done + 1);
  uint32_t* colsum = taddr_slot + 2;  // [4]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid < 4) colsum[tid] = 0;
  if (warp == WARPS) {
    tc::tmem_alloc(taddr_slot, 32);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < WARPS / kGroup; ++i) {
      mbar_init(&full[i], kGroup);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  const uint32_t stride = gridDim.x * WARPS;
  // consecutive units on consecutive SMs (few units: one warp of every SM), or, with
  // the entries, on consecutive warps: neighbouring polynomials' sectors of a row
  auto first = [&](int w) -> uint32_t {
    return kFlat ? blockIdx.x * WARPS + w : (uint32_t)w * gridDim.x + blockIdx.x;
  };

  if (warp == WARPS) {
    if (lane == 0) {
      // kind::i8, u8 x u8 -> s32, A and B MN-major, M = 128, N = 16
      const uint32_t idesc = tc::idesc_u8(128, 16) | (1u << 15) | (1u << 16);
      const uint64_t da = tc::smem_desc(s0, 2048, 128);
      const uint64_t db = tc::smem_desc(s0 + S::OFF_B, 128, 256);
      mma_loop<WARPS>(
          full, empty, done, nunits, stride, first,
          [&](int w, uint32_t acc) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              tc::mma_u8(tbase + 16 * h, tc::desc_plus(da, w * kUnitA + h * 1024),
                         tc::desc_plus(db, w * kPjB), idesc, acc);
          },
          err);
    }
    __syncwarp();
  } else {
    unsigned char* at = sm + warp * kUnitA + unit_a_off(0, lane);
    unsigned char* bt = sm + S::OFF_B + warp * kPjB + lane * 16;
    const unsigned long long npoly = cols / d;
    // byte selectors of the quad transpose (step 1: lanes l, l ^ 1; step 2: l, l ^ 2)
    const uint32_t sel1 = (lane & 1) ? 0x3715u : 0x6240u;
    const uint32_t sel2 = (lane & 2) ? 0x3276u : 0x5410u;
    uint32_t bsum[4] = {0, 0, 0, 0};
    uint32_t unit = first(warp);
    uint32_t part = unit / per_part, ci = unit % per_part;
    if constexpr (kMany) part += part0;
    const uint32_t step_part = stride / per_part, step_ci = stride % per_part;
    uint64_t* grp_full = &full[warp / kGroup];
    uint64_t* grp_empty = &empty[warp / kGroup];
    // a warp whose group still has a unit arrives with it
    uint32_t lead = first(warp / kGroup * kGroup);
    for (uint32_t it = 0; lead < nunits; ++it, unit += stride, lead += stride) {
      if (unit >= nunits) {
        if (tiles_free(grp_empty, it, lane, err) && lane == 0) mbar_arrive(grp_full);
        break;
      }
      unsigned long long c, jj = 0;
      uint32_t kk = 0;
      if constexpr (kFlat) {
        const uint32_t groups = per_part / d;  // polynomials / 32
        jj = (unsigned long long)(ci % groups) * 32 + lane;
        kk = ci / groups;
        c = jj * d + kk;
      } else {
        c = (unsigned long long)ci * kUnitCols + lane;
      }
      uint32_t w[16];
      uint32_t x = 0;
      if (c < cols) {
        x = __ldg(parts + (unsigned long long)part * cols + c);
        if constexpr (kWholeBlocks)
          chacha20_block(key, (uint32_t)c, part, w);
        else
          keystream_bytes(key, part, c * (unsigned long long)packed_len, packed_len, w);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = 0xFFFFFFFFu;  // padding column: x = 0
      }
      // the previous unit's MMAs must be done reading the tiles
      if (!tiles_free(grp_empty, it, lane, err)) break;
      store_entries(at, w);
      *reinterpret_cast<uint4*>(bt) = make_uint4(x, 0, 0, 0);
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(grp_full);
#pragma unroll
      for (int i = 0; i < 4; ++i) bsum[i] += (x >> (8 * i)) & 0xFFu;
      if constexpr (kFlat) {
        // word s of keystream word g: rows 16 g + 4 j + s (j = 0 .. 3) of this lane's
        // polynomial; after the transpose row 16 g + 4 (lane & 3) + s of
        // polynomials jj - (lane & 3) .. + 3
        int8_t* rowp = flat + ((unsigned long long)part * d + kk) * npoly + (jj - (lane & 3)) +
                       (unsigned long long)(4 * (lane & 3)) * plane;
#pragma unroll
        for (int g = 0; g < 16; ++g) {
          const uint32_t m = packed_entries(w[g]);
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            const uint32_t v = (m >> (2 * s)) & 0x03030303u;
            const uint32_t e = (v + 0x7F7F7F7Fu) ^ 0x80808080u;  // M = M' - 1 per byte
            const uint32_t a = __byte_perm(e, __shfl_xor_sync(0xffffffffu, e, 1), sel1);
            const uint32_t o = __byte_perm(a, __shfl_xor_sync(0xffffffffu, a, 2), sel2);
            if (16 * g + 4 * (lane & 3) + s < rows) *reinterpret_cast<uint32_t*>(rowp) = o;
            rowp += plane;
          }
          rowp += 12 * plane;
        }
      }
      part += step_part;
      ci += step_ci;
      if (ci >= per_part) {
        ci -= per_part;
        ++part;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t v = bsum[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) atomicAdd(&colsum[i], v);
    }
  }
  __syncthreads();  // every MMA is done, the byte sums are complete
  tc::fence_after_sync();
  if (warp < 4 && first(0) < nunits) {  // a CTA without units accumulated nothing
    uint32_t dv[2][4];
    tc::tmem_ld4(tc::tmem_addr(tbase, 32 * warp, 0), dv[0]);
    tc::tmem_ld4(tc::tmem_addr(tbase, 32 * warp, 16), dv[1]);
    tc::tmem_ld_wait(dv[0]);
    tc::tmem_ld_wait(dv[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = tile_row_to_row(128 * h + 32 * warp + lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) dv[h][i] = unscale(dv[h][i], lane);
      const long long v = weigh(dv[h], colsum);
      if (row < rows)
        atomicAdd(&gsum[row], (unsigned long long)(fold ? (long long)residue(v, q) : v));
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == WARPS) tc::tmem_dealloc(tbase, 32);
}

// out[i] = the signed sum gsum[i] mod q.
__global__ void jl_finish_kernel(const unsigned long long* __restrict__ gsum,
                                 uint32_t* __restrict__ out, int n, uint32_t q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = residue((long long)gsum[i], q);
}

// Entry -> int8 table for one keystream byte: 4 rows, 2 bits each.
__device__ __forceinline__ uint32_t entries_of_byte(uint32_t byte) {
  uint32_t out = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t c = (byte >> (2 * i)) & 3u;
    const uint32_t v = c == 0 ? 0x01u : (c == 1 ? 0xFFu : 0x00u);
    out |= v << (8 * i);
  }
  return out;
}

// flat[row][part][k][j] (int8) for col = j*d + k. A warp handles one (part, k)
// and 128 consecutive j, 4 per lane, so each row store is a 4-byte word and
// a warp writes 128 contiguous bytes per row.
template <bool kWholeBlocks>
__global__ void __launch_bounds__(kJlThreads) jl_flat_kernel(unsigned long long cols, int d,
                                                             int num_parts, int rows,
                                                             int packed_len, ChachaKey key,
                                                             int8_t* __restrict__ flat) {
  __shared__ uint32_t lut[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = entries_of_byte(i);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long n = cols / d;
  const unsigned long long jchunks = (n + 127) / 128;
  const unsigned long long total = (unsigned long long)num_parts * d * jchunks;
  const unsigned long long plane = (unsigned long long)num_parts * cols;  // bytes per row
  const unsigned long long stride = (unsigned long long)gridDim.x * kJlWarps;
  const bool vec_ok = (n % 4) == 0 && (reinterpret_cast<uintptr_t>(flat) & 3u) == 0;
  for (unsigned long long wk = (unsigned long long)blockIdx.x * kJlWarps + warp; wk < total;
       wk += stride) {
    const unsigned long long jc = wk % jchunks;
    const unsigned long long pk = wk / jchunks;  // part * d + k
    const uint32_t part = (uint32_t)(pk / d);
    const uint32_t k = (uint32_t)(pk % d);
    const unsigned long long j0 = jc * 128 + lane * 4;
    uint32_t w[4][16];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long j = j0 + u;
      if (j < n) {
        if constexpr (kWholeBlocks)
          chacha20_block(key, (uint32_t)(j * d + k), part, w[u]);
        else
          keystream64(key, part, (j * d + k) * (unsigned long long)packed_len, w[u]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) w[u][i] = 0xFFFFFFFFu;
      }
    }
    int8_t* base = flat + pk * n + j0;
#pragma unroll
    for (int b = 0; b < 64; ++b) {
      if (b >= packed_len) break;
      uint32_t e[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) e[u] = lut[(w[u][b >> 2] >> ((b & 3) * 8)) & 0xFFu];
      // transpose 4 columns x 4 rows of bytes: out[r] = (e0.r, e1.r, e2.r, e3.r)
      const uint32_t t01l = __byte_perm(e[0], e[1], 0x5140);
      const uint32_t t23l = __byte_perm(e[2], e[3], 0x5140);
      const uint32_t t01h = __byte_perm(e[0], e[1], 0x7362);
      const uint32_t t23h = __byte_perm(e[2], e[3], 0x7362);
      uint32_t o[4];
      o[0] = __byte_perm(t01l, t23l, 0x5410);
      o[1] = __byte_perm(t01l, t23l, 0x7632);
      o[2] = __byte_perm(t01h, t23h, 0x5410);
      o[3] = __byte_perm(t01h, t23h, 0x7632);
#pragma unroll
      for (int r4 = 0; r4 < 4; ++r4) {
        const int row = b * 4 + r4;
        if (row >= rows) break;
        int8_t* dst = base + (unsigned long long)row * plane;
        if (vec_ok && j0 + 3 < n) {
          *reinterpret_cast<uint32_t*>(dst) = o[r4];
        } else {
          for (int u = 0; u < 4; ++u)
            if (j0 + u < n) dst[u] = (int8_t)((o[r4] >> (8 * u)) & 0xFFu);
        }
      }
    }
  }
}


// ---------------------------------------------------------------------------
// JL evaluations (aggregation side): evals[m] = sum_{i,j} conj(pi_{m,i,j}) s_{i,j}
// (jl_rows_flat_to_conjugated_polys + the jl_evals loop of prove_step,
// main_protocol/mod.rs:885-923, step_prover.rs:185-206), without the int8
// entries ever being stored. Coefficient t of conj(pi) * s is
// sum_u pi_u s'[u + t] with s' the negacyclic extension (s'[v] = -s[v - d] for
// v >= d), so coefficient t of evals[m] is the JL projection of the witness
// with every polynomial multiplied by X^-t. One keystream therefore serves all
// d = 64 coefficients: column (j, u) of the B tile holds the 64 words
// s'_j[u + t], t = 0 .. 63, as 256 bytes (N = 256), and D'[r][4t + i] =
// sum_c M'[r][c] byte_i(s'[u_c + t]) accumulates in all 512 tensor-memory
// columns (two 128-row halves). The M' = M + 1 correction
// S[t][i] = sum_c byte_i(s'[u_c + t]) comes from per-position byte sums of each
// coefficient and its negation: sum_{v >= t} P_i[v] + sum_{v < t} N_i[v].
//
// A unit is 32 coefficients (half a polynomial) of one part. The B tile is a
// Hankel matrix, word (u, t) = s'[u + t]: core matrix (k-group kg, t-group g) depends
// on 2 kg + g alone, so the tile is 22 overlapping core matrices (128 bytes each)
// instead of 64, and the descriptor's strides are 2 and 1 of them. Bound and
// hand-over as in the projection (20 producer warps: 11 KB of tiles each); the
// tensor pipe is the second resource, 256 cycles per unit of about 400.
// Measured at 64 x 131072 columns: 0.78 ms before (one chunk of 256 columns per CTA
// at a time, table lookups, every rotation written out), 0.47 ms now.
// ---------------------------------------------------------------------------
constexpr int kEvD = 64, kEvRows = 256;
constexpr int kEvWarps = 20;
constexpr int kEvThreads = (kEvWarps + 1) * 32;
constexpr uint32_t kEvCores = 22;                       // 2 kg + g, kg < 4, g < 16
constexpr uint32_t kEvB = kEvCores * 128;
constexpr uint32_t kEvOffB = kEvWarps * kUnitA;
constexpr uint32_t kEvOffExt = kEvOffB + kEvWarps * kEvB;  // s', 128 words per warp
constexpr uint32_t kEvOffBar = kEvOffExt + kEvWarps * 512;
constexpr uint32_t kEvSmem = kEvOffBar + (2 * kEvWarps / kGroup + 1) * 8 + 16 + 128;
static_assert(kEvSmem <= 232448, "shared memory budget");
// after the last MMA the tiles hold the corrections: P[64][4], N[64][4], S[64][4]
constexpr uint32_t kEvOffSums = 0, kEvOffS = 2048;

__global__ void __launch_bounds__(kEvThreads, 1) jl_eval_tc_kernel(
    const uint32_t* __restrict__ parts, unsigned long long cols, ChachaKey key, uint32_t nunits,
    uint32_t per_part, unsigned long long* __restrict__ gsum, uint32_t q, bool fold,
    int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 127u) & ~127u) - raw);
  const uint32_t s0 = smem_addr(sm);
  uint32_t* sums = reinterpret_cast<uint32_t*>(sm + kEvOffSums);  // [0,256): P, [256,512): N
  uint32_t* corr = reinterpret_cast<uint32_t*>(sm + kEvOffS);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + kEvOffBar);
  uint64_t* empty = full + kEvWarps / kGroup;
  uint64_t* done = empty + kEvWarps / kGroup;
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == kEvWarps) {
    tc::tmem_alloc(taddr_slot, 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < kEvWarps / kGroup; ++i) {
      mbar_init(&full[i], kGroup);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  const uint32_t stride = gridDim.x * kEvWarps;  // even: a warp keeps its half polynomial
  auto first = [&](int w) -> uint32_t { return (uint32_t)w * gridDim.x + blockIdx.x; };

  uint32_t psum[4] = {0, 0, 0, 0}, nsum[4] = {0, 0, 0, 0};
  uint32_t u0 = 0;
  if (warp == kEvWarps) {
    if (lane == 0) {
      // kind::i8, u8 x u8 -> s32, A and B MN-major, M = 128, N = 256
      const uint32_t idesc = tc::idesc_u8(128, 256) | (1u << 15) | (1u << 16);
      const uint64_t da = tc::smem_desc(s0, 2048, 128);
      const uint64_t db = tc::smem_desc(s0 + kEvOffB, 256, 128);
      mma_loop<kEvWarps>(
          full, empty, done, nunits, stride, first,
          [&](int w, uint32_t acc) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              tc::mma_u8(tbase + 256 * h, tc::desc_plus(da, w * kUnitA + h * 1024),
                         tc::desc_plus(db, w * kEvB), idesc, acc);
          },
          err);
    }
    __syncwarp();
  } else {
    unsigned char* at = sm + warp * kUnitA + unit_a_off(0, lane);
    unsigned char* bt = sm + kEvOffB + warp * kEvB;
    uint32_t* ext = reinterpret_cast<uint32_t*>(sm + kEvOffExt + warp * 512);
    uint32_t unit = first(warp);
    uint32_t part = unit / per_part, ci = unit % per_part;
    const uint32_t step_part = stride / per_part, step_ci = stride % per_part;
    u0 = (unit & 1) * kUnitCols;  // per_part is even: the unit's half polynomial
    uint64_t* grp_full = &full[warp / kGroup];
    uint64_t* grp_empty = &empty[warp / kGroup];
    // a warp whose group still has a unit arrives with it
    uint32_t lead = first(warp / kGroup * kGroup);
    for (uint32_t it = 0; lead < nunits; ++it, unit += stride, lead += stride) {
      if (unit >= nunits) {
        if (tiles_free(grp_empty, it, lane, err) && lane == 0) mbar_arrive(grp_full);
        break;
      }
      const unsigned long long c = (unsigned long long)ci * kUnitCols + lane;
      const uint32_t* poly = parts + (unsigned long long)part * cols + (c & ~(kEvD - 1ull));
      const uint32_t x0 = __ldg(poly + lane), x1 = __ldg(poly + kUnitCols + lane);
      uint32_t w[16];
      chacha20_block(key, (uint32_t)c, part, w);  // 256 rows: column c is block c
      const uint32_t n0 = x0 == 0 ? 0u : q - x0, n1 = x1 == 0 ? 0u : q - x1;
      const uint32_t x = u0 ? x1 : x0, xn = u0 ? n1 : n0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        psum[i] += (x >> (8 * i)) & 0xFFu;
        nsum[i] += (xn >> (8 * i)) & 0xFFu;
      }
      // the previous unit's MMAs must be done reading the tiles
      if (!tiles_free(grp_empty, it, lane, err)) break;
      ext[lane] = x0;
      ext[32 + lane] = x1;
      ext[64 + lane] = n0;
      ext[96 + lane] = n1;
      store_entries(at, w);
      __syncwarp();
      // row r of core matrix cm: words s'[u0 + 4 cm + r .. + 3]
#pragma unroll
      for (uint32_t i = lane; i < kEvCores * 8; i += 32) {
        const uint32_t* src = ext + u0 + 4 * (i >> 3) + (i & 7);
        *reinterpret_cast<uint4*>(bt + 16 * i) = make_uint4(src[0], src[1], src[2], src[3]);
      }
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(grp_full);
      part += step_part;
      ci += step_ci;
      if (ci >= per_part) {
        ci -= per_part;
        ++part;
      }
    }
  }
  __syncthreads();  // every MMA is done: the tiles' shared memory is free
  // per-position byte sums of the coefficients and of their negations
  for (int i = tid; i < 512; i += kEvThreads) sums[i] = 0;
  __syncthreads();
  if (warp < kEvWarps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      atomicAdd(&sums[4 * (u0 + lane) + i], psum[i]);
      atomicAdd(&sums[256 + 4 * (u0 + lane) + i], nsum[i]);
    }
  }
  __syncthreads();
  if (tid < 4 * kEvD) {
    // S[t][i] = sum_{v >= t} P[v][i] + sum_{v < t} N[v][i], thread (t, i) = (tid / 4, tid % 4)
    const int t = tid >> 2, i = tid & 3;
    uint32_t acc = 0;
    for (int v = 0; v < kEvD; ++v) acc += v >= t ? sums[4 * v + i] : sums[256 + 4 * v + i];
    corr[tid] = acc;
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp < 16 && first(0) < nunits) {
    // warp: lane quarter warp % 4 of half (warp / 4) % 2, 32 of the 64 coefficients
    const int h = (warp >> 2) & 1, wl = warp & 3, tbeg = 32 * (warp >> 3);
    const int row = tile_row_to_row(128 * h + 32 * wl + lane);
    const uint32_t base = tc::tmem_addr(tbase, 32 * wl, 256 * h);
#pragma unroll 1
    for (int t0 = tbeg; t0 < tbeg + 32; t0 += 2) {
      uint32_t dv[8];
      tc::tmem_ld8(base + 4 * t0, dv);
      tc::tmem_ld_wait(dv);
#pragma unroll
      for (int i = 0; i < 8; ++i) dv[i] = unscale(dv[i], lane);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const long long v = weigh(dv + 4 * k, corr + 4 * (t0 + k));
        atomicAdd(&gsum[(size_t)row * kEvD + t0 + k],
                  (unsigned long long)(fold ? (long long)residue(v, q) : v));
      }
      __syncwarp();
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kEvWarps) tc::tmem_dealloc(tbase, 512);
}

// Signed 64-bit sums over all columns stay exact without a reduction per CTA while
// columns * 255 * (1 + 2^8 + 2^16 + 2^24) < 2^63.
bool must_fold(unsigned long long columns) { return columns >= (1ull << 30); }

}  // namespace

size_t jl_scratch_bytes(size_t rows) { return rows * sizeof(unsigned long long); }

int launch_jl_project(const FieldParams& f, const uint8_t seed[32], size_t rows,
                      const uint32_t* parts, size_t num_parts, size_t cols, size_t d,
                      uint32_t* p_out, int8_t* flat_out, void* scratch, size_t scratch_bytes,
                      int num_sms, int* err, cudaStream_t s) {
  if (rows == 0 || rows > 256 || d == 0 || cols % d != 0 || num_parts == 0 ||
      num_parts > 0xFFFFFFFFull)
    return GRID_ERR_INVALID_PARAMETERS;
  if (scratch_bytes < jl_scratch_bytes(rows)) return GRID_ERR_INVALID_PARAMETERS;
  const ChachaKey key = chacha::make_key(seed);
  const int packed_len = (int)((rows + 3) / 4);
  unsigned long long* gsum = static_cast<unsigned long long*>(scratch);
  cudaError_t e = cudaMemsetAsync(gsum, 0, rows * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return cuda_status(e);
  // the int8 entries come out of the projection kernel itself when the
  // columns split into 32 polynomials per coefficient and rows fill the blocks
  const unsigned long long npoly = cols / d;
  const bool fused_flat = flat_out && packed_len == 64 && d % 8 == 0 && npoly % 32 == 0 &&
                          (reinterpret_cast<uintptr_t>(flat_out) & 3u) == 0;
  const unsigned long long per_part =
      fused_flat ? npoly / 32 * d : (cols + kUnitCols - 1) / kUnitCols;
  const unsigned long long plane = (unsigned long long)num_parts * cols;  // flat bytes per row
  if (cols > 0) {
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return cuda_status(e);
    const unsigned long long step = parts_per_launch(per_part, num_parts);
    if (!step) return GRID_ERR_INVALID_PARAMETERS;
    auto run = [&](auto kernel, auto shape, int* cache) -> int {
      using S = decltype(shape);
      int bps = 0;
      int rc = prepare_kernel(kernel, S::SMEM, S::THREADS, dev, cache, &bps);
      for (unsigned long long at = 0; !rc && at < num_parts; at += step) {
        const unsigned long long nunits =
            per_part * std::min(step, (unsigned long long)num_parts - at);
        kernel<<<unit_grid(nunits, S::WARPS, num_sms), S::THREADS, S::SMEM, s>>>(
            parts, cols, (int)rows, packed_len, key, (uint32_t)nunits, (uint32_t)per_part,
            (uint32_t)d, plane, fused_flat ? flat_out : nullptr, gsum, f.q, must_fold(plane), err,
            (uint32_t)at);
        rc = cuda_status(cudaGetLastError());
      }
      return rc;
    };
    static int cache_whole[kMaxDevices] = {}, cache_part[kMaxDevices] = {},
               cache_flat[kMaxDevices] = {}, cache_many[2][kMaxDevices] = {};
    const PjShape<false> plain;
    int rc;
    if (fused_flat)  // 2^31 units' entries fit no memory
      rc = step < num_parts ? GRID_ERR_INVALID_PARAMETERS
                            : run(jl_tc_kernel<true, true>, PjShape<true>(), cache_flat);
    else if (step < num_parts)
      rc = packed_len == 64 ? run(jl_tc_kernel<true, false, true>, plain, cache_many[1])
                            : run(jl_tc_kernel<false, false, true>, plain, cache_many[0]);
    else
      rc = packed_len == 64 ? run(jl_tc_kernel<true>, plain, cache_whole)
                            : run(jl_tc_kernel<false>, plain, cache_part);
    if (rc) return rc;
  }
  jl_finish_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(gsum, p_out, (int)rows, f.q);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e);
  if (flat_out && cols > 0 && !fused_flat) {
    const unsigned long long n = cols / d;
    const unsigned long long work = (unsigned long long)num_parts * d * ((n + 127) / 128);
    unsigned long long blocks = (work + kJlWarps - 1) / kJlWarps;
    const unsigned long long cap = (unsigned long long)num_sms * 8;
    if (blocks > cap) blocks = cap;
    if (packed_len == 64)
      jl_flat_kernel<true><<<(unsigned)blocks, kJlThreads, 0, s>>>(
          cols, (int)d, (int)num_parts, (int)rows, packed_len, key, flat_out);
    else
      jl_flat_kernel<false><<<(unsigned)blocks, kJlThreads, 0, s>>>(
          cols, (int)d, (int)num_parts, (int)rows, packed_len, key, flat_out);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_status(e);
  }
  return GRID_OK;
}


size_t jl_evals_scratch_bytes() { return (size_t)kEvRows * kEvD * sizeof(unsigned long long); }

// evals: kEvRows x d words. Only the LaBRADOR shape (256 rows, d = 64) has a
// kernel; other shapes return GRID_ERR_UNSUPPORTED_SIZE.
int launch_jl_evals(const FieldParams& f, const uint8_t seed[32], size_t rows,
                    const uint32_t* parts, size_t num_parts, size_t cols, size_t d,
                    uint32_t* evals, void* scratch, size_t scratch_bytes, int num_sms, int* err,
                    cudaStream_t s) {
  if (rows != (size_t)kEvRows || d != (size_t)kEvD) return GRID_ERR_UNSUPPORTED_SIZE;
  if (cols == 0 || cols % d != 0 || num_parts == 0 || num_parts > 0xFFFFFFFFull)
    return GRID_ERR_INVALID_PARAMETERS;
  if (scratch_bytes < jl_evals_scratch_bytes()) return GRID_ERR_INVALID_PARAMETERS;
  const ChachaKey key = chacha::make_key(seed);
  unsigned long long* gsum = static_cast<unsigned long long*>(scratch);
  cudaError_t e = cudaMemsetAsync(gsum, 0, jl_evals_scratch_bytes(), s);
  if (e != cudaSuccess) return cuda_status(e);
  const unsigned long long per_part = cols / kUnitCols;  // d = 64: a whole, even number
  if (parts_per_launch(per_part, num_parts) < num_parts)  // 2^31 units fit no memory
    return GRID_ERR_INVALID_PARAMETERS;
  const unsigned long long nunits = per_part * num_parts;
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return cuda_status(e);
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  int rc = prepare_kernel(jl_eval_tc_kernel, kEvSmem, kEvThreads, dev, bps_cache, &bps);
  if (rc) return rc;
  jl_eval_tc_kernel<<<unit_grid(nunits, kEvWarps, num_sms), kEvThreads, kEvSmem, s>>>(
      parts, cols, key, (uint32_t)nunits, (uint32_t)per_part, gsum, f.q,
      must_fold((unsigned long long)num_parts * cols), err);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  const int n = kEvRows * kEvD;
  jl_finish_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(gsum, evals, n, f.q);
  return cuda_status(cudaGetLastError());
}

}  // namespace grid
