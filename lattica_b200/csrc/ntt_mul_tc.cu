// Tensor-core negacyclic products for d = 64 (tcgen05, kind::i8):
// out = INTT(NTT(a) (.) b), b given in the evaluation domain (natural slots), the
// product a Montgomery product as in every other path.
//
// Reference path replaced: the "NTT -> Montgomery pointwise -> INTT" chain of a
// negacyclic product over TwistedNttPlan (algebra/src/poly/ntt.rs:75-126), bit-exact.
//
// The forward is the byte-plane transform of ntt_tc_common.cuh. The inverse works on half
// the columns: psi^(-64 m) = (-1)^m, so with S_k = Z_k + Z_(k+32) and D_k = Z_k - Z_(k+32)
// (k < 32) the even outputs are sum_k S_k psi^(-(2k+1) m) / 64 and the odd ones the same sum
// over D_k: two products of 32 words by 32 columns instead of one of 64 by 64. Its half
// of the multiply-adds is worth two additions a pair of words, since at 2^22 polynomials
// the MMAs' power, not their time, holds the kernel back (0.55 ms without any MMA, 0.70 ms
// alone and 0.78 ms under the power cap with two full transforms), and its matrix takes
// 32 KB of shared memory instead of 64.
//
// A tile is 128 polynomials. Four groups of four epilogue warps, one warp of each per SM
// sub-partition, run apart from each other, so a sub-partition's integer pipe is fed by
// one while another waits for its MMAs or its tensor-memory loads:
//   loader (warp 17): TMA of a in half-tile boxes (three in a ring, each released once its
//     MMAs are done), of b in 16-column boxes, L2 prefetch of both
//   MMA (warp 16): fwd(j) once its boxes landed and tile j - 1's columns are read; then
//     inv(j - 1) once its operand is written and tile j - 2's columns are read
//   F0, F1 (warps 0-7): 32 forward columns each, k = 16 h .. + 15 and the same + 32, in
//     two batches of 8 + 8: combine the planes, multiply by b, write S and D
//   E0, E1 (warps 8-15): 32 outputs each in two batches, m = 2 i and 2 i + 1 from the two
//     products; staged per group and stored by TMA
// Measured at 2^22 polynomials: 0.64 ms alone and 0.75 to 0.78 ms in a loop that reaches the
// power cap; with both full matrices in shared memory, one epilogue phase after the other in
// all 16 warps and the results staged in the input's two buffers 0.78 to 0.84 ms. Without
// the MMAs 0.56 ms, without the integer arithmetic 0.57 (768 bytes a polynomial at the
// measured HBM rate: 0.49).
// Every wait is bounded.
#include <cuda.h>
#include <cuda_runtime.h>

#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_tc.cuh"
#include "ntt_tc_common.cuh"

namespace grid {
namespace {

using namespace tcx;

constexpr int D = 64;
constexpr int NXA = 3;                           // input boxes in the ring
constexpr uint32_t QUARTER = ROWS * 64;          // 128 rows x 16 words
constexpr uint32_t OFF_W = 0;                    // forward matrix
constexpr uint32_t OFF_G = OFF_W + WMAT;         // inverse: even, odd outputs (16 KB each)
constexpr uint32_t OFF_XA = OFF_G + 2 * BOX;
constexpr uint32_t OFF_PP = OFF_XA + NXA * BOX;  // S, D (inverse's A)
constexpr uint32_t OFF_B = OFF_PP + TILE;        // b: four boxes of 16 words
constexpr uint32_t OFF_ST = OFF_B + 4 * QUARTER; // one staged quarter of results per E group
constexpr uint32_t OFF_BAR = OFF_ST + 2 * QUARTER;
constexpr uint32_t SMEM_BYTES = OFF_BAR + 32 * 8 + 16 + 1024;  // + alignment slack
static_assert(SMEM_BYTES <= 232448, "shared memory budget");
constexpr int GROUP_WARPS = 4;

enum Bar : int {
  AFULL = 0,            // [3] input box landed
  AFREE = AFULL + NXA,  // [3] its MMAs done
  BFULL = AFREE + NXA,  // [2] boxes h and h + 2 of b landed
  BFREE = BFULL + 2,    // [2] read by group F_h
  FDONE = BFREE + 2,    // forward done
  FREAD,                // its columns read
  PREADY,               // S and D written
  IDONE,                // inverse done (S and D read)
  EREAD,                // its columns read
  DRAIN,                // every MMA done
  WFULL,                // the matrices landed
  NBARS
};
static_assert(NBARS <= 32, "barrier slots");

// Byte offset of (row, 16-byte chunk) in a 64-byte-swizzled 128 x 64-byte tile.
__device__ __forceinline__ uint32_t sw64(uint32_t row, uint32_t c) {
  return row * 64 + ((c ^ ((row >> 1) & 3u)) << 4);
}

// True iff every warp of the group (named barrier id) passes ok.
__device__ __forceinline__ bool group_all(int id, bool ok) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)ok), "r"(id)
      : "memory");
  return r != 0;
}

__global__ void __launch_bounds__(THREADS, 1)
    ntt_mul_tc_kernel(const __grid_constant__ CUtensorMap tmap_a,
                      const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_out, const uint32_t* a,
                      const uint32_t* b, unsigned long long npolys,
                      const uint4* __restrict__ wtab, const uint4* __restrict__ gtab, const TcConsts k,
                      int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(bars + 32);

  if (warp == MMA_WARP) {
    if (lane == 0) {
      for (int i = 0; i < NXA; ++i) {
        mbar_init(&bars[AFULL + i], 1);
        mbar_init(&bars[AFREE + i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&bars[BFULL + i], 1);
        mbar_init(&bars[BFREE + i], GROUP_WARPS);
      }
      mbar_init(&bars[FDONE], 1);
      mbar_init(&bars[FREAD], 2 * GROUP_WARPS);
      mbar_init(&bars[PREADY], 2 * GROUP_WARPS);
      mbar_init(&bars[IDONE], 1);
      mbar_init(&bars[EREAD], 2 * GROUP_WARPS);
      mbar_init(&bars[DRAIN], 1);
      mbar_init(&bars[WFULL], 1);
      fence_mbar_init();
      tc::fence_async_smem();
      mbar_arrive_expect_tx(&bars[WFULL], WMAT + 2 * BOX);
      bulk_load(sm + OFF_W, wtab, WMAT, &bars[WFULL]);
      bulk_load(sm + OFF_G, gtab, 2 * BOX, &bars[WFULL]);
    }
    __syncwarp();
    tc::tmem_alloc(taddr_slot, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  grid_dep_wait();
  grid_dep_launch();

  const unsigned long long ntiles = (npolys + ROWS - 1) / ROWS;
  const uint32_t n = blockIdx.x < ntiles
                         ? (uint32_t)((ntiles - 1 - blockIdx.x) / gridDim.x + 1)
                         : 0u;  // tiles of this CTA
  auto row0 = [&](uint32_t j) -> unsigned long long {
    return ((unsigned long long)blockIdx.x + (unsigned long long)j * gridDim.x) * ROWS;
  };

  if (warp == LOAD_WARP) {
    // ------------------------------------------------------------ loader
    if (lane == 0) {
      bool ok = true;
      uint32_t boxes = 0, bloads[2] = {};
      auto prefetch = [&](uint32_t j) {
        if (j >= n) return;
        const unsigned long long r0 = row0(j), left = npolys - r0;
        const uint32_t bytes = (uint32_t)((left < ROWS ? left : ROWS) * D * 4);
        prefetch_l2(a + r0 * D, bytes);
        prefetch_l2(b + r0 * D, bytes);
      };
      prefetch(0);
      prefetch(1);
      for (uint32_t t = 0; ok && t < n; ++t) {
        const int y = (int)row0(t);
        for (int h = 0; ok && h < 2; ++h) {  // box h: words 32 h .. 32 h + 31
          const uint32_t slot = boxes % NXA, use = boxes / NXA;
          if (use) ok = mbar_wait(&bars[AFREE + slot], (use - 1) & 1, err);
          if (!ok) break;
          mbar_arrive_expect_tx(&bars[AFULL + slot], BOX);
          tma_load_2d(s0 + OFF_XA + slot * BOX, &tmap_a, 32 * h, y, smem_addr(&bars[AFULL + slot]));
          ++boxes;
        }
        for (int h = 0; ok && h < 2; ++h) {  // columns 16 h .. + 15 and 32 + 16 h .. + 15
          if (t) ok = mbar_wait(&bars[BFREE + h], (t - 1) & 1, err);
          if (!ok) break;
          mbar_arrive_expect_tx(&bars[BFULL + h], 2 * QUARTER);
          for (int g = h; g < 4; g += 2)
            tma_load_2d(s0 + OFF_B + g * QUARTER, &tmap_b, 16 * g, y, smem_addr(&bars[BFULL + h]));
          ++bloads[h];
        }
        prefetch(t + 2);
      }
      // no copy may still be writing shared memory when the CTA exits
      for (uint32_t i = 0; i < NXA; ++i) {
        const uint32_t loads = boxes > i ? (boxes - i + NXA - 1) / NXA : 0;
        if (loads) mbar_wait_sleep(&bars[AFULL + i], (loads - 1) & 1, err);
      }
      for (int i = 0; i < 2; ++i)
        if (bloads[i]) mbar_wait_sleep(&bars[BFULL + i], (bloads[i] - 1) & 1, err);
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------ MMA issue
    if (lane == 0) {
      const uint32_t idesc_f = tc::idesc_u8(ROWS, 256), idesc_i = tc::idesc_u8(ROWS, 128);
      const uint64_t dw = desc_sw128(s0 + OFF_W), dx = desc_sw128(s0 + OFF_XA);
      const uint64_t dg = desc_sw128(s0 + OFF_G), dp = desc_sw128(s0 + OFF_PP);
      auto inverse = [&](uint32_t j) -> bool {  // inv(j): even outputs, then odd
        if (!mbar_wait(&bars[PREADY], j & 1, err)) return false;
        if (j && !mbar_wait(&bars[EREAD], (j - 1) & 1, err)) return false;
        tc::fence_after_sync();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int s = 0; s < 4; ++s)
            tc::mma_u8(tbase + 256 + 128 * h, tc::desc_plus(dp, h * BOX + 32 * s),
                       tc::desc_plus(dg, h * BOX + 32 * s), idesc_i, s != 0);
        tc::mma_commit(&bars[IDONE]);
        return true;
      };
      bool ok = mbar_wait(&bars[WFULL], 0, err);
      uint32_t boxes = 0;
      for (uint32_t j = 0; ok && j < n; ++j) {
        if (j) ok = mbar_wait(&bars[FREAD], (j - 1) & 1, err);
#pragma unroll
        for (int kb = 0; kb < 2; ++kb, ++boxes) {
          const uint32_t slot = boxes % NXA;
          ok = ok && mbar_wait(&bars[AFULL + slot], (boxes / NXA) & 1, err);
          if (!ok) break;
          tc::fence_after_sync();
          const uint64_t da = tc::desc_plus(dx, slot * BOX);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            tc::mma_u8(tbase, tc::desc_plus(da, 32 * s),
                       tc::desc_plus(dw, kb * (WMAT / 2) + 32 * s), idesc_f, (kb | s) != 0);
          tc::mma_commit(&bars[AFREE + slot]);
        }
        if (ok) tc::mma_commit(&bars[FDONE]);
        if (ok && j) ok = inverse(j - 1);
      }
      if (ok && n) inverse(n - 1);
      // every MMA is done before shared and tensor memory are released
      tc::mma_commit(&bars[DRAIN]);
      mbar_wait_sleep(&bars[DRAIN], 0, err);
    }
    __syncwarp();
  } else {
    const uint32_t wl = warp & 3, h = (warp >> 2) & 1;
    const uint32_t row = 32 * wl + lane;
    // word i of 8 from its planes
    auto combine8 = [&](const uint32_t (&e)[4][8], int i) -> uint32_t {
      const uint32_t lo = e[0][i] + 256u * e[1][i], hi = e[2][i] + 256u * e[3][i];
      return redc64(mad_wide(hi, 65536u, (uint64_t)lo), k.q, k.qinv);
    };
    if (warp < 2 * GROUP_WARPS) {
      // ------------------------------------------------- F: columns 16 h .. and + 32
      const uint32_t taddr = tc::tmem_addr(tbase, 32 * wl, 16 * h);
      const unsigned char* b0 = sm + OFF_B + h * QUARTER;  // columns + 32: 2 QUARTER on
      unsigned char* pp = sm + OFF_PP;
      bool ok = true;
      for (uint32_t j = 0; ok && j < n; ++j) {
        ok = lane0_wait(&bars[FDONE], j & 1, lane, err);
        if (!ok) break;
        tc::fence_after_sync();
#pragma unroll 1
        for (uint32_t bt = 0; bt < 2; ++bt) {
          uint32_t e0[4][8], e1[4][8];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            tc::tmem_ld8(taddr + 64 * l + 8 * bt, e0[l]);
            tc::tmem_ld8(taddr + 64 * l + 32 + 8 * bt, e1[l]);
          }
          tc::tmem_ld_wait32(e0);
          tc::tmem_ld_wait32(e1);
          if (bt == 1) {  // the columns are free for fwd(j + 1)
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[FREAD]);
          }
          uint32_t z0[8], z1[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            z0[i] = combine8(e0, i);
            z1[i] = combine8(e1, i);
          }
          if (bt == 0 && !(ok = lane0_wait(&bars[BFULL + h], j & 1, lane, err))) break;
#pragma unroll
          for (int c = 0; c < 2; ++c) {  // Montgomery products with b: z * b < q * 2^32
            const uint32_t off = sw64(row, 2 * bt + c);
            const uint4 v0 = *reinterpret_cast<const uint4*>(b0 + off);
            const uint4 v1 = *reinterpret_cast<const uint4*>(b0 + 2 * QUARTER + off);
            const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t p0 = redc64(mad_wide(z0[4 * c + i], w0[i], 0ull), k.q, k.qinv);
              const uint32_t p1 = redc64(mad_wide(z1[4 * c + i], w1[i], 0ull), k.q, k.qinv);
              z0[4 * c + i] = add_canon(p0, p1, k.q);
              z1[4 * c + i] = sub_lazy(p0, p1, k.q);
            }
          }
          if (bt == 1) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[BFREE + h]);
          }
          // inv(j - 1) must be done reading S and D
          if (bt == 0 && j && !(ok = lane0_wait(&bars[IDONE], (j - 1) & 1, lane, err))) break;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t off = sw128(row, 0, 4 * h + 2 * bt + c, BOX);
            *reinterpret_cast<uint4*>(pp + off) =
                make_uint4(z0[4 * c], z0[4 * c + 1], z0[4 * c + 2], z0[4 * c + 3]);
            *reinterpret_cast<uint4*>(pp + BOX + off) =
                make_uint4(z1[4 * c], z1[4 * c + 1], z1[4 * c + 2], z1[4 * c + 3]);
          }
          __syncwarp();
        }
        if (!ok) break;
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[PREADY]);
      }
    } else {
      // ------------------------------------------------- E: outputs 32 h .. + 31
      const uint32_t taddr = tc::tmem_addr(tbase, 32 * wl, 256 + 16 * h);
      const int bar_id = 1 + (int)h;
      const bool elected = wl == 0 && lane == 0;
      unsigned char* st = sm + OFF_ST + h * QUARTER;
      bool ok = true;
      for (uint32_t j = 0; ok && j < n; ++j) {
        ok = lane0_wait(&bars[IDONE], j & 1, lane, err);
        tc::fence_after_sync();
#pragma unroll 1
        for (uint32_t bt = 0; bt < 2; ++bt) {
          uint32_t e0[4][8], e1[4][8], res[16];
#pragma unroll
          for (int l = 0; l < 4; ++l) {
            tc::tmem_ld8(taddr + 32 * l + 8 * bt, e0[l]);
            tc::tmem_ld8(taddr + 128 + 32 * l + 8 * bt, e1[l]);
          }
          tc::tmem_ld_wait32(e0);
          tc::tmem_ld_wait32(e1);
          if (bt == 1) {  // the columns are free for inv(j + 1)
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[EREAD]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            res[2 * i] = combine8(e0, i);
            res[2 * i + 1] = combine8(e1, i);
          }
          if (elected) bulk_wait_read_all();  // the group's previous store has read st
          if (!(ok = group_all(bar_id, ok))) break;  // the group leaves together
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(st + sw64(row, c)) =
                make_uint4(res[4 * c], res[4 * c + 1], res[4 * c + 2], res[4 * c + 3]);
          tc::fence_async_smem();
          group_all(bar_id, true);
          if (elected) {
            tma_store_2d(&tmap_out, (int)(32 * h + 16 * bt), (int)row0(j), smem_addr(st));
            bulk_commit();
          }
          __syncwarp();
        }
      }
      if (elected) bulk_wait_all();
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
}

uint64_t mulmod(uint64_t x, uint64_t y, uint64_t q) {
  return (uint64_t)((unsigned __int128)x * y % q);
}

}  // namespace

// The inverse's matrices in the layout of OFF_G: row 32 l + i of matrix t, K byte 4 k + i',
// holds byte l of 2^(8i') psi^(-(2k+1) m) 64^-1 2^32 mod q, m = 2 i + t. Appended to out.
void build_tc_mul_table(uint32_t q, uint64_t psi, uint64_t ninv, std::vector<unsigned char>& out) {
  uint64_t pw[2 * D];  // 64^-1 psi^e in Montgomery form
  pw[0] = mulmod(ninv, ((uint64_t)1 << 32) % q, q);
  for (uint32_t e = 1; e < 2 * D; ++e) pw[e] = mulmod(pw[e - 1], psi, q);
  const size_t base = out.size();
  out.resize(base + 2 * BOX);
  for (uint32_t m = 0; m < D; ++m)
    for (uint32_t kk = 0; kk < D / 2; ++kk) {
      uint64_t w = pw[(2 * D - (2 * kk + 1) * m % (2 * D)) % (2 * D)];
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t kb = 4 * kk + i;
        for (uint32_t l = 0; l < 4; ++l)
          out[base + sw128(32 * l + m / 2, m % 2, kb / 16, BOX) + kb % 16] =
              (unsigned char)(w >> (8 * l));
        w = mulmod(w, 256, q);  // next byte of the word: times 2^8
      }
    }
}

int launch_ntt_mul_tc(const grid_gpu_plan* p, const uint32_t* a, const uint32_t* b, uint32_t* out,
                      size_t npolys, cudaStream_t s) {
  if (npolys == 0) return GRID_OK;
  if (npolys > (size_t)INT32_MAX - ROWS) return GRID_ERR_INVALID_PARAMETERS;  // TMA row coordinate
  EncodeTiled enc = encoder();
  if (!enc) return GRID_ERR_CUDA;
  // rows of 64 words: a in boxes of 32 words x 128 rows (128-byte swizzle), b and out
  // of 16 words x 128 rows (64-byte swizzle)
  CUtensorMap map_a, map_b, map_out;
  const cuuint64_t dims[2] = {64, (cuuint64_t)npolys};
  const cuuint64_t strides[1] = {256};
  const cuuint32_t box_a[2] = {32, ROWS}, box_q[2] = {16, ROWS};
  const cuuint32_t estr[2] = {1, 1};
  auto make = [&](CUtensorMap* m, const void* ptr, const cuuint32_t* box, CUtensorMapSwizzle sw) {
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(ptr), dims, strides, box,
               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (!make(&map_a, a, box_a, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make(&map_b, b, box_q, CU_TENSOR_MAP_SWIZZLE_64B) ||
      !make(&map_out, out, box_q, CU_TENSOR_MAP_SWIZZLE_64B))
    return GRID_ERR_CUDA;
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  const int st = prepare_kernel(ntt_mul_tc_kernel, SMEM_BYTES, THREADS, p->device, bps_cache, &bps);
  if (st) return st;
  const unsigned long long tiles = (npolys + ROWS - 1) / ROWS;
  const unsigned long long grid =
      tiles < (unsigned long long)p->num_sms ? tiles : (unsigned long long)p->num_sms;
  const TcConsts k{p->f.q, p->f.qinv};
  const char* tab = static_cast<const char*>(p->d_tcw);  // forward, inverse, this inverse
  return launch_chained(ntt_mul_tc_kernel, dim3((unsigned)grid), THREADS, SMEM_BYTES, s, map_a, map_b,
                        map_out, a, b, (unsigned long long)npolys,
                        reinterpret_cast<const uint4*>(tab),
                        reinterpret_cast<const uint4*>(tab + 2 * WMAT), k, p->d_err);
}

}  // namespace grid
