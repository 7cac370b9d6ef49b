// Grouped contractions over point-major evaluations: many independent
// commitments t_i = A[:, :n_i] s_i of uneven length n_i (uneven batched
// commitments) per evaluation point e,
//     out_e[i][r] = sum_{k < n_i} s_i,e[k] * A_e[r][k] * 2^-32 (mod q),
// the point-major counterpart of grouped_tc.cu. The witnesses' forward
// transform stored [point][poly] (ntt_tc.cu, point-major mode over a tile
// list); matrices keep point-major evaluations [point][row][ld].
//
// A work item is (tile, K range, one evaluation point); a tile holds up to 128
// instances of one matrix (the MMA's M), sorted longest first. A tile's words at a point
// lie in blocks of 128: the first block of every instance, then the second of every
// instance that has one, ... (batch.cu), zero past an instance's end. So the K words
// 128 c .. + 127 of all J live instances are J consecutive rows of 512 bytes, and a chunk,
// 32 words of each, is at most four TMA boxes of 8 to 64 rows. Per chunk:
//  * one lane of warp 4 loads it (up to seven rows more, of other instances);
//  * warps 6 and 7 zero the slot's rows from J on as far as they are not zero yet;
//  * warps 0-3 build the byte planes of the matrix rows, from words loaded one chunk
//    ahead: B row c NP + r, K byte 4k + i = byte c - i of A_e[r][k], so that column
//    c NP + r of the product is the sum of its bytes' products of weight 2^(8c), c < 7
//    (emm_pm.cu's method);
//  * one lane of warp 5 issues four MMAs (M 128, N 7 NP, K 32) into a tensor-memory
//    accumulator (two, alternating per item, up to 16 rows; one beyond, where two would
//    leave the SM to one CTA) and commits them to the slots' barriers and, after the
//    item's last chunk, to the accumulator's;
//  * warps 8-11 combine the classes of a finished item, reduce once and add
//    each canonical word into the 64-bit accumulator of its output poly and
//    point, so K ranges of one instance may run in different items.
// CTAs take the work list's items with a grid stride (longest first), every
// role walking the same sequence. Instance rows past a tile's count and B rows
// past the matrix's reach only results that are not stored, so they are never
// cleared. Every wait is bounded.
//
// Bound: reading the evaluations (4.4 TB/s with 8 and 16 rows), then, with 32 rows, the
// construction of the classes. Both launches of 4096 instances of 64 to 8192 polys, by a
// profiler: 480 and 422 us with four warps copying every row's 128 bytes from rows an
// instance apart (cp.async, eight lanes a row: as many issue slots as everything else) and
// one CTA per SM; 271 and 252 with blocks and TMA; 268 and 203 with unscaled classes
// instead of four planes of 2^(8i) A (three modular products a word).
#include <cuda_runtime.h>

#include <algorithm>

#include "batch_tables.cuh"
#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_tc.cuh"
#include "ntt_tc_common.cuh"

namespace grid {
namespace {

using namespace tcx;

constexpr int kGpBuildWarps = 4;
constexpr int kGpLoadWarp = 4, kGpMmaWarp = 5;
constexpr int kGpZeroWarp0 = 6, kGpZeroWarps = 2;
constexpr int kGpEpiWarp0 = 8, kGpEpiWarps = 4;
constexpr int kGpThreads = (kGpEpiWarp0 + kGpEpiWarps) * 32;
constexpr int KCH = 32;     // K words per chunk: one 128-byte swizzled row
constexpr int KBLK = 128;   // K words per block of the evaluations

template <int NP>
struct GpShape {
  static constexpr int NMMA = 7 * NP;            // B rows: seven classes
  static constexpr uint32_t ASLOT = 128u * 128;  // 128 instance rows x 128 bytes
  static constexpr uint32_t BSLOT = NMMA * 128u;
  static constexpr int NSB = 2;
  static constexpr int NACC = NP > 16 ? 1 : 2;   // accumulators
  static constexpr uint32_t kBudget = 112640;  // two CTAs per SM
  static constexpr int NSA = (int)((kBudget - NSB * BSLOT) / ASLOT);
  static constexpr uint32_t OFF_B = NSA * ASLOT;
  static constexpr uint32_t OFF_BAR = OFF_B + NSB * BSLOT;
  static constexpr int NBARS = 3 * NSA + 2 * NSB + 5;
  static constexpr uint32_t SMEM = OFF_BAR + NBARS * 8 + 16 + 1024;  // + alignment slack
  static constexpr uint32_t TCOLS = 256;
  static_assert(NACC * NMMA <= TCOLS && NMMA % 16 == 0, "tensor-memory allocation");
  static_assert(2 * (SMEM + 1024) <= 233472, "two CTAs per SM");
};

// Boxes of 32 words of 64, 32, 16 and 8 rows of the evaluations.
struct GpMaps {
  CUtensorMap box[4];
};

__device__ __forceinline__ uint32_t item_chunks(const WorkDev& w) {
  return (w.k1 - w.k0 + KCH - 1) / KCH;
}

// What the roles know of the K words kc .. + 31 of a tile: J live instances, in the rows
// from `row` on (of 512 bytes) of the point's evaluations, words kc % 128 .. + 31 of each.
struct Chunk {
  uint32_t row, live;
};
__device__ __forceinline__ Chunk chunk_at(const uint4* __restrict__ xtiles, uint32_t x0,
                                          uint32_t kc) {
  const uint32_t w = xtiles[x0 + kc / KBLK].w;
  return Chunk{x0 + (w >> 8), w & 0xFFu};
}

template <int NP>
__global__ void __launch_bounds__(kGpThreads, 2)
    batch_pm_kernel(const __grid_constant__ GpMaps maps, const WorkDev* __restrict__ work,
                    unsigned nwork, const TileDev* __restrict__ tiles,
                    const ItemDev* __restrict__ rows, const MatDev* __restrict__ mats,
                    const uint4* __restrict__ xtiles, unsigned long long* __restrict__ acc, int d,
                    const FieldParams f, int* __restrict__ err) {
  using S = GpShape<NP>;
  constexpr int NSA = S::NSA, NSB = S::NSB, NMMA = S::NMMA, NACC = S::NACC;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + S::OFF_BAR);  // slot's copies landed
  uint64_t* zeroed = full + NSA;                                  // its dead rows are zero
  uint64_t* a_free = zeroed + NSA;                                // slot's MMAs done
  uint64_t* built = a_free + NSA;                                 // B slot written
  uint64_t* b_free = built + NSB;                                 // B slot's MMAs done
  uint64_t* acc_full = b_free + NSB;                              // [2] item's MMAs done
  uint64_t* acc_empty = acc_full + 2;                             // [2] item's results read
  uint64_t* drain = acc_empty + 2;                                // every MMA done (exit)
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == kGpMmaWarp) {
    tc::tmem_alloc(taddr_slot, S::TCOLS);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < NSA; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&zeroed[i], kGpZeroWarps);
      mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < NSB; ++i) {
      mbar_init(&built[i], kGpBuildWarps);
      mbar_init(&b_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], kGpEpiWarps);
    }
    mbar_init(drain, 1);
    fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  bool ok = true;

  if (warp == kGpLoadWarp) {
    // ------------------------------------------------------------ loads
    if (lane == 0) {
      uint32_t gc = 0;  // chunks of this CTA so far
      for (unsigned wi = blockIdx.x; ok && wi < nwork; wi += gridDim.x) {
        const WorkDev w = work[wi];
        const uint32_t x0 = (uint32_t)(rows[tiles[w.tile].first].s_off / KBLK);
        const uint32_t nch = item_chunks(w);
        Chunk ch = chunk_at(xtiles, x0, w.k0);
        for (uint32_t c = 0; c < nch; ++c, ++gc) {
          const uint32_t sl = gc % NSA, kc = w.k0 + c * KCH;
          if (c && kc % KBLK == 0) ch = chunk_at(xtiles, x0, kc);
          if (gc >= (uint32_t)NSA && !(ok = mbar_wait_sleep(&a_free[sl], ((gc / NSA) - 1) & 1, err)))
            break;
          const uint32_t bar = smem_addr(&full[sl]);
          const uint32_t nrows = (ch.live + 7) & ~7u;
          mbar_arrive_expect_tx(&full[sl], nrows * 128);
          uint32_t r = 0;
          for (int b = 0; b < 4; ++b) {  // 64 rows (twice for more than 120), 32, 16, 8
            const uint32_t box = 64u >> b;
            while (nrows - r >= box) {
              tma_load_3d(s0 + sl * S::ASLOT + r * 128, &maps.box[b], (int)(kc % KBLK),
                          (int)(ch.row + r), (int)w.eg, bar);
              r += box;
            }
          }
        }
      }
      // nothing may still be writing shared memory at exit
      for (uint32_t i = 0; i < (uint32_t)NSA; ++i) {
        const uint32_t uses = gc > i ? (gc - i + NSA - 1) / NSA : 0;
        if (uses) mbar_wait_sleep(&full[i], (uses - 1) & 1, err);
      }
    }
    __syncwarp();
  } else if (warp >= kGpZeroWarp0 && warp < kGpZeroWarp0 + kGpZeroWarps) {
    // ------------------------------------------------------------ dead rows
    // A slot remembers from which row on it holds zeros for the current item; the
    // rows up to there that a chunk does not fill with live instances are cleared.
    const uint32_t half = warp - kGpZeroWarp0;
    uint32_t gc = 0, from[NSA];
    for (unsigned wi = blockIdx.x; ok && wi < nwork; wi += gridDim.x) {
      const WorkDev w = work[wi];
      const TileDev tl = tiles[w.tile];
      const uint32_t x0 = (uint32_t)(rows[tl.first].s_off / KBLK);
      const uint32_t nch = item_chunks(w);
#pragma unroll
      for (int i = 0; i < NSA; ++i) from[i] = tl.count;  // the slots' rows hold older data
      Chunk ch = chunk_at(xtiles, x0, w.k0);
      for (uint32_t c = 0; c < nch; ++c, ++gc) {
        const uint32_t sl = gc % NSA, kc = w.k0 + c * KCH;
        if (c && kc % KBLK == 0) ch = chunk_at(xtiles, x0, kc);
        if (!(ok = lane0_wait(&full[sl], (gc / NSA) & 1, lane, err))) break;
        uint32_t end = 0;
#pragma unroll
        for (int i = 0; i < NSA; ++i) {
          if (i == (int)sl) {
            end = from[i];
            from[i] = ch.live;
          }
        }
        end = min(max(end, (ch.live + 7) & ~7u), tl.count);  // the load's last box included
        if (ch.live < end) {
          unsigned char* slot = sm + sl * S::ASLOT;
          for (uint32_t u = ch.live * 8 + half * 32 + lane; u < end * 8; u += 32 * kGpZeroWarps)
            *reinterpret_cast<uint4*>(slot + u * 16) = make_uint4(0, 0, 0, 0);
          fence_proxy_async_smem();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&zeroed[sl]);
      }
    }
  } else if (warp == kGpMmaWarp) {
    // ------------------------------------------------------------ MMA issue
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_u8(128, NMMA);
      uint32_t gc = 0, it = 0;
      for (unsigned wi = blockIdx.x; ok && wi < nwork; wi += gridDim.x, ++it) {
        const uint32_t buf = it % NACC;
        if (it >= NACC && !(ok = mbar_wait_sleep(&acc_empty[buf], (it / NACC - 1) & 1, err))) break;
        tc::fence_after_sync();
        const uint32_t nch = item_chunks(work[wi]);
        for (uint32_t c = 0; c < nch; ++c, ++gc) {
          const uint32_t sl = gc % NSA, bs = gc % NSB;
          if (!(ok = mbar_wait_sleep(&full[sl], (gc / NSA) & 1, err)) ||
              !(ok = mbar_wait_sleep(&zeroed[sl], (gc / NSA) & 1, err)) ||
              !(ok = mbar_wait_sleep(&built[bs], (gc / NSB) & 1, err)))
            break;
          tc::fence_after_sync();
          const uint32_t sa = s0 + sl * S::ASLOT, sb = s0 + S::OFF_B + bs * S::BSLOT;
#pragma unroll
          for (int s = 0; s < 4; ++s)
            tc::mma_u8(tbase + buf * NMMA, desc_sw128(sa + 32 * s), desc_sw128(sb + 32 * s),
                       idesc, (c | (uint32_t)s) != 0);
          tc::mma_commit(&a_free[sl]);
          tc::mma_commit(&b_free[bs]);
        }
        tc::mma_commit(&acc_full[buf]);
      }
      // every MMA done before shared and tensor memory are released (at once
      // if none ran)
      tc::mma_commit(drain);
      mbar_wait_sleep(drain, 0, err);
    }
    __syncwarp();
  } else if (warp < kGpBuildWarps) {
    // ------------------------------------------------------------ B planes
    constexpr int kWords = NP * KCH / (kGpBuildWarps * 32);
    const int n_base = threadIdx.x >> 5, kk = lane;
    uint32_t gc = 0;
    for (unsigned wi = blockIdx.x; ok && wi < nwork; wi += gridDim.x) {
      const WorkDev w = work[wi];
      const MatDev mt = mats[tiles[w.tile].matrix];
      const uint32_t mrows = mt.rows;
      const uint32_t* ye = mt.evals_pm +
                           ((unsigned long long)w.eg * mrows + n_base) * mt.ld_pm;
      const uint32_t nch = item_chunks(w);
      uint32_t next[kWords];
      auto load = [&](uint32_t c) {
        const uint32_t kw = w.k0 + c * KCH + kk;
#pragma unroll
        for (int i = 0; i < kWords; ++i) {
          const uint32_t n = n_base + kGpBuildWarps * i;
          next[i] = c < nch && n < mrows && kw < mt.ld_pm
                        ? __ldg(ye + (unsigned long long)(kGpBuildWarps * i) * mt.ld_pm + kw)
                        : 0u;
        }
      };
      load(0);
      for (uint32_t c = 0; c < nch; ++c, ++gc) {
        const uint32_t bs = gc % NSB;
        uint32_t y[kWords];
#pragma unroll
        for (int i = 0; i < kWords; ++i) y[i] = next[i];
        load(c + 1);
        if (gc >= (uint32_t)NSB && !(ok = lane0_wait(&b_free[bs], ((gc / NSB) - 1) & 1, lane, err)))
          break;
        unsigned char* bt = sm + S::OFF_B + bs * S::BSLOT;
#pragma unroll
        for (int i = 0; i < kWords; ++i) {
          const int n = n_base + kGpBuildWarps * i;
          if (n >= (int)mrows) continue;
          const uint32_t v = __byte_perm(y[i], 0, 0x0123);  // bytes 3, 2, 1, 0
          unsigned char* dst = bt + sw128(n, 0, kk >> 2, 0) + 4 * (kk & 3);
          *reinterpret_cast<uint32_t*>(dst) = v >> 24;
          *reinterpret_cast<uint32_t*>(dst + NP * 128) = v >> 16;
          *reinterpret_cast<uint32_t*>(dst + 2 * NP * 128) = v >> 8;
          *reinterpret_cast<uint32_t*>(dst + 3 * NP * 128) = v;
          *reinterpret_cast<uint32_t*>(dst + 4 * NP * 128) = v << 8;
          *reinterpret_cast<uint32_t*>(dst + 5 * NP * 128) = v << 16;
          *reinterpret_cast<uint32_t*>(dst + 6 * NP * 128) = v << 24;
        }
        fence_proxy_async_smem();  // the planes are read by the tensor cores
        __syncwarp();
        if (lane == 0) mbar_arrive(&built[bs]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3;  // tensor-memory lanes 32 quarter .. + 31
    const uint32_t j = 32 * quarter + lane;
    uint32_t it = 0;
    for (unsigned wi = blockIdx.x; ok && wi < nwork; wi += gridDim.x, ++it) {
      const uint32_t buf = it % NACC;
      const WorkDev w = work[wi];
      const TileDev tl = tiles[w.tile];
      const uint32_t mrows = mats[tl.matrix].rows;
      const unsigned long long toff = j < tl.count ? rows[tl.first + j].t_off : 0ull;
      // the item's whole K loop: sleep in the barrier rather than poll
      bool got = true;
      if (lane == 0) got = mbar_wait_sleep(&acc_full[buf], (it / NACC) & 1, err);
      __syncwarp();
      if (!(ok = __shfl_sync(0xffffffffu, got, 0))) break;
      tc::fence_after_sync();
      const uint32_t taddr = tc::tmem_addr(tbase, 32 * quarter, buf * NMMA);
#pragma unroll 1
      for (int n0 = 0; n0 < (int)mrows; n0 += 8) {
        uint32_t ds[7][8];
#pragma unroll
        for (int c = 0; c < 7; ++c) tc::tmem_ld8(taddr + c * NP + n0, ds[c]);
        tc::tmem_ld_wait7(ds);
        if (j < tl.count) {
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            const uint32_t n = n0 + jj;
            if (n >= mrows) continue;
            atomicAdd(&acc[(toff + n) * (unsigned long long)d + w.eg],
                      (unsigned long long)reduce_classes(ds[0][jj], ds[1][jj], ds[2][jj],
                                                         ds[3][jj], ds[4][jj], ds[5][jj],
                                                         ds[6][jj], f));
          }
        }
        __syncwarp();  // the whole warp issues the next loads
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kGpMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, S::TCOLS);
  }
}

template <int NP>
int launch_np(const grid_gpu_plan* p, const WorkDev* work, unsigned nwork, const TileDev* tiles,
              const ItemDev* items, const MatDev* mats, const uint4* xtiles,
              const uint32_t* s_pm, uint64_t ps, unsigned long long* acc, cudaStream_t s) {
  using S = GpShape<NP>;
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  const int rc = prepare_kernel(batch_pm_kernel<NP>, S::SMEM, kGpThreads, p->device, bps_cache,
                                &bps, true);
  if (rc) return rc;
  // the evaluations as [point][ps / 128 rows][128 words]
  EncodeTiled enc = encoder();
  if (!enc) return GRID_ERR_CUDA;
  GpMaps maps;
  for (int b = 0; b < 4; ++b) {
    const cuuint64_t dims[3] = {KBLK, ps / KBLK, p->d};
    const cuuint64_t strides[2] = {KBLK * 4, ps * 4};
    const cuuint32_t box[3] = {KCH, 64u >> b, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    if (enc(&maps.box[b], CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t*>(s_pm), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return GRID_ERR_CUDA;
  }
  // Two CTAs per SM (GpShape, at most 80 registers). The occupancy query answers 1 for any kernel
  // that allocates tensor memory, whatever its registers and shared memory.
  const unsigned grid = std::min<unsigned>(nwork, 2u * (unsigned)p->num_sms);
  batch_pm_kernel<NP><<<grid, kGpThreads, S::SMEM, s>>>(
      maps, work, nwork, tiles, items, mats, xtiles, acc, (int)p->d,
      p->f, p->d_err);
  return cuda_status(cudaGetLastError());
}

}  // namespace

int launch_batch_pm(const grid_gpu_plan* p, int cls, const WorkDev* work, unsigned nwork,
                    const TileDev* tiles, const ItemDev* items, const MatDev* mats,
                    const uint4* xtiles, const uint32_t* s_pm, uint64_t ps, unsigned long long* acc, cudaStream_t s) {
  if (nwork == 0) return GRID_OK;
  switch (cls) {
    case TC_D16: return launch_np<16>(p, work, nwork, tiles, items, mats, xtiles, s_pm, ps, acc, s);
    case TC_D32: return launch_np<32>(p, work, nwork, tiles, items, mats, xtiles, s_pm, ps, acc, s);
    default: return GRID_ERR_INVALID_PARAMETERS;  // point-major tiles are dense commitments
  }
}

}  // namespace grid
