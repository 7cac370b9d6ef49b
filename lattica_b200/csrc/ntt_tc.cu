// Tensor-core twisted negacyclic NTT / INTT for d = 64 (tcgen05, kind::i8).
//
// Reference path replaced: TwistedNttPlan::{forward,inverse}_in_place_trusted
// (algebra/src/poly/ntt.rs:75-104), bit-exact.
//
// The transform is a linear map over Z_q: natural-order slot j of the forward
// output is sum_k x_k psi^((2j+1) k) and the inverse is its inverse matrix
// (d^-1 folded in). Both run as exact integer matrix products on the 8-bit
// tensor cores:
//  * a tile of 128 polynomials is read as a 128 x 256 byte matrix in its
//    natural memory order, byte 4k + i = byte i of word x_k;
//  * with W' = W * 2^32 mod q (Montgomery form) and W^(i) = 2^(8i) W' mod q,
//    B[64 l + j][4k + i] = byte l of W^(i)[j][k]. Then the MMA product
//    E[64 l + j] = sum_{k,i} byte_i(x_k) byte_l(W^(i)[j][k]) satisfies
//    sum_k W'[j][k] x_k = sum_l 2^(8l) E_l[j] (mod q), each E entry
//    < 256 * 255^2 < 2^24 (exact in int32): eight MMAs (M = 128, N = 256,
//    K = 32) per transform, straight from the TMA-loaded tile;
//  * the epilogue forms v = E_0 + 2^8 E_1 + 2^16 E_2 + 2^24 E_3 < 2^49 and
//    one Montgomery reduction returns the canonical word.
// Operands use the 128-byte-swizzled K-major layout that TMA writes: a 128 x
// 256 byte tile is two boxes (K bytes 0-127, 128-255) of 128-byte rows, row r
// of a box at 128 r with 16-byte chunk c at position c ^ (r % 8).
// One persistent CTA per SM: warp 17 moves data (TMA loads of input tiles into a
// ring of four buffers, TMA stores of the results that the epilogue leaves in them,
// L2 prefetch), warp 16 issues the MMAs into two sets of tensor-memory columns in
// turn, warps 0-15 reduce one tile while the next is multiplied. Epilogue warp w owns
// tensor-memory lanes 32 (w % 4) .. + 31 (its rows) and columns 16 (w / 4) .. + 15 of
// each E_l block. The B matrix comes by one bulk copy beside the first tiles' loads.
// Bound by HBM: 512 bytes a polynomial. At 2^22
// polynomials in place 0.36 ms forward and 0.34 inverse (0.91 and 0.97 of the measured
// rate); with two buffers and one set of columns 0.39 and 0.44. A buffer is refilled once
// the store issued before the newest one has read it: a point-major store (64 rows of 512
// bytes) takes a microsecond to do so, and with the loader waiting for each as it issued
// it 6.9 million polynomials took 0.725 ms; 0.552 so (0.98 of the measured rate).
// Every wait is bounded. Products INTT(NTT(a) (.) b) have a kernel of their own
// (ntt_mul_tc.cu).
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_tc.cuh"
#include "ntt_tc_common.cuh"

namespace grid {
namespace {

using namespace tcx;

constexpr int D = 64;
constexpr int NBUF = 4;
// Offsets from the 1 KB-aligned base of dynamic shared memory.
constexpr uint32_t OFF_XA = 0;                     // input tiles, then their results
constexpr uint32_t OFF_W = OFF_XA + NBUF * TILE;   // B matrix
constexpr uint32_t OFF_BAR = OFF_W + WMAT;
constexpr uint32_t SMEM_BYTES = OFF_BAR + (2 * NBUF + 5) * 8 + 16 + 1024;  // + alignment slack
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

enum Bar : int {
  AFULL = 0,             // [4] input tile landed in buffer i
  STAGED = AFULL + NBUF, // [4] result tile written into buffer i
  FDONE = STAGED + NBUF, // [2] transform done into column set i
  FREAD = FDONE + 2,     // [2] column set read
  WFULL = FREAD + 2,     // B matrix landed
  NBARS
};

// MODE_FWD / MODE_INV / MODE_FWD_PM. Tile j of this CTA uses buffer j % 4 and column set
// j % 2: the MMA warp transforms it once it landed and tile j - 2's columns are read,
// the epilogue overwrites the buffer with the result, the loader stores it and loads
// tile j + 4 there. A barrier's next phase always needs an action of its waiter, so no
// parity wait can meet a barrier two phases on.
template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
    ntt_tc_kernel(const __grid_constant__ CUtensorMap tmap_a,
                  const __grid_constant__ CUtensorMap tmap_out, const uint32_t* a,
                  unsigned long long npolys, const uint4* __restrict__ wtab, const TcConsts k,
                  int* __restrict__ err, const uint4* ptiles,
                  unsigned long long nptiles, uint32_t row_polys) {
  constexpr bool kPm = MODE == MODE_FWD_PM;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(bars + NBARS);

  if (warp == MMA_WARP) {
    if (lane == 0) {
      for (int i = 0; i < NBUF; ++i) {
        mbar_init(&bars[AFULL + i], 1);
        mbar_init(&bars[STAGED + i], EPI_WARPS);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&bars[FDONE + i], 1);
        mbar_init(&bars[FREAD + i], EPI_WARPS);
      }
      mbar_init(&bars[WFULL], 1);
      fence_mbar_init();
      tc::fence_async_smem();
      mbar_arrive_expect_tx(&bars[WFULL], WMAT);
      bulk_load(sm + OFF_W, wtab + (MODE == MODE_INV ? WMAT / 16 : 0), WMAT, &bars[WFULL]);
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

  // Point-major mode with a tile list (ptiles): tile t reads 128 polys from
  // row x, stores them at column y, and rows from z on (past an instance) as 0.
  // With row_polys the tiles stay within rows of that many polys: a tile's result box
  // ends at its row's end (the 3D output map clips it), tile t / row_tiles being the row.
  const bool listed = kPm && ptiles != nullptr;
  const bool by_row = kPm && row_polys != 0;
  const uint32_t row_tiles = by_row ? (row_polys + ROWS - 1) / ROWS : 1u;
  const unsigned long long ntiles = listed || by_row ? nptiles : (npolys + ROWS - 1) / ROWS;
  const uint32_t n = blockIdx.x < ntiles
                         ? (uint32_t)((ntiles - 1 - blockIdx.x) / gridDim.x + 1)
                         : 0u;  // tiles of this CTA
  auto tile_index = [&](uint32_t j) -> unsigned long long {
    return (unsigned long long)blockIdx.x + (unsigned long long)j * gridDim.x;
  };
  // first source row / destination row (point-major: column) of tile j
  auto tile_row0 = [&](uint32_t j) -> unsigned long long {
    if (by_row) {
      const uint32_t t = (uint32_t)tile_index(j);
      return (unsigned long long)(t / row_tiles) * row_polys + (t % row_tiles) * ROWS;
    }
    return listed ? load_dep(&ptiles[tile_index(j)].x) : tile_index(j) * ROWS;
  };
  auto tile_out0 = [&](uint32_t j) -> unsigned long long {
    return listed ? load_dep(&ptiles[tile_index(j)].y) : tile_index(j) * ROWS;
  };
  auto tile_valid = [&](uint32_t j) -> uint32_t {
    return listed ? load_dep(&ptiles[tile_index(j)].z) : (uint32_t)ROWS;
  };

  if (warp == LOAD_WARP) {
    // ------------------------------------------------------------ loader
    if (lane == 0) {
      uint32_t loads = 0;
      bool ok = true;
      auto prefetch = [&](uint32_t j) {
        if (j >= n) return;
        const unsigned long long r0 = tile_row0(j), left = npolys - r0;
        prefetch_l2(a + r0 * D, (uint32_t)((left < ROWS ? left : ROWS) * D * 4));
      };
      auto load = [&](uint32_t j) {
        const uint32_t dst = s0 + OFF_XA + (j % NBUF) * TILE;
        uint64_t* bar = &bars[AFULL + j % NBUF];
        mbar_arrive_expect_tx(bar, TILE);
        tma_load_2d(dst, &tmap_a, 0, (int)tile_row0(j), smem_addr(bar));
        tma_load_2d(dst + BOX, &tmap_a, 32, (int)tile_row0(j), smem_addr(bar));
        ++loads;
        prefetch(j + 2);
      };
      for (uint32_t j = 0; j < n && j < (uint32_t)NBUF; ++j) load(j);
      for (uint32_t j = 0; j < n; ++j) {
        const uint32_t src = s0 + OFF_XA + (j % NBUF) * TILE;
        if (!(ok = mbar_wait(&bars[STAGED + j % NBUF], (j / NBUF) & 1, err))) break;
        if (by_row) {
          const uint32_t tr = (uint32_t)tile_index(j);
          tma_store_3d(&tmap_out, (int)((tr % row_tiles) * ROWS), (int)(tr / row_tiles), 0, src);
        } else if constexpr (kPm) {  // [64 points][128 polys] -> columns of the [d][npolys] output
          tma_store_2d(&tmap_out, (int)tile_out0(j), 0, src);
        } else {
          tma_store_2d(&tmap_out, 0, (int)tile_row0(j), src);
          tma_store_2d(&tmap_out, 32, (int)tile_row0(j), src + BOX);
        }
        bulk_commit();
        // not the store just issued, but the one before it frees its buffer
        if (j >= 1 && j - 1 + NBUF < n) {
          bulk_wait_read_older();
          load(j - 1 + NBUF);
        }
      }
      bulk_wait_all();
      if (!ok)  // no copy may still be writing shared memory when the CTA exits
        for (uint32_t i = 0; i < NBUF; ++i) {
          const uint32_t uses = loads > i ? (loads - i + NBUF - 1) / NBUF : 0;
          if (uses) mbar_wait_sleep(&bars[AFULL + i], (uses - 1) & 1, err);
        }
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------ MMA issue
    uint32_t issued = 0;
    if (lane == 0) {
      bool ok = mbar_wait(&bars[WFULL], 0, err);
      for (uint32_t j = 0; ok && j < n; ++j) {
        ok = mbar_wait(&bars[AFULL + j % NBUF], (j / NBUF) & 1, err);
        if (ok && j >= 2) ok = mbar_wait(&bars[FREAD + (j & 1)], ((j >> 1) - 1) & 1, err);
        if (!ok) break;
        tc::fence_after_sync();
        issue_transform(tbase + 256 * (j & 1), s0 + OFF_XA + (j % NBUF) * TILE, s0 + OFF_W);
        tc::mma_commit(&bars[FDONE + (j & 1)]);
        ++issued;
      }
      // every MMA issued is done before shared and tensor memory are released
      for (uint32_t i = 0; i < 2; ++i) {
        const uint32_t uses = issued > i ? (issued - i + 1) / 2 : 0;
        if (uses) mbar_wait_sleep(&bars[FDONE + i], (uses - 1) & 1, err);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue
    const uint32_t wl = warp & 3, cq = warp >> 2;
    const uint32_t row = 32 * wl + lane;
    const uint32_t lane_off = ((32 * wl) << 16) + 16 * cq;
    for (uint32_t j = 0; j < n; ++j) {
      if (!lane0_wait(&bars[FDONE + (j & 1)], (j >> 1) & 1, lane, err)) break;
      tc::fence_after_sync();
      uint32_t res[16];
      reduce16(tbase + 256 * (j & 1) + lane_off, k, res, [&] {
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[FREAD + (j & 1)]);  // columns free for tile j + 2
      });
      // 16 words (columns 16 cq .. + 15 of this row) over the input tile, swizzled; the
      // point-major mode writes the tile transposed, [point][row] (a warp's 32
      // rows of one point are 32 consecutive words: no bank conflict)
      unsigned char* tile = sm + OFF_XA + (j % NBUF) * TILE;
      if constexpr (kPm) {
        uint32_t* t = reinterpret_cast<uint32_t*>(tile);
        const bool keep = row < tile_valid(j);
#pragma unroll
        for (int c = 0; c < 16; ++c) t[(16 * cq + c) * ROWS + row] = keep ? res[c] : 0u;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(tile + sw128(row, cq >> 1, (cq & 1) * 4 + c, BOX)) =
              make_uint4(res[4 * c], res[4 * c + 1], res[4 * c + 2], res[4 * c + 3]);
      }
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[STAGED + j % NBUF]);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
}

// The point-major mode's layout: ptiles / nptiles / ps_out, a tile list over
// [64][ps_out]; row_polys, rows of that many polys, npolys / row_polys of them, at
// [64][rows][pm_stride(row_polys)]; neither, consecutive tiles over [64][npolys]
// (npolys a multiple of 4).
template <int MODE>
int run_tc(const grid_gpu_plan* p, const uint32_t* a, uint32_t* out, size_t npolys,
           cudaStream_t s, const uint4* ptiles = nullptr,
           unsigned long long nptiles = 0, unsigned long long ps_out = 0,
           uint32_t row_polys = 0) {
  EncodeTiled enc = encoder();
  if (!enc) return GRID_ERR_CUDA;
  // Rows of 64 words, boxes of 32 words x 128 rows with 128-byte swizzle.
  CUtensorMap map_a, map_out;
  const cuuint64_t dims[2] = {64, (cuuint64_t)npolys};
  const cuuint64_t strides[1] = {256};
  const cuuint32_t box[2] = {32, ROWS};
  const cuuint32_t estr[2] = {1, 1};
  for (int m = 0; m < 2; ++m)
    if (enc(m ? &map_out : &map_a, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2,
            m ? (void*)out : (void*)const_cast<uint32_t*>(a), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return GRID_ERR_CUDA;
  if (MODE == MODE_FWD_PM && row_polys) {
    const cuuint64_t rows = npolys / row_polys, ld = pm_stride(row_polys);
    const cuuint64_t rdims[3] = {row_polys, rows, 64};
    const cuuint64_t rstrides[2] = {ld * 4, rows * ld * 4};
    const cuuint32_t rbox[3] = {ROWS, 1, 64};
    const cuuint32_t rstr[3] = {1, 1, 1};
    if (enc(&map_out, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, (void*)out, rdims, rstrides, rbox, rstr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return GRID_ERR_CUDA;
    nptiles = rows * ((row_polys + ROWS - 1) / ROWS);
  } else if (MODE == MODE_FWD_PM) {
    // output [64 points][ps], ps a multiple of 4 (rows of whole 16-byte units); one
    // box of 128 polys x 64 points per tile
    const cuuint64_t ps = ps_out ? ps_out : (cuuint64_t)npolys;
    const cuuint64_t pdims[2] = {ps, 64};
    const cuuint64_t pstrides[1] = {ps * 4};
    const cuuint32_t pbox[2] = {ROWS, 64};
    if (enc(&map_out, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)out, pdims, pstrides, pbox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return GRID_ERR_CUDA;
  }
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  const int st =
      prepare_kernel(ntt_tc_kernel<MODE>, SMEM_BYTES, THREADS, p->device, bps_cache, &bps);
  if (st) return st;
  const unsigned long long tiles = nptiles ? nptiles : (npolys + ROWS - 1) / ROWS;
  const unsigned long long grid =
      tiles < (unsigned long long)p->num_sms ? tiles : (unsigned long long)p->num_sms;
  TcConsts k;
  k.q = p->f.q;
  k.qinv = p->f.qinv;
  return launch_chained(ntt_tc_kernel<MODE>, dim3((unsigned)grid), THREADS, SMEM_BYTES, s, map_a,
                        map_out, a, (unsigned long long)npolys,
                        reinterpret_cast<const uint4*>(p->d_tcw), k, p->d_err, ptiles, nptiles,
                        row_polys);
}

}  // namespace

// The driver's tensor-map encoder, looked up once through the runtime (the
// library does not link the driver library directly).
tcx::EncodeTiled tcx::encoder() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  });
  return fn;
}

bool ntt_tc_available(const grid_gpu_plan* p) { return p->d == 64 && p->d_tcw != nullptr; }

int launch_ntt_tc_pm_tiles(const grid_gpu_plan* p, const uint32_t* a, size_t npolys,
                           uint32_t* out, unsigned long long ps_out, const uint4* ptiles,
                           unsigned long long nptiles, cudaStream_t s) {
  if (nptiles == 0) return GRID_OK;
  if (!ptiles || a == out) return GRID_ERR_INVALID_PARAMETERS;
  // TMA coordinates (source rows, destination columns) are 32-bit; the row
  // stride of the [64][ps_out] output is a multiple of 16 bytes
  if (npolys > (size_t)INT32_MAX - ROWS || ps_out > (unsigned long long)INT32_MAX - ROWS ||
      ps_out % 4)
    return GRID_ERR_INVALID_PARAMETERS;
  return run_tc<MODE_FWD_PM>(p, a, out, npolys, s, ptiles, nptiles, ps_out);
}

int launch_ntt_tc_pm(const grid_gpu_plan* p, const uint32_t* a, size_t rows, size_t n,
                     uint32_t* out, cudaStream_t s) {
  const size_t npolys = rows * n;
  if (npolys == 0) return GRID_OK;
  // tiles of other CTAs still read the input while a tile's columns land
  if (a == out) return GRID_ERR_INVALID_PARAMETERS;
  if (npolys > (size_t)INT32_MAX - ROWS) return GRID_ERR_INVALID_PARAMETERS;  // TMA coordinates
  // rows of whole 16-byte units follow one another without a gap: one long row, whose
  // tiles need not end with each of them
  return run_tc<MODE_FWD_PM>(p, a, out, npolys, s, nullptr, 0, 0,
                             n % 4 ? (uint32_t)n : 0u);
}

int launch_ntt_tc(const grid_gpu_plan* p, int mode, const uint32_t* a, uint32_t* out,
                  size_t npolys, cudaStream_t s) {
  if (npolys == 0) return GRID_OK;
  if (npolys > (size_t)INT32_MAX - ROWS) return GRID_ERR_INVALID_PARAMETERS;  // TMA row coordinate
  switch (mode) {
    case MODE_FWD: return run_tc<MODE_FWD>(p, a, out, npolys, s);
    case MODE_INV: return run_tc<MODE_INV>(p, a, out, npolys, s);
    default: return GRID_ERR_INVALID_PARAMETERS;
  }
}

// B matrices in the tiles' 128-byte-swizzled K-major layout, 64 KB per
// transform (256 rows x 256 K bytes, two boxes of 128 K bytes): row
// n = 64 l + j, K byte 4k + i holds byte l of W^(i)[j][k] = 2^(8i) W'[j][k]
// mod q, W' the transform matrix in Montgomery form. Forward, then inverse.
void build_tc_tables(uint32_t q, uint32_t d, uint64_t psi, uint64_t ninv,
                     std::vector<unsigned char>& out) {
  out.assign(2 * WMAT, 0);
  auto mulm = [q](uint64_t x, uint64_t y) { return (uint64_t)((unsigned __int128)x * y % q); };
  // psi^e, e < 2 d, in Montgomery form; psi^-e is psi^(2d - e)
  std::vector<uint64_t> pw(2 * d);
  pw[0] = ((uint64_t)1 << 32) % q;
  for (uint32_t e = 1; e < 2 * d; ++e) pw[e] = mulm(pw[e - 1], psi);
  for (uint32_t j = 0; j < d; ++j)
    for (uint32_t kk = 0; kk < d; ++kk) {
      // forward: slot j <- x_k psi^((2j+1)k); inverse: out_j <- X_k d^-1 psi^-((2k+1)j)
      const uint32_t ef = ((2 * j + 1) * kk) % (2 * d);
      const uint32_t ei = (2 * d - ((2 * kk + 1) * j) % (2 * d)) % (2 * d);
      uint64_t w[2] = {pw[ef], mulm(pw[ei], ninv)};
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t kb = 4 * kk + i, h = kb / 128, kc = kb % 128;
        for (uint32_t l = 0; l < 4; ++l) {
          const uint32_t n = 64 * l + j;
          const uint32_t off = sw128(n, h, kc / 16, WMAT / 2) + kc % 16;
          for (int t = 0; t < 2; ++t) out[t * WMAT + off] = (unsigned char)(w[t] >> (8 * l));
        }
        for (int t = 0; t < 2; ++t) w[t] = mulm(w[t], 256);  // next byte: times 2^8
      }
    }
}

}  // namespace grid
