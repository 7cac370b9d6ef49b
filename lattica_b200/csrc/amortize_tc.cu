// The amortized witness on the tensor cores for d = 64 (tcgen05, kind::i8):
//     z_j = sum_i c_i s_ij 2^-32 mod (X^64 + 1, q),  j < n, i < r,
// without a transform of the witness (compute_amortized_witness,
// labrador/src/main_protocol/amortization.rs:61-84).
//
// A product by c_i is a linear map of the 64 coefficients of s_ij: as in the transform
// (ntt_tc.cu), a tile of 128 polynomials is a 128 x 256 byte matrix A in its natural
// order, byte 4m + b = byte b of coefficient m, and with c~ the negacyclic extension of
// c_i (c~_t = -c_(t + 64) for t < 0) and x_b = 2^(8b) c~_(k - m) mod q,
//     B[l][k][4m + b] = byte l of x_b
// makes sum_l 2^(8l) (A B^T)[l][k] coefficient k of the product mod q. The sums over the i
// of a CTA accumulate in tensor memory (at most 64 of them: below 2^30), and one reduction
// ends them all.
//
// B depends on k - m alone. With the outputs in reverse (row k' = 63 - k) its words
// depend on k' + m, so the 8-row x 16-byte core matrices at (k' / 8, m / 4) on
// 2 (k' / 8) + m / 4: 30 of them per plane l instead of 128, and the descriptor's strides
// are two and one of them. A whole matrix is 15 KB and four MMAs of 64 columns per 32
// bytes of K take the place of one of 256 (1536 cycles a tile and i instead of 1010; the
// 64 KB of the whole matrix would take longer to write).
//
// A CTA takes one tile of 128 polys and a range of i. Warp 9 loads the tiles of s (TMA, 128-byte
// swizzle), warps 0-7 build the matrices, warp 8 issues the MMAs, warps 0-7 reduce the
// result. Where n gives fewer tiles than SMs the range is split and a second kernel adds
// the splits. Bound: the MMAs (1536 cycles a step of 0.8 us), at small sizes the chain of
// launch, first load, steps and reduction. r = 64, n = 2048: 52 us a call with the
// transforms of s and c, the products per point and the inverse, 20 now; n = 100000: 1372
// and 470; r = 6, n = 100: 35 and 19; r = 3, n = 100000: 131 and 47. r = 5000, n = 10: 650 to 730
// us with the chain, one thread a word over all i, 76 now. Plans without the tensor-core
// transform and more than 2^31 polys keep the chain of transforms.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_tc.cuh"
#include "ntt_tc_common.cuh"

namespace grid {
namespace {

using namespace tcx;

constexpr int D = 64;
constexpr int kBuildWarps = 8;               // and the epilogue
constexpr int kBuilders = kBuildWarps * 32;
constexpr int kMma = kBuildWarps, kLoad = kBuildWarps + 1;
constexpr int kThreads = (kBuildWarps + 2) * 32;
constexpr int NA = 4, NB = 3;                // tiles of s, matrices
constexpr int kCores = 30;                   // per plane
constexpr uint32_t kPlane = kCores * 128, kMat = 4 * kPlane;
constexpr int kMaxSum = 64;                  // i per CTA: 64 * 2^24 stays below 2^31
constexpr size_t kMaxR = 65535u * kMaxSum;   // splits in the grid's second dimension
constexpr uint32_t OFF_B = NA * TILE;
constexpr uint32_t OFF_T = OFF_B + NB * kMat;          // [2][4 planes][128] words by k' + m
constexpr uint32_t OFF_BAR = OFF_T + 2 * 4 * 128 * 4;
constexpr uint32_t SMEM = OFF_BAR + (2 * NA + 2 * NB + 1) * 8 + 16 + 1024;  // + alignment slack
static_assert(SMEM <= 232448, "shared memory budget");
static_assert(kBuilders >= 128, "one builder per word of c~");

struct Consts {
  uint4 w, wq;  // 2^(8b) 2^32 mod q and companions
};

// The builder warps' own barrier (named barrier 1; the CTA's is 0).
__device__ __forceinline__ void builders_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(kBuilders) : "memory");
}

__global__ void __launch_bounds__(kThreads, 1)
    amortize_tc_kernel(const __grid_constant__ CUtensorMap map_s, const uint32_t* c,
                       uint32_t* __restrict__ out, uint32_t r, uint32_t n, const Consts w,
                       const FieldParams f, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + OFF_BAR);  // [NA] tile landed
  uint64_t* afree = full + NA;                                 // [NA] its MMAs done
  uint64_t* built = afree + NA;                                // [NB] matrix written
  uint64_t* bfree = built + NB;                                // [NB] its MMAs done
  uint64_t* done = bfree + NB;                                 // every MMA done
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == kMma) {
    tc::tmem_alloc(taddr_slot, 256);
    tc::tmem_relinquish();
    if (lane == 0) {
      for (int i = 0; i < NA; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&afree[i], 1);
      }
      for (int i = 0; i < NB; ++i) {
        mbar_init(&built[i], kBuildWarps);
        mbar_init(&bfree[i], 1);
      }
      mbar_init(done, 1);
      fence_mbar_init();
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  grid_dep_launch();
  grid_dep_wait();  // s and c, and the workspace's previous readers
  const uint32_t j0 = blockIdx.x * ROWS;
  const uint32_t i0 = (uint32_t)((uint64_t)r * blockIdx.y / gridDim.y);
  const uint32_t cnt = (uint32_t)((uint64_t)r * (blockIdx.y + 1) / gridDim.y) - i0;

  if (warp == kLoad) {
    // ------------------------------------------------------------ tiles of s
    if (lane == 0) {
      uint32_t t = 0;
      for (; t < cnt; ++t) {
        const uint32_t sl = t % NA;
        if (t >= (uint32_t)NA && !mbar_wait(&afree[sl], (t / NA - 1) & 1, err)) break;
        const int row = (int)((i0 + t) * n + j0);  // rows past n are another i's, not stored
        mbar_arrive_expect_tx(&full[sl], TILE);
        tma_load_2d(s0 + sl * TILE, &map_s, 0, row, smem_addr(&full[sl]));
        tma_load_2d(s0 + sl * TILE + BOX, &map_s, 32, row, smem_addr(&full[sl]));
      }
      // nothing may still be writing shared memory at exit
      for (uint32_t i = 0; i < (uint32_t)NA; ++i) {
        const uint32_t uses = t > i ? (t - i + NA - 1) / NA : 0;
        if (uses) mbar_wait_sleep(&full[i], (uses - 1) & 1, err);
      }
    }
    __syncwarp();
  } else if (warp == kMma) {
    // ------------------------------------------------------------ MMA issue
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_u8(ROWS, D);
      for (uint32_t t = 0; t < cnt; ++t) {
        const uint32_t sl = t % NA, bs = t % NB;
        if (!mbar_wait(&full[sl], (t / NA) & 1, err) || !mbar_wait(&built[bs], (t / NB) & 1, err))
          break;
        tc::fence_after_sync();
        const uint64_t db = tc::smem_desc(s0 + OFF_B + bs * kMat, 128, 256);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const uint64_t da = desc_sw128(s0 + sl * TILE + (s >> 2) * BOX + 32 * (s & 3));
#pragma unroll
          for (int l = 0; l < 4; ++l)
            tc::mma_u8(tbase + D * l, da, tc::desc_plus(db, l * kPlane + 256 * s), idesc,
                       (t | (uint32_t)s) != 0);
        }
        tc::mma_commit(&afree[sl]);
        tc::mma_commit(&bfree[bs]);
      }
      tc::mma_commit(done);
      mbar_wait_sleep(done, 0, err);  // before shared and tensor memory are released
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ matrices
    const int tid = threadIdx.x;
    bool ok = true;
    uint32_t next = 0;
    // word e = k' + m of the matrix: c~_(63 - e)
    auto load = [&](uint32_t t) {
      next = tid < 127 && t < cnt
                 ? load_dep(c + (unsigned long long)(i0 + t) * D + ((127 - tid) & 63))
                 : 0u;
    };
    load(0);
    for (uint32_t t = 0; t < cnt; ++t) {
      uint32_t* words = reinterpret_cast<uint32_t*>(sm + OFF_T) + (t & 1) * 512;
      if (tid < 128) {  // word 127 is zero, read by no row
        uint32_t x[4] = {mont_c(next, w.w.x, w.wq.x, f.q), mont_c(next, w.w.y, w.wq.y, f.q),
                         mont_c(next, w.w.z, w.wq.z, f.q), mont_c(next, w.w.w, w.wq.w, f.q)};
        if (tid > 63) {
#pragma unroll
          for (int b = 0; b < 4; ++b) x[b] = x[b] ? f.q - x[b] : 0u;
        }
        const uint32_t lo = __byte_perm(x[0], x[1], 0x5140), hi = __byte_perm(x[2], x[3], 0x5140);
        const uint32_t lo2 = __byte_perm(x[0], x[1], 0x7362), hi2 = __byte_perm(x[2], x[3], 0x7362);
        words[tid] = __byte_perm(lo, hi, 0x5410);
        words[128 + tid] = __byte_perm(lo, hi, 0x7632);
        words[256 + tid] = __byte_perm(lo2, hi2, 0x5410);
        words[384 + tid] = __byte_perm(lo2, hi2, 0x7632);
        load(t + 1);
      }
      const uint32_t bs = t % NB;
      if (ok && t >= (uint32_t)NB) ok = lane0_wait(&bfree[bs], (t / NB - 1) & 1, lane, err);
      builders_sync();
      if (!ok) continue;  // the other warps still meet at the barrier
      unsigned char* mat = sm + OFF_B + bs * kMat;
      for (int u = tid; u < 4 * kCores * 8; u += kBuilders) {
        const int l = u / (kCores * 8), row = u % (kCores * 8);  // core row / 8, its row % 8
        const uint32_t* src = words + 128 * l + 4 * (row >> 3) + (row & 7);
        *reinterpret_cast<uint4*>(mat + u * 16) = make_uint4(src[0], src[1], src[2], src[3]);
      }
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&built[bs]);
    }
    // ------------------------------------------------------------ result
    bool got = true;
    if (lane == 0) got = mbar_wait_sleep(done, 0, err);
    __syncwarp();
    ok = ok && __shfl_sync(0xffffffffu, got, 0);
    if (ok) {
      tc::fence_after_sync();
      const uint32_t quarter = warp & 3, half = warp >> 2;
      const uint32_t j = j0 + 32 * quarter + lane;
      uint32_t* dst = out + ((unsigned long long)blockIdx.y * n + j) * D;
#pragma unroll 1
      for (uint32_t n0 = 32 * half; n0 < 32 * half + 32; n0 += 8) {
        uint32_t e[4][8], z[8];
#pragma unroll
        for (int l = 0; l < 4; ++l)
          tc::tmem_ld8(tc::tmem_addr(tbase, 32 * quarter, D * l + n0), e[l]);
        tc::tmem_ld_wait32(e);
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          uint64_t v = mad_wide(e[1][x], 256u, (uint64_t)e[0][x]);
          v = mad_wide(e[2][x], 65536u, v);
          v = mad_wide(e[3][x], 16777216u, v);
          z[7 - x] = redc64(v, f.q, f.qinv);  // columns are the coefficients in reverse
        }
        if (j < n) {
          uint4* at = reinterpret_cast<uint4*>(dst + 56 - n0);
          at[0] = make_uint4(z[0], z[1], z[2], z[3]);
          at[1] = make_uint4(z[4], z[5], z[6], z[7]);
        }
        __syncwarp();  // the whole warp issues the next loads
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kMma) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 256);
  }
}

// z = the sum of the splits' words mod q, four words per thread.
__global__ void __launch_bounds__(256) amortize_sum_kernel(const uint4* part,
                                                           uint4* __restrict__ z,
                                                           unsigned long long words4, int splits,
                                                           uint32_t q) {
  grid_dep_launch();
  grid_dep_wait();
  const unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= words4) return;
  uint4 a = load_dep(part + i);
#pragma unroll 8
  for (int s = 1; s < splits; ++s) {
    const uint4 b = load_dep(part + s * words4 + i);
    a = make_uint4(add_canon(a.x, b.x, q), add_canon(a.y, b.y, q), add_canon(a.z, b.z, q),
                   add_canon(a.w, b.w, q));
  }
  z[i] = a;
}

}  // namespace

// Splits of the range of i: the least number of rounds over the SMs times the steps of a
// CTA, which starts and ends in about as long as four steps (0.8 us each).
int amortize_tc_splits(size_t r, size_t n, int num_sms) {
  const size_t tiles = (n + ROWS - 1) / ROWS;
  const size_t most = std::min<size_t>(r, (size_t)num_sms);
  size_t best = 0, cost = 0;
  for (size_t s = (r + kMaxSum - 1) / kMaxSum; s <= std::max(most, (r + kMaxSum - 1) / kMaxSum); ++s) {
    const size_t rounds = (tiles * s + num_sms - 1) / num_sms;
    const size_t now = rounds * ((r + s - 1) / s + 4);
    if (!best || now < cost) {
      best = s;
      cost = now;
    }
  }
  return (int)best;
}

bool amortize_tc_fits(const grid_gpu_plan* p, size_t r, size_t n) {
  return ntt_tc_available(p) && r <= kMaxR && r * n <= (size_t)INT32_MAX - ROWS;
}

// part: r x n polys of scratch.
int launch_amortize_tc(const grid_gpu_plan* p, const uint32_t* S, const uint32_t* c, size_t r,
                       size_t n, uint32_t* z, uint32_t* part, cudaStream_t s) {
  EncodeTiled enc = encoder();
  if (!enc) return GRID_ERR_CUDA;
  CUtensorMap map;
  const cuuint64_t dims[2] = {D, (cuuint64_t)(r * n)};
  const cuuint64_t strides[1] = {D * 4};
  const cuuint32_t box[2] = {32, ROWS};
  const cuuint32_t estr[2] = {1, 1};
  if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint32_t*>(S), dims, strides, box,
          estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return GRID_ERR_CUDA;
  static int cache[kMaxDevices] = {};
  int bps = 0;
  int rc = prepare_kernel(amortize_tc_kernel, SMEM, kThreads, p->device, cache, &bps);
  if (rc) return rc;
  Consts w;
  uint32_t x[4], xq[4];
  for (int b = 0; b < 4; ++b) {
    x[b] = (uint32_t)(((unsigned __int128)1 << (32 + 8 * b)) % p->f.q);
    xq[b] = x[b] * p->f.qinv;
  }
  w.w = make_uint4(x[0], x[1], x[2], x[3]);
  w.wq = make_uint4(xq[0], xq[1], xq[2], xq[3]);
  const int splits = amortize_tc_splits(r, n, p->num_sms);
  // z may lie over s or c: CTAs still read those while the first ones store
  auto over = [&](const uint32_t* x, size_t polys) {
    return z < x + polys * D && x < z + n * D;
  };
  const bool direct = splits == 1 && !over(S, r * n) && !over(c, r);
  const unsigned tiles = (unsigned)((n + ROWS - 1) / ROWS);
  rc = launch_chained(amortize_tc_kernel, dim3(tiles, (unsigned)splits), kThreads, SMEM, s, map, c,
                      direct ? z : part, (uint32_t)r, (uint32_t)n, w, p->f, p->d_err);
  if (rc || direct) return rc;
  const unsigned long long words4 = (unsigned long long)n * (D / 4);
  return launch_chained(amortize_sum_kernel, dim3((unsigned)((words4 + 255) / 256)), 256, 0, s,
                        reinterpret_cast<const uint4*>(part), reinterpret_cast<uint4*>(z), words4,
                        splits, p->f.q);
}

}  // namespace grid
