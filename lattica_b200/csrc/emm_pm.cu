// Evaluation-domain products on the tensor cores over point-major operands:
//     out_e[m][n] = sum_k X_e[m][k] * Y_e[n][k] * 2^-32 (mod q)
// where X_e = X + e M ldx and Y_e = Y + e N ldy hold the words of evaluation
// point e row-major ([point][row][k], row strides of whole 16-byte units): the
// layout the forward transform's point-major mode writes (ntt_tc.cu) and prepared
// matrices keep beside their poly-major evaluations. The products are those of
// emm_tc.cu (the Ajtai commitment's, the Gram matrix's and garbage h's contraction).
//
// Byte planes, without scaling. With x = sum_i 2^(8i) x_i and y = sum_l 2^(8l) y_l in
// bytes, sum_k x_k y_k = sum_s 2^(8s) D_s, D_s = sum_{i+l=s} sum_k x_i y_l, s = 0 .. 6.
// A_i (rows x 128 K bytes per chunk) holds byte i of the X words, the four B_l
// stand one above the other (row l NP + n), so that the product of A_i with all of B is
// added to tensor-memory columns i NP .. (i + 4) NP: class s at columns s NP.
// The planes A_i stand one above the other too: of 33 to 64 rows, P = 2 of them fit the
// 128 rows of one MMA (N = 4 NP), 4 / P MMAs per 32 K words. Rows g ROWS_A + m of
// the product with planes i .. i + P - 1 hold byte i + g, so class s of those rows is at
// columns (s - g) NP, and the row blocks' reduced sums, block g's times 2^(8g), are added
// at the end. D_s < 4 K 255^2 < 2^31 for K <= 8192 per CTA. V = sum_s 2^(8s) D_s <
// 2^80 is reduced once per block. (64 x 64 rows, n = 2048, garbage h and z together:
// 87.4 us with one plane per MMA, 83.7 with two. Of up to 32 rows four would fit, but the
// MMAs are short there and four blocks to reduce cost more: the Gram of r = 30, n = 1021
// 20.9 us with one, 22.8 with four.)
// Planes of 2^(8i) y cost three Montgomery products a word of Y, on eight warps that
// bounded the kernel (about 1500 cycles per 32 K words of a 64-row Gram, MMAs 504); the
// planes are now a 4 x 4 byte transpose of four consecutive words (two byte permutes and
// one store a word, about 250 cycles per 128 K words), and the Gram's planes are its
// A and its B at once. Measured (round of r = 64, n = 2048, the commitment's and the
// Gram's product under ncu, caches cold): 19.8 and 35.8 us before, 16.5 and 18 now.
// Result (m, n) depends only on A row m and B rows l NP + n, so rows past the
// operands' are never cleared: whatever they hold reaches only results that
// are not stored; an A plane shorter than 128 rows is read into whatever follows it.
//
// One CTA per (evaluation point, K range), 10 warps:
//  * warp 8 (one lane) loads the X (and Y) rows of each 128-word chunk with TMA into
//    a ring of raw slots (zero fill past K), refilling a slot once it is transposed;
//  * warps 0-7 write the chunk's planes into a ring of plane slots, once the rows
//    landed and the slot's previous MMAs are done;
//  * warp 9 (one lane) issues 16 / P MMAs (M 128, N 4 NP, K 32) per chunk into tensor
//    memory, cleared beforehand, and commits them to the plane slot's mbarrier;
//  * after the last chunk warps 0-7 combine the classes, reduce, stage the
//    point's results in shared memory and store them contiguously, [split][e]
//    [output], for the sum over K ranges that follows.
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

constexpr int kPmBuildWarps = 8;
constexpr int kPmBuilders = kPmBuildWarps * 32;
constexpr int kPmLoadWarp = kPmBuildWarps;
constexpr int kPmMmaWarp = kPmBuildWarps + 1;
constexpr int kPmThreads = (kPmBuildWarps + 2) * 32;
constexpr int KCH = 128;       // K words per chunk: one 128-byte swizzled row per plane
constexpr int kPmMaxK = 8192;  // K words per CTA: 4 * 8192 * 255^2 < 2^31

// NP: Y rows padded to 16 .. 64; MX: X rows per A plane (8, 64 or 128; the Gram's planes
// are B's, NP rows).
template <int NP, int MX, bool UPPER>
struct PmShape {
  static constexpr int NMMA = 4 * NP;                         // B rows: four byte planes
  static constexpr int ROWS_A = UPPER ? NP : MX;
  static constexpr int P = ROWS_A > 64 || ROWS_A <= 32 ? 1 : 2;  // planes per MMA
  static constexpr int NC = 8 - P;                            // blocks of NP columns
  static constexpr uint32_t XRAW = ROWS_A * KCH * 4u;
  static constexpr uint32_t RAW = XRAW + (UPPER ? 0u : NP * KCH * 4u);  // X rows, Y rows
  static constexpr uint32_t PLANES_A = 4u * ROWS_A * KCH;
  static constexpr uint32_t PLANES = RAW;                     // a byte of plane per byte of word
  static constexpr uint32_t TCOLS = 7 * NP <= 128 ? 128u : 7 * NP <= 256 ? 256u : 512u;
  // As many CTAs per SM (up to four) as tensor memory and one slot of each kind allow;
  // within their shares a second raw slot, then a second plane slot, as they fit (a load
  // takes longer than the MMAs, 1.5 us against 1 for 64 x 64 rows, so it is the raw
  // rows that have to be ahead).
  static constexpr int BY_SMEM = (int)(220u * 1024 / (RAW + PLANES + 2048));
  static constexpr int BY_TMEM = (int)(512 / TCOLS);
  static constexpr int PER_SM = BY_SMEM < BY_TMEM ? (BY_SMEM < 1 ? 1 : BY_SMEM) : BY_TMEM;
  static constexpr uint32_t kBudget = 224u * 1024 / PER_SM - 2048;
  static constexpr int NSX = 2 * RAW + PLANES <= kBudget ? 2 : 1;
  static constexpr int NSP = NSX * RAW + 2 * PLANES <= kBudget ? 2 : 1;
  static constexpr uint32_t OFF_RAW = NSP * PLANES;           // planes first, then raw rows
  static constexpr uint32_t OFF_BAR = OFF_RAW + NSX * RAW;
  static constexpr int NBARS = 2 * NSX + 2 * NSP + 1;
  // the MMA reads 128 rows from its first A plane: the last one's run past its slot
  static constexpr uint32_t END = OFF_BAR + NBARS * 8 + 16;
  static constexpr uint32_t A_END = OFF_RAW - PLANES + ((4u - P) * ROWS_A + 128u) * 128u;
  static constexpr uint32_t SMEM = (END > A_END ? END : A_END) + 1024;  // + alignment slack
  static_assert(SMEM <= 232448, "shared memory budget");
  // the point's results are staged in the first plane slot
  static_assert(PLANES >= P * (UPPER ? (uint32_t)NP * (NP + 1) / 2 : (uint32_t)MX * NP) * 4,
                "staging");
};

// The builder warps' own barrier (named barrier 1; the CTA's is 0).
__device__ __forceinline__ void builders_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(kPmBuilders) : "memory");
}

// One row's 128 words (lane l: words 4 l .. 4 l + 3) as four rows of bytes: plane p at
// dst + p * plane_bytes, its 16-byte chunk l / 4 swizzled.
__device__ __forceinline__ void split_row(const unsigned char* src, unsigned char* planes, int row,
                                          uint32_t plane_bytes, int lane) {
  const uint4 w = *reinterpret_cast<const uint4*>(src + row * (KCH * 4) + lane * 16);
  const uint32_t a = __byte_perm(w.x, w.y, 0x5140), b = __byte_perm(w.z, w.w, 0x5140);
  const uint32_t c = __byte_perm(w.x, w.y, 0x7362), d = __byte_perm(w.z, w.w, 0x7362);
  unsigned char* dst = planes + sw128(row, 0, lane >> 2, 0) + 4 * (lane & 3);
  *reinterpret_cast<uint32_t*>(dst) = __byte_perm(a, b, 0x5410);
  *reinterpret_cast<uint32_t*>(dst + plane_bytes) = __byte_perm(a, b, 0x7632);
  *reinterpret_cast<uint32_t*>(dst + 2 * plane_bytes) = __byte_perm(c, d, 0x5410);
  *reinterpret_cast<uint32_t*>(dst + 3 * plane_bytes) = __byte_perm(c, d, 0x7632);
}

template <int NP, int MX, bool UPPER>
__global__ void __launch_bounds__(kPmThreads)
    emm_pm_kernel(const __grid_constant__ CUtensorMap tmap_x,
                  const __grid_constant__ CUtensorMap tmap_y, uint32_t* __restrict__ part, int M,
                  int N, int K, int k_per_split, uint32_t box_bytes, const FieldParams f,
                  int* __restrict__ err) {
  using S = PmShape<NP, MX, UPPER>;
  constexpr int NSX = S::NSX, NSP = S::NSP, NMMA = S::NMMA, P = S::P;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + S::OFF_BAR);  // raw slot landed
  uint64_t* raw_free = full + NSX;                                // raw slot transposed
  uint64_t* built = raw_free + NSX;                               // plane slot written
  uint64_t* pl_free = built + NSP;                                // plane slot's MMAs done
  uint64_t* done = pl_free + NSP;                                 // every MMA done
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int e = blockIdx.x;
  const int kbeg = blockIdx.y * k_per_split;
  const int kend = min(K, kbeg + k_per_split);
  const int nch = kend > kbeg ? (kend - kbeg + KCH - 1) / KCH : 0;

  if (warp == kPmMmaWarp) {
    tc::tmem_alloc(taddr_slot, S::TCOLS);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < NSX; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&raw_free[i], kPmBuildWarps);
    }
    for (int i = 0; i < NSP; ++i) {
      mbar_init(&built[i], kPmBuildWarps);
      mbar_init(&pl_free[i], 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;
  if (warp < 4) {  // the classes start at zero: MMAs of different A_i share them
#pragma unroll
    for (int c = 0; c < S::NC * NP; c += 16) tc::tmem_zero16(tc::tmem_addr(tbase, 32 * warp, c));
    tc::tmem_st_wait();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  grid_dep_wait();
  grid_dep_launch();

  if (warp == kPmLoadWarp) {
    // ------------------------------------------------------------ TMA loads
    if (lane == 0) {
      int issued = 0;
      for (int c = 0; c < nch; ++c) {
        const int sl = c % NSX;
        if (c >= NSX && !mbar_wait(&raw_free[sl], ((c / NSX) - 1) & 1, err)) break;
        const uint32_t sr = s0 + S::OFF_RAW + sl * S::RAW;
        const uint32_t bar = smem_addr(&full[sl]);
        mbar_arrive_expect_tx(&full[sl], box_bytes);
        tma_load_3d(sr, &tmap_x, kbeg + c * KCH, 0, e, bar);
        if (!UPPER) tma_load_3d(sr + S::XRAW, &tmap_y, kbeg + c * KCH, 0, e, bar);
        ++issued;
      }
      // no copy may still be writing shared memory when the CTA exits
      for (int sl = 0; sl < NSX; ++sl) {
        const int loads = issued > sl ? (issued - sl + NSX - 1) / NSX : 0;
        if (loads) mbar_wait_sleep(&full[sl], (loads - 1) & 1, err);
      }
    }
    __syncwarp();
  } else if (warp == kPmMmaWarp) {
    // ------------------------------------------------------------ MMA issue
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_u8(128, NMMA);
      for (int c = 0; c < nch; ++c) {
        const int ps = c % NSP;
        if (!mbar_wait(&built[ps], (c / NSP) & 1, err)) break;
        tc::fence_after_sync();
        const uint32_t sa = s0 + ps * S::PLANES;
        const uint64_t da = desc_sw128(sa), db = desc_sw128(UPPER ? sa : sa + S::PLANES_A);
        const int steps = min(4, (kend - kbeg - c * KCH + 31) / 32);  // of 32 K bytes
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          if (ks >= steps) break;
#pragma unroll
          for (int i = 0; i < 4; i += P)
            tc::mma_u8(tbase + i * NP, tc::desc_plus(da, i * S::ROWS_A * 128 + 32 * ks),
                       tc::desc_plus(db, 32 * ks), idesc, 1u);
        }
        tc::mma_commit(&pl_free[ps]);
      }
      // completes once every MMA issued above has (at once if none was)
      tc::mma_commit(done);
      mbar_wait_sleep(done, 0, err);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ byte planes
    bool ok = true;
    for (int c = 0; ok && c < nch; ++c) {
      const int sl = c % NSX, ps = c % NSP;
      ok = lane0_wait(&full[sl], (c / NSX) & 1, lane, err);
      if (ok && c >= NSP) ok = lane0_wait(&pl_free[ps], ((c / NSP) - 1) & 1, lane, err);
      if (!ok) break;
      const unsigned char* src = sm + S::OFF_RAW + sl * S::RAW;
      unsigned char* planes = sm + ps * S::PLANES;
#pragma unroll 4
      for (int r = warp; r < M; r += kPmBuildWarps)
        split_row(src, planes, r, S::ROWS_A * 128u, lane);
      if (!UPPER)
#pragma unroll 4
        for (int r = warp; r < N; r += kPmBuildWarps)
          split_row(src + S::XRAW, planes + S::PLANES_A, r, NP * 128u, lane);
      tc::fence_async_smem();  // the planes are read by the tensor cores, the raw slot
      __syncwarp();            // refilled by TMA
      if (lane == 0) {
        mbar_arrive(&built[ps]);
        mbar_arrive(&raw_free[sl]);
      }
    }
    // ------------------------------------------------------------ epilogue
    ok = ok && lane0_wait(done, 0, lane, err);
    tc::fence_after_sync();
    // every builder reaches the barrier below (a failed wait skips only work)
    const int outputs = UPPER ? M * (M + 1) / 2 : M * N;
    uint32_t* stage = reinterpret_cast<uint32_t*>(sm);  // the planes: MMAs are done
    const int block = (32 * (warp & 3) + lane) / S::ROWS_A;
    const int m = (32 * (warp & 3) + lane) % S::ROWS_A;
    if (ok && 32 * (warp & 3) < P * S::ROWS_A) {
      // warp w reads tensor-memory lanes 32 (w % 4) .. + 31 (rows m of a block) and
      // column groups of 8 starting at 8 (w / 4)
      const uint32_t taddr = tc::tmem_addr(tbase, 32 * (warp & 3), 0);
#pragma unroll 1
      for (int n0 = 8 * (warp >> 2); n0 < N; n0 += 8 * (kPmBuildWarps / 4)) {
        uint32_t ds[7][8] = {};
#pragma unroll
        for (int c = 0; c < S::NC; ++c) tc::tmem_ld8(taddr + c * NP + n0, ds[c]);
        tc::tmem_ld_wait7(ds);
        if (m < M && block < P) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int n = n0 + j;
            if (n >= N || (UPPER && n < m)) continue;
            const int idx = UPPER ? m * M - (m * (m - 1)) / 2 + (n - m) : m * N + n;
            stage[block * outputs + idx] = reduce_classes(ds[0][j], ds[1][j], ds[2][j], ds[3][j],
                                                          ds[4][j], ds[5][j], ds[6][j], f, block);
          }
        }
        __syncwarp();  // the whole warp issues the next loads
      }
    }
    builders_sync();
    if (ok) {
      uint32_t* o = part + ((size_t)blockIdx.y * gridDim.x + e) * outputs;
      for (int i = threadIdx.x; i < outputs; i += kPmBuilders) {
        uint32_t v = stage[i];
#pragma unroll
        for (int g = 1; g < P; ++g) v = add_mod(v, stage[g * outputs + i], f.q);
        o[i] = v;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kPmMmaWarp) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, S::TCOLS);
  }
}

// A [d][rows][K] point-major operand (row stride ld words) as a 3D tensor map
// with boxes of 128 words x all rows x one point.
bool make_pm_map(CUtensorMap* map, const uint32_t* base, int K, int rows, int ld, int d) {
  EncodeTiled enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)d};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)rows * ld * 4};
  const cuuint32_t box[3] = {(cuuint32_t)KCH, (cuuint32_t)rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t*>(base), dims, strides,
             box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NP, int MX, bool UPPER>
int launch_pm(const grid_gpu_plan* p, const uint32_t* X, const uint32_t* Y, int M, int N, int K,
              int ldx, int ldy, uint32_t* part, const EmmPmGeometry& g, cudaStream_t s) {
  using S = PmShape<NP, MX, UPPER>;
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  const int rc = prepare_kernel(emm_pm_kernel<NP, MX, UPPER>, S::SMEM, kPmThreads, p->device,
                                bps_cache, &bps, true);
  if (rc) return rc;
  CUtensorMap mx, my;
  if (!make_pm_map(&mx, X, K, M, ldx, (int)p->d)) return GRID_ERR_CUDA;
  if (UPPER)
    my = mx;
  else if (!make_pm_map(&my, Y, K, N, ldy, (int)p->d))
    return GRID_ERR_CUDA;
  const uint32_t box_bytes = (uint32_t)(KCH * 4) * (uint32_t)(UPPER ? M : M + N);
  return launch_chained(emm_pm_kernel<NP, MX, UPPER>, dim3(p->d, g.splits), kPmThreads, S::SMEM, s,
                        mx, my, part, M, N, K, g.k_per_split, box_bytes, p->f, p->d_err);
}

template <int NP>
int launch_np(const grid_gpu_plan* p, const uint32_t* X, const uint32_t* Y, int M, int N, int K,
              int ldx, int ldy, int mode, uint32_t* part, const EmmPmGeometry& g, cudaStream_t s) {
  if (mode == EMM_UPPER)
    return launch_pm<NP, 64, true>(p, X, X, M, N, K, ldx, ldx, part, g, s);
  // a matrix times one to eight vectors (outer commitments, single commits): short
  // planes, so that four CTAs fit an SM and hide each other's loads
  if (M <= 8) return launch_pm<NP, 8, false>(p, X, Y, M, N, K, ldx, ldy, part, g, s);
  return M <= 64 ? launch_pm<NP, 64, false>(p, X, Y, M, N, K, ldx, ldy, part, g, s)
                 : launch_pm<NP, 128, false>(p, X, Y, M, N, K, ldx, ldy, part, g, s);
}

template <int NP>
int per_sm(int M, int mode) {
  return mode == EMM_UPPER ? PmShape<NP, 64, true>::PER_SM
         : M <= 8          ? PmShape<NP, 8, false>::PER_SM
         : M <= 64         ? PmShape<NP, 64, false>::PER_SM
                           : PmShape<NP, 128, false>::PER_SM;
}

}  // namespace

bool emm_pm_geometry(const grid_gpu_plan* p, int M, int N, int K, int mode, EmmPmGeometry* g) {
  // the inverse transform that follows (launch_sum_inverse) is compiled for d = 64
  if (!p->pm_emm || is_crt(p) || p->d != 64 || M <= 0 || N <= 0 || K <= 0 || M > 128 || N > 64)
    return false;
  if (mode == EMM_UPPER && M != N) return false;
  g->np = N <= 16 ? 16 : N <= 32 ? 32 : N <= 48 ? 48 : 64;
  // one CTA per evaluation point and K range: split K into whole chunks so that the
  // SMs' slots are about full, at most kPmMaxK words each
  const int chunks = (K + KCH - 1) / KCH;
  const int slots = g->np == 16   ? per_sm<16>(M, mode)
                    : g->np == 32 ? per_sm<32>(M, mode)
                    : g->np == 48 ? per_sm<48>(M, mode)
                                  : per_sm<64>(M, mode);
  int want = slots * p->num_sms / (int)p->d;
  if (want > chunks) want = chunks;
  if (want < 1) want = 1;
  int cps = (chunks + want - 1) / want;
  if (cps * KCH > kPmMaxK) cps = kPmMaxK / KCH;
  g->k_per_split = cps * KCH;
  g->splits = (chunks + cps - 1) / cps;
  return true;
}

size_t emm_pm_workspace_words(const grid_gpu_plan* p, int M, int N, int K, int mode) {
  EmmPmGeometry g;
  if (!emm_pm_geometry(p, M, N, K, mode, &g)) return 0;
  const size_t outputs = mode == EMM_UPPER ? (size_t)M * (M + 1) / 2 : (size_t)M * N;
  return (size_t)g.splits * outputs * p->d;
}

int launch_emm_pm(const grid_gpu_plan* p, const uint32_t* X, const uint32_t* Y, int M, int N,
                  int K, int ldx, int ldy, int mode, bool symmetrize, uint32_t* out,
                  const LimbSpec& limbs, uint32_t* work, cudaStream_t s, bool in_round) {
  EmmPmGeometry g;
  if (!emm_pm_geometry(p, M, N, K, mode, &g) || ldx < K || ldx % 4) return GRID_ERR_INVALID_PARAMETERS;
  if (mode != EMM_UPPER && (ldy < K || ldy % 4)) return GRID_ERR_INVALID_PARAMETERS;
  if (symmetrize && (mode != EMM_DENSE || M != N)) return GRID_ERR_INVALID_PARAMETERS;
  if (!work) return GRID_ERR_NULL_POINTER;
  auto unaligned = [](const void* a) { return reinterpret_cast<uintptr_t>(a) % 16 != 0; };
  if (unaligned(X) || (mode != EMM_UPPER && unaligned(Y))) return GRID_ERR_MISALIGNED;
  int rc;
  switch (g.np) {
    case 16: rc = launch_np<16>(p, X, Y, M, N, K, ldx, ldy, mode, work, g, s); break;
    case 32: rc = launch_np<32>(p, X, Y, M, N, K, ldx, ldy, mode, work, g, s); break;
    case 48: rc = launch_np<48>(p, X, Y, M, N, K, ldx, ldy, mode, work, g, s); break;
    default: rc = launch_np<64>(p, X, Y, M, N, K, ldx, ldy, mode, work, g, s); break;
  }
  if (rc) return rc;
  // point-major partials [split][e][output] -> coefficients [output][64]
  const int outputs = mode == EMM_UPPER ? M * (M + 1) / 2 : M * N;
  return launch_sum_inverse(p, work, outputs, g.splits, symmetrize ? M : 0, out, limbs, s,
                            in_round);
}

}  // namespace grid
