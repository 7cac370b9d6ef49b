// Tensor-core negacyclic products for d = 256 (tcgen05, kind::i8):
// out = INTT(NTT(a) (.) b), b given in the evaluation domain (natural slots),
// the product a Montgomery product as in every other path.
//
// Reference path replaced: the "NTT -> Montgomery pointwise -> INTT" chain of a
// negacyclic product over TwistedNttPlan (algebra/src/poly/ntt.rs:75-126,
// forward slot j = x(psi^(2j+1)), inverse with d^-1), bit-exact.
//
// Split 256 = 64 x 4. With coefficient n = 4 b + a and slot j = j2 + 64 j1 (b, j2 < 64;
// a, j1 < 4), psi a primitive 512th root, w = psi^(2 j2 + 1) and i = psi^128, i^2 = -1:
//   X_{j2 + 64 j1} = sum_a i^(j1 a) w^(a - 2) N_a[j2],
//   N_a[j2]        = sum_b psi^(2 (2 j2 + 1)(2 b + 1)) x_{4 b + a}.
// N_a is a 64-point transform of every fourth coefficient as it stands, so the four of a
// polynomial are four rows of one tensor-core product by the byte-plane method of the
// d = 64 kernel (ntt_tc_common.cuh), and everything of four points and the twists is
// done between the two products, by one thread for the four slots of a j2, with the
// product by b: 8 modular products and 16 additions for 4 words (14 and 19 with 4-point
// steps and twists before the forward and after the inverse product, and another pass
// through shared memory). The inverse mirrors it:
//   out_{4 b + a} = sum_j2 psi^(-2 (2 j2 + 1)(2 b + 1)) 256^-1 w^(2 - a) u_a[j2],
//   u_a[j2]       = sum_j1 i^(-j1 a) Z_{j2 + 64 j1}.
// The matrix psi^(2 (2 j + 1)(2 k + 1)) is symmetric and changes its sign under inversion
// with j reversed (psi^256 = -1), so one matrix in shared memory serves both directions,
// the inverse's operand in reverse order of j2; it holds i / 16 times that, whose square
// is the factor -1 / 256.
//
// A tile is 32 polynomials = 128 rows (row 32 a + p, tensor-memory lane the same). One
// persistent CTA per SM; its tiles go to two groups of eight warps in turn, each with an A
// operand, a buffer X and 256 tensor-memory columns of its own, so that one computes while
// the other waits for its MMAs, its exchanges or its loads:
//   loader (warp 18): bulk-loads tile j into X[j % 2] once F(j-2) has read its exchange
//     there, and b's tile j once F(j-1) has read the previous one; L2 prefetch of a and b
//   group (warps 8 (j % 2) .. + 7): P(j) every fourth word -> A; F(j) forward results,
//     exchanged through X, 4-point steps, twists and (x) b -> A; E(j) inverse
//     results, exchanged through A, to global memory
//   MMA (warp 16 + j % 2): fwd(j) after P(j), inv(j) after F(j), into the same columns.
// A wait that timed out ends a role's waits, not its steps, so the others still meet it at
// their barriers; every wait is bounded.
// Bound: instruction issue and the integer pipes (0.66 and 0.58 of their cycles), then the
// waits of two groups that overlap only each other. 2^20 polynomials: 1.20 ms with sixteen
// warps in step (0.47 of the issue slots), with the 4-point steps outside the products or,
// a fifth fewer instructions, between them; 1.10 with two groups; 1.08 with the MMA and
// loader lanes asleep in their waits rather than polling.
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

#include "grid_async.cuh"
#include "grid_field.cuh"
#include "grid_internal.h"
#include "grid_tc.cuh"
#include "ntt_tc_common.cuh"

namespace grid {
namespace {

using namespace tcx;

constexpr int D = 256;
constexpr int PT = ROWS / 4;                // polys per tile
constexpr int GROUP_WARPS = 8, GROUP = GROUP_WARPS * 32;
constexpr int MMA0 = 2 * GROUP_WARPS, LOADER = MMA0 + 2;
constexpr int THREADS256 = (LOADER + 1) * 32;
constexpr uint32_t XT = PT * D * 4;         // 32 KB
static_assert(XT == TILE, "a tile of words and its operand have the same size");

// Offsets from the 1 KB-aligned base of dynamic shared memory.
constexpr uint32_t OFF_W = 0;               // the 64-point matrix (B of both transforms)
constexpr uint32_t OFF_A = OFF_W + WMAT;    // [2] A operand, then E's exchange
constexpr uint32_t OFF_X = OFF_A + 2 * TILE;  // [2] input tile, then F's exchange
constexpr uint32_t OFF_B = OFF_X + 2 * XT;  // b's tile
constexpr uint32_t OFF_BAR = OFF_B + XT;
constexpr uint32_t OFF_TADDR = OFF_BAR + 18 * 8;
constexpr uint32_t SMEM_BYTES = OFF_TADDR + 16 + 1024;  // + alignment slack
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

// Device table: the matrix image (WMAT bytes), then {w, w q^-1 mod 2^32}
// Montgomery constants: w^-2, w^-1, w, w^2 of every j2 [4][64], and i.
constexpr uint32_t TW_W = WMAT / 8;  // in uint2 units
constexpr uint32_t TW_I = TW_W + 256;
constexpr size_t TABLE_BYTES = WMAT + (256 + 1) * 8 + 8;

// Barriers, one of each per group.
enum Bar : int {
  AFULL = 0,          // input tile landed
  XFREE = 2,          // X read for the last time
  BFULL = 4,          // b's tile landed
  BFREE = 6,          // F has read b's tile
  PREP = 8,           // forward operand written
  FDONE = 10,
  PREADY = 12,        // inverse operand written
  IDONE = 14,
  WFULL = 16,         // the matrix landed (one barrier)
  NBARS
};

// The warps of a group (named barrier 1 or 2).
__device__ __forceinline__ void group_sync(int g) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(GROUP) : "memory");
}

__device__ __forceinline__ uint32_t mulc(uint32_t x, uint2 w, uint32_t q) {
  return mont_c(x, w.x, w.y, q);
}

__global__ void __launch_bounds__(THREADS256, 1)
    ntt256_tc_mulinv_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                            uint32_t* out, unsigned long long npolys,
                            const unsigned char* __restrict__ table, const TcConsts k,
                            uint32_t r1, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  const uint32_t raw = smem_addr(sm_raw);
  unsigned char* sm = sm_raw + (((raw + 1023u) & ~1023u) - raw);
  const uint32_t s0 = smem_addr(sm);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  uint32_t* taddr_slot = reinterpret_cast<uint32_t*>(sm + OFF_TADDR);
  const uint2* tw = reinterpret_cast<const uint2*>(table);

  if (warp == MMA0) {
    if (lane == 0) {
      for (int i = 0; i < NBARS; ++i)
        mbar_init(&bars[i], (i & ~1) == XFREE || (i & ~1) == BFREE || (i & ~1) == PREP ||
                                    (i & ~1) == PREADY
                                ? GROUP_WARPS
                                : 1);
      fence_mbar_init();
      tc::fence_async_smem();
      mbar_arrive_expect_tx(&bars[WFULL], WMAT);
      bulk_load(sm + OFF_W, table, WMAT, &bars[WFULL]);
    }
    __syncwarp();
    tc::tmem_alloc(taddr_slot, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *taddr_slot;

  const unsigned long long ntiles = (npolys + PT - 1) / PT;
  const uint32_t n = blockIdx.x < ntiles
                         ? (uint32_t)((ntiles - 1 - blockIdx.x) / gridDim.x + 1)
                         : 0u;  // tiles of this CTA
  auto poly0 = [&](uint32_t j) -> unsigned long long {
    return ((unsigned long long)blockIdx.x + (unsigned long long)j * gridDim.x) * PT;
  };
  auto tile_bytes = [&](uint32_t j) -> uint32_t {
    const unsigned long long left = npolys - poly0(j);
    return (uint32_t)(left < PT ? left : PT) * D * 4;
  };

  if (warp == LOADER) {
    // ------------------------------------------------------------ loader
    if (lane == 0) {
      bool ok = true;
      uint32_t xs = 0, bs = 0;  // tiles requested
      auto prefetch = [&](uint32_t j) {
        if (j >= n) return;
        prefetch_l2(a + poly0(j) * D, tile_bytes(j));
        prefetch_l2(b + poly0(j) * D, tile_bytes(j));
      };
      for (uint32_t j = 0; j < 3; ++j) prefetch(j);
      for (uint32_t j = 0; ok && j < n; ++j) {
        const uint32_t g = j & 1, u = j >> 1;
        if (u && !(ok = mbar_wait_sleep(&bars[XFREE + g], (u - 1) & 1, err))) break;
        mbar_arrive_expect_tx(&bars[AFULL + g], tile_bytes(j));
        bulk_load(sm + OFF_X + g * XT, a + poly0(j) * D, tile_bytes(j), &bars[AFULL + g]);
        ++xs;
        if (j && !(ok = mbar_wait_sleep(&bars[BFREE + (g ^ 1)], ((j - 1) >> 1) & 1, err))) break;
        mbar_arrive_expect_tx(&bars[BFULL + g], tile_bytes(j));
        bulk_load(sm + OFF_B, b + poly0(j) * D, tile_bytes(j), &bars[BFULL + g]);
        ++bs;
        prefetch(j + 3);
      }
      // nothing may still be writing shared memory at exit
      for (uint32_t g = 0; g < 2; ++g) {
        if (xs > g) mbar_wait_sleep(&bars[AFULL + g], ((xs - g - 1) >> 1) & 1, err);
        if (bs > g) mbar_wait_sleep(&bars[BFULL + g], ((bs - g - 1) >> 1) & 1, err);
      }
    }
    __syncwarp();
  } else if (warp >= MMA0) {
    // ------------------------------------------------------------ MMA issue
    const uint32_t g = warp - MMA0;
    if (lane == 0) {
      uint32_t fwd = 0, inv = 0;
      const bool ready = mbar_wait_sleep(&bars[WFULL], 0, err);
      for (uint32_t j = g, u = 0; ready && j < n; j += 2, ++u) {
        if (!mbar_wait_sleep(&bars[PREP + g], u & 1, err)) break;
        tc::fence_after_sync();
        issue_transform(tbase + 256 * g, s0 + OFF_A + g * TILE, s0 + OFF_W);
        tc::mma_commit(&bars[FDONE + g]);
        ++fwd;
        if (!mbar_wait_sleep(&bars[PREADY + g], u & 1, err)) break;
        tc::fence_after_sync();
        issue_transform(tbase + 256 * g, s0 + OFF_A + g * TILE, s0 + OFF_W);
        tc::mma_commit(&bars[IDONE + g]);
        ++inv;
      }
      // every MMA issued is done before shared and tensor memory are released
      if (fwd) mbar_wait_sleep(&bars[FDONE + g], (fwd - 1) & 1, err);
      if (inv) mbar_wait_sleep(&bars[IDONE + g], (inv - 1) & 1, err);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ groups
    const uint32_t g = warp / GROUP_WARPS;
    const uint32_t aa = warp & 3, half = (warp >> 2) & 1;  // row block, columns 32 half .. + 31
    const uint32_t p = lane;                               // polynomial of this thread's row
    const uint32_t taddr = tc::tmem_addr(tbase, 32 * aa, 256 * g + 32 * half);
    const uint32_t q = k.q;
    bool ok = true;
    // Outside the reductions a thread has word / slot index bb of the polynomials
    // pp0 + 4 it: its twists are fixed.
    const uint32_t bb = threadIdx.x & 63, pp0 = (threadIdx.x & (GROUP - 1)) >> 6;
    const uint2 wm2 = tw[TW_W + bb], wm1 = tw[TW_W + 64 + bb], w1 = tw[TW_W + 128 + bb],
                w2 = tw[TW_W + 192 + bb], im = tw[TW_I];
    unsigned char* const opnd = sm + OFF_A + g * TILE;
    uint32_t* const x = reinterpret_cast<uint32_t*>(sm + OFF_X + g * XT);
    const uint32_t* const bt = reinterpret_cast<const uint32_t*>(sm + OFF_B);
    // word of K index kk of row 32 a + pp of the A operand
    auto operand = [&](uint32_t a_, uint32_t pp, uint32_t kk) -> uint32_t* {
      return reinterpret_cast<uint32_t*>(
          opnd + sw128(32 * a_ + pp, kk >> 5, (kk & 31) >> 2, BOX) + 4 * (kk & 3));
    };
    // Reduced results from the layout of the rows to buffer `to`: word 64 a + c of
    // polynomial p at that index with its low 5 bits XORed with p (the 32 lanes hit 32
    // banks, here and where a warp reads 32 consecutive c of one polynomial)
    auto exchange = [&](uint32_t* to) {
      __syncwarp();
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        uint32_t res[16];
        reduce16(taddr + 16 * h, k, res);
#pragma unroll
        for (int t = 0; t < 16; ++t)
          to[p * D + ((64 * aa + 32 * half + 16 * h + t) ^ p)] = res[t];
        __syncwarp();
      }
      tc::fence_before_sync();
      group_sync(g);
    };
    auto arrive = [&](int bar) {
      if (lane == 0) mbar_arrive(&bars[bar + g]);
    };

    for (uint32_t j = g, u = 0; j < n; j += 2, ++u) {
      // P(j)
      ok = ok && lane0_wait(&bars[AFULL + g], u & 1, lane, err);
#pragma unroll 4
      for (int it = 0; it < 8; ++it) {
        const uint32_t pp = pp0 + 4 * it;
        const uint4 v = reinterpret_cast<const uint4*>(x)[pp * (D / 4) + bb];
        *operand(0, pp, bb) = v.x;
        *operand(1, pp, bb) = v.y;
        *operand(2, pp, bb) = v.z;
        *operand(3, pp, bb) = v.w;
      }
      tc::fence_async_smem();
      __syncwarp();
      arrive(PREP);
      // F(j)
      ok = ok && lane0_wait(&bars[FDONE + g], u & 1, lane, err);
      tc::fence_after_sync();
      exchange(x);
      ok = ok && lane0_wait(&bars[BFULL + g], u & 1, lane, err);
#pragma unroll 2
      for (int it = 0; it < 8; ++it) {
        const uint32_t pp = pp0 + 4 * it;
        uint32_t v[4], z[4];
#pragma unroll
        for (int a_ = 0; a_ < 4; ++a_) v[a_] = x[pp * D + ((64 * a_ + bb) ^ pp)];
        v[0] = mulc(v[0], wm2, q);
        v[1] = mulc(v[1], wm1, q);
        v[3] = mulc(v[3], w1, q);
        // all canonical: b is any word
        const uint32_t c0 = add_canon(v[0], v[2], q), c1 = sub_lazy(v[0], v[2], q);
        const uint32_t e0 = add_canon(v[1], v[3], q);
        const uint32_t e1 = mulc(sub_lazy(v[1], v[3], q), im, q);
        z[0] = add_canon(c0, e0, q);
        z[2] = sub_lazy(c0, e0, q);
        z[1] = add_canon(c1, e1, q);
        z[3] = sub_lazy(c1, e1, q);
#pragma unroll
        for (int j1 = 0; j1 < 4; ++j1)
          z[j1] = redc64(mad_wide(z[j1], bt[pp * D + 64 * j1 + bb], 0ull), q, k.qinv);
        const uint32_t t0 = add_canon(z[0], z[2], q), d0 = sub_lazy(z[0], z[2], q);
        const uint32_t t1 = add_canon(z[1], z[3], q);
        const uint32_t d1 = mulc(sub_lazy(z[1], z[3], q), im, q);
        *operand(0, pp, 63 - bb) = mulc(add_lazy(t0, t1, r1), w2, q);
        *operand(1, pp, 63 - bb) = mulc(sub_lazy(d0, d1, q), w1, q);
        *operand(2, pp, 63 - bb) = sub_lazy(t0, t1, q);
        *operand(3, pp, 63 - bb) = mulc(add_lazy(d0, d1, r1), wm1, q);
      }
      tc::fence_async_smem();  // the operand, and X before its refill by a bulk copy
      __syncwarp();
      arrive(BFREE);
      arrive(XFREE);
      arrive(PREADY);
      // E(j)
      ok = ok && lane0_wait(&bars[IDONE + g], u & 1, lane, err);
      tc::fence_after_sync();
      uint32_t* ex = reinterpret_cast<uint32_t*>(opnd);
      exchange(ex);
      const unsigned long long first = poly0(j);
      const uint32_t valid = tile_bytes(j) / (D * 4);
      uint4* o = reinterpret_cast<uint4*>(out + first * D) + bb;
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const uint32_t pp = pp0 + 4 * it;
        const uint32_t* xr = ex + pp * D;
        if (ok && pp < valid)
          o[pp * (D / 4)] = make_uint4(xr[bb ^ pp], xr[(64 + bb) ^ pp], xr[(128 + bb) ^ pp],
                                       xr[(192 + bb) ^ pp]);
      }
      group_sync(g);  // the exchange is read before P(j + 2) writes the operand there
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == MMA0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
}

}  // namespace

bool ntt256_tc_available(const grid_gpu_plan* p) { return p->d == 256 && p->d_tcw != nullptr; }

int launch_ntt256_tc(const grid_gpu_plan* p, const uint32_t* a, const uint32_t* b, uint32_t* out,
                     size_t npolys, cudaStream_t s) {
  if (npolys == 0) return GRID_OK;
  static int bps_cache[kMaxDevices] = {};
  int bps = 0;
  const int st =
      prepare_kernel(ntt256_tc_mulinv_kernel, SMEM_BYTES, THREADS256, p->device, bps_cache, &bps);
  if (st) return st;
  const unsigned long long tiles = (npolys + PT - 1) / PT;
  const unsigned long long grid =
      tiles < (unsigned long long)p->num_sms ? tiles : (unsigned long long)p->num_sms;
  TcConsts k;
  k.q = p->f.q;
  k.qinv = p->f.qinv;
  ntt256_tc_mulinv_kernel<<<(unsigned)grid, THREADS256, SMEM_BYTES, s>>>(
      a, b, out, (unsigned long long)npolys, static_cast<const unsigned char*>(p->d_tcw), k,
      p->f.r1, p->d_err);
  return cuda_status(cudaGetLastError());
}

// The 64-point matrix image (row 64 l + j, K byte 4k + i = byte l of
// 2^(8i) (psi^128 / 16) psi^(2 (2 j + 1)(2 k + 1)) 2^32 mod q, 128-byte-swizzled K-major),
// then the twists as {Montgomery word, word * q^-1 mod 2^32}.
void build_tc256_tables(uint32_t q, uint64_t psi, std::vector<unsigned char>& out) {
  out.assign(TABLE_BYTES, 0);
  auto mulm = [q](uint64_t x, uint64_t y) { return (uint64_t)((unsigned __int128)x * y % q); };
  auto powm = [&](uint64_t x, uint64_t e) {
    uint64_t r = 1;
    x %= q;
    while (e) {
      if (e & 1) r = mulm(r, x);
      x = mulm(x, x);
      e >>= 1;
    }
    return r;
  };
  uint32_t qinv = 1;
  for (int i = 0; i < 5; ++i) qinv *= 2u - q * qinv;
  const uint64_t R = ((uint64_t)1 << 32) % q;
  std::vector<uint64_t> power(2 * D, 1);  // of psi
  for (uint32_t e = 1; e < 2 * D; ++e) power[e] = mulm(power[e - 1], psi);
  const uint64_t im = power[128];
  const uint64_t scale = mulm(mulm(im, powm(16, q - 2)), R);
  for (uint32_t j = 0; j < 64; ++j)
    for (uint32_t kk = 0; kk < 64; ++kk) {
      uint64_t w = mulm(power[(2 * (2 * j + 1) * (2 * kk + 1)) % (2 * D)], scale);
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t kb = 4 * kk + i, h = kb / 128, kc = kb % 128;
        for (uint32_t l = 0; l < 4; ++l)
          out[sw128(64 * l + j, h, kc / 16, WMAT / 2) + kc % 16] = (unsigned char)(w >> (8 * l));
        w = mulm(w, 256);  // next byte of x_k: times 2^8
      }
    }
  auto put = [&](uint32_t idx, uint64_t value) {
    const uint32_t wm = (uint32_t)mulm(value, R);
    const uint32_t pair[2] = {wm, wm * qinv};
    std::memcpy(out.data() + (size_t)idx * 8, pair, 8);
  };
  for (uint32_t j2 = 0; j2 < 64; ++j2) {
    const uint32_t e = 2 * j2 + 1, order = 2 * D;
    put(TW_W + j2, power[order - 2 * e % order]);
    put(TW_W + 64 + j2, power[order - e]);
    put(TW_W + 128 + j2, power[e]);
    put(TW_W + 192 + j2, power[2 * e % order]);
  }
  put(TW_I, im);
}

}  // namespace grid
