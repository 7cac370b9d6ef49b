// C ABI for prepared matrices, commitments, the Gram matrix, the JL
// projection, decompositions and the fused LaBRADOR prover round.
#include <cuda_runtime.h>

#include <cstring>
#include <new>

#include "grid_internal.h"

using namespace grid;

namespace {

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// The forward transform stores the evaluations of M x K witness polys
// point-major and the product with Y (N rows) runs on the TMA-fed tensor-core
// kernel (emm_pm.cu).
bool pm_fits(const grid_gpu_plan* p, size_t M, size_t N, size_t K, int mode) {
  EmmPmGeometry g;
  return ntt_tc_available(p) && emm_pm_geometry(p, (int)M, (int)N, (int)K, mode, &g);
}

// The plan whose products a call runs: p, or the first auxiliary prime's (all alike).
const grid_gpu_plan* residue_plan(const grid_gpu_plan* p) { return is_crt(p) ? p->crt[0] : p; }

// Evaluations of rows of n polys and the products' partials on plan e: for the point-major
// products (and the gathering ones, should a matrix lack its copy), or those alone.
struct EvalsLayout {
  const grid_gpu_plan* e;
  bool pm;
  size_t stride;  // polys per row
  EvalsLayout(const grid_gpu_plan* plan, bool point_major, size_t n)
      : e(plan), pm(point_major), stride(point_major ? pm_stride(n) : n) {}
  size_t work(size_t M, size_t N, size_t K, int mode) const {
    return pm ? emm_workspace_words(e, (int)M, (int)N, (int)K, mode)
              : emm_gather_words(e, (int)M, (int)N, (int)K, mode);
  }
};

// Workspace layouts. On a ring plan without an NTT for q (is_crt) a call runs the
// prime's own call for each auxiliary prime in turn, on the inputs as they are (the
// forward transforms reduce any 32-bit words, ring_crt.cu) and in the same workspace,
// and keeps the three residue results; the reconstruction writes the output.
//
// The sizes are what a call runs best in. One that is given less runs by the gathering
// products if those fit (point-major rows are padded to whole 16-byte units and have more
// K ranges, the vector products a partial per CTA): a caller may size its workspace for the
// largest of several shapes.
size_t commit_ws_bytes(const grid_gpu_plan* p, size_t rows, size_t cols, size_t batch) {
  if (is_crt(p))
    return 3 * words_bytes(batch * rows * p->d) + commit_ws_bytes(p->crt[0], rows, cols, batch);
  if (commit_small_fits(p, rows, cols, batch)) return 0;  // one launch, no intermediate
  if (commit_vec_fits(p, rows, cols, batch))
    return words_bytes(commit_vec_words(p, rows, cols, 0, batch));
  const EvalsLayout l(p, true, cols);
  return words_bytes(batch * l.stride * p->d) +
         words_bytes(l.work(batch, rows, cols, EMM_DENSE));
}

bool gram_pm(const grid_gpu_plan* p, size_t r, size_t n) {
  return pm_fits(residue_plan(p), r, r, n, EMM_UPPER);
}

size_t gram_ws_bytes(const grid_gpu_plan* p, size_t r, size_t n, bool pm) {
  const EvalsLayout l(residue_plan(p), pm, n);
  const size_t base = words_bytes(r * l.stride * p->d) + words_bytes(l.work(r, r, n, EMM_UPPER));
  return is_crt(p) ? base + 3 * words_bytes(r * (r + 1) / 2 * p->d) : base;
}

bool garbage_h_pm(const grid_gpu_plan* p, size_t r, size_t n) {
  return pm_fits(residue_plan(p), r, r, n, EMM_DENSE);
}

size_t garbage_h_ws_bytes(const grid_gpu_plan* p, size_t r, size_t n, bool pm) {
  const EvalsLayout l(residue_plan(p), pm, n);
  const size_t base = 2 * words_bytes(r * l.stride * p->d) + words_bytes(r * r * p->d) +
                      words_bytes(l.work(r, r, n, EMM_DENSE));
  return is_crt(p) ? base + 3 * words_bytes(r * r * p->d) : base;
}

size_t amortize_ws_bytes(const grid_gpu_plan* p, size_t r, size_t n) {
  const size_t base = words_bytes(r * n * p->d) + words_bytes(r * p->d);
  return is_crt(p) ? base + 3 * words_bytes(n * p->d) : base;
}

bool round_pm(const grid_gpu_plan* p, size_t r, size_t n, size_t kappa) {
  const grid_gpu_plan* e = residue_plan(p);
  return pm_fits(e, r, kappa, n, EMM_DENSE) && pm_fits(e, r, r, n, EMM_UPPER);
}

// Partials of the round's two products, one after the other.
size_t round_work(const EvalsLayout& l, size_t r, size_t n, size_t kappa) {
  const size_t t = l.work(r, kappa, n, EMM_DENSE), g = l.work(r, r, n, EMM_UPPER);
  return t > g ? t : g;
}

size_t round_ws_bytes(const grid_gpu_plan* p, size_t r, size_t n, size_t kappa, size_t jl_rows,
                      bool pm) {
  const size_t d = p->d;
  const EvalsLayout l(residue_plan(p), pm, n);
  const size_t base = words_bytes(r * l.stride * d) + words_bytes(round_work(l, r, n, kappa)) +
                      words_bytes(r * kappa * d) +
                      round_up(jl_scratch_bytes(jl_rows ? jl_rows : 1), 256);
  return is_crt(p) ? base + 3 * (words_bytes(r * kappa * d) + words_bytes(r * (r + 1) / 2 * d))
                   : base;
}

bool dims_ok(size_t a, size_t b, size_t c) {
  // all kernels index rows/cols/K with int
  return a > 0 && b > 0 && c > 0 && a < (1u << 30) && b < (1u << 30) && c < (1u << 30);
}

// a * b * c words of 4 bytes stay far below SIZE_MAX (no wrap in any size sum).
bool words_fit(size_t a, size_t b, size_t c) {
  size_t x;
  return !__builtin_mul_overflow(a, b, &x) && !__builtin_mul_overflow(x, c, &x) &&
         x < (1ull << 56);
}

// r x n witness polys and the r x r products over them (Gram, garbage h, amortization).
bool square_dims_ok(const grid_gpu_plan* p, size_t r, size_t n) {
  return dims_ok(r, n, 1) && words_fit(r, n, p->d) && words_fit(r, r, p->d);
}

// The evaluations of matrix m (plan, shape and ld set) from A, and, where products on
// the TMA-fed tensor-core kernel apply, their point-major copy in the same allocation
// (left out where memory holds the evaluations alone: products gather those then).
int prepare_evals(grid_gpu_matrix* m, const uint32_t* A, bool a_is_evals, cudaStream_t st) {
  const grid_gpu_plan* p = m->plan;
  const size_t polys = m->rows * m->cols, words = polys * p->d;
  bool pm = pm_fits(p, 1, m->rows, m->cols, EMM_DENSE);
  const size_t part = words_bytes(words), ld = pm_stride(m->cols);
  cudaError_t e = cudaMalloc(&m->d_evals, pm ? part + m->rows * ld * p->d * 4 : words * 4);
  if (pm && e == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();  // or the next launch's check would report it
    pm = false;
    e = cudaMalloc(&m->d_evals, words * 4);
  }
  int rc = cuda_status(e);
  if (rc) return rc;
  if (a_is_evals)
    rc = cuda_status(cudaMemcpyAsync(m->d_evals, A, words * 4, cudaMemcpyDeviceToDevice, st));
  else
    rc = launch_ntt(p, MODE_FWD, A, nullptr, m->d_evals, polys, st);
  if (!rc && pm) {
    m->d_evals_pm = m->d_evals + part / 4;
    m->ld_pm = ld;
    rc = launch_to_point_major(m->d_evals, m->d_evals_pm, m->rows, m->cols, ld, (int)p->d, st);
  }
  return rc;
}

// Two products of a few vectors as one (both too long for the one-launch kernel).
bool linear_vec_fits(const grid_gpu_matrix* A, const grid_gpu_matrix* B, size_t batch) {
  const grid_gpu_plan* p = A->plan;
  return commit_vec_fits(p, A->rows, A->cols + B->cols, batch) &&
         !commit_small_fits(p, A->rows, A->cols, batch) &&
         !commit_small_fits(p, B->rows, B->cols, batch);
}

// t = A * s for `batch` vectors, into t (coefficients). ws from a Carver.
int commit_core(const grid_gpu_matrix* A, const uint32_t* s, size_t batch, uint32_t* t,
                Carver& cv, cudaStream_t st) {
  const grid_gpu_plan* p = A->plan;
  if (is_crt(p)) {
    if (!crt_bound_ok(p, A->cols)) return GRID_ERR_INVALID_PARAMETERS;
    const size_t tw = batch * A->rows * p->d;
    uint32_t* tj[3] = {cv.take<uint32_t>(tw), cv.take<uint32_t>(tw), cv.take<uint32_t>(tw)};
    if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
    const size_t mark = cv.used;
    for (int j = 0; j < 3; ++j) {
      const int rc = commit_core(A->crt[j], s, batch, tj[j], cv, st);
      if (rc) return rc;
      cv.used = mark;  // the next prime reuses the same workspace
    }
    return crt_combine(p, tj[0], tj[1], tj[2], tw, t, st);
  }
  if (commit_small_fits(p, A->rows, A->cols, batch))
    return launch_commit_small(p, A->d_evals, A->rows, A->cols, A->ld, s, batch, t, st);
  const Carver given = cv;
  if (commit_vec_fits(p, A->rows, A->cols, batch)) {
    uint32_t* part = cv.take<uint32_t>(commit_vec_words(p, A->rows, A->cols, 0, batch));
    if (cv.ok)
      return launch_commit_vec(p, VecOperand{A->d_evals, s, A->cols, A->ld}, nullptr, A->rows,
                               batch, t, part, st);
    cv = given;
  }
  if (A->d_evals_pm && pm_fits(p, batch, A->rows, A->cols, EMM_DENSE)) {
    const size_t ldx = pm_stride(A->cols);
    uint32_t* s_hat = cv.take<uint32_t>(batch * ldx * p->d);
    uint32_t* work = cv.take<uint32_t>(
        emm_pm_workspace_words(p, (int)batch, (int)A->rows, (int)A->cols, EMM_DENSE));
    if (cv.ok) {
      const int rc = launch_ntt_tc_pm(p, s, batch, A->cols, s_hat, st);
      if (rc) return rc;
      return launch_emm_pm(p, s_hat, A->d_evals_pm, (int)batch, (int)A->rows, (int)A->cols,
                           (int)ldx, (int)A->ld_pm, EMM_DENSE, false, t, LimbSpec(), work, st);
    }
    cv = given;
  }
  uint32_t* s_hat = cv.take<uint32_t>(batch * A->cols * p->d);
  const size_t ew = emm_gather_words(p, (int)batch, (int)A->rows, (int)A->cols, EMM_DENSE);
  uint32_t* work = ew ? cv.take<uint32_t>(ew) : nullptr;
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  int rc = launch_ntt(p, MODE_FWD, s, nullptr, s_hat, batch * A->cols, st);
  if (!rc)
    rc = launch_emm(p, s_hat, A->d_evals, (int)batch, (int)A->rows, (int)A->cols, (int)A->ld,
                    EMM_DENSE, t, work, st);
  if (rc) return rc;
  return launch_ntt(p, MODE_INV, t, nullptr, t, batch * A->rows, st);
}

// t = A m + B r, t2: scratch of t's size (coefficients).
int linear_core(const grid_gpu_matrix* A, const grid_gpu_matrix* B, const uint32_t* m,
                const uint32_t* r, size_t batch, uint32_t* t, uint32_t* t2, Carver& cv,
                cudaStream_t st) {
  const grid_gpu_plan* p = A->plan;
  const Carver given = cv;
  if (linear_vec_fits(A, B, batch)) {
    uint32_t* part = cv.take<uint32_t>(commit_vec_words(p, A->rows, A->cols, B->cols, batch));
    const VecOperand second{B->d_evals, r, B->cols, B->ld};
    if (cv.ok)
      return launch_commit_vec(p, VecOperand{A->d_evals, m, A->cols, A->ld}, &second, A->rows,
                               batch, t, part, st);
    cv = given;
  }
  int rc = commit_core(A, m, batch, t, cv, st);
  cv = given;  // the second product reuses the first one's workspace
  if (!rc) rc = commit_core(B, r, batch, t2, cv, st);
  // A_msg*m + A_open*r: INTT is linear, so adding the coefficient forms is exact.
  if (!rc) rc = launch_add(p, t, t2, batch * B->rows * p->d, st);
  return rc;
}

size_t linear_ws_bytes(const grid_gpu_matrix* A, const grid_gpu_matrix* B, size_t batch) {
  const grid_gpu_plan* p = A->plan;
  if (linear_vec_fits(A, B, batch))
    return words_bytes(commit_vec_words(p, A->rows, A->cols, B->cols, batch));
  return commit_ws_bytes(p, A->rows, A->cols, batch) + commit_ws_bytes(p, B->rows, B->cols, batch);
}

}  // namespace

int grid::gram_min_workspace(const grid_gpu_plan* p, size_t r, size_t n, size_t* bytes) {
  if (!p || !bytes) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  *bytes = gram_ws_bytes(p, r, n, false);
  return GRID_OK;
}

extern "C" {

/* ---- prepared matrices ------------------------------------------------- */

int grid_gpu_matrix_create_dev(grid_gpu_plan* p, const uint32_t* A, size_t rows, size_t cols,
                               int a_is_evals, grid_gpu_matrix** out, void* stream) {
  if (!p || !out || !A) return GRID_ERR_NULL_POINTER;
  *out = nullptr;
  if (!dims_ok(rows, cols, 1)) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(A)) return GRID_ERR_MISALIGNED;
  if (!words_fit(rows, cols, p->d)) return GRID_ERR_INVALID_PARAMETERS;
  if (is_crt(p) && a_is_evals) return p->ntt_status;  // q has no evaluation domain
  grid_gpu_matrix* m = new (std::nothrow) grid_gpu_matrix();
  if (!m) return GRID_ERR_OUT_OF_MEMORY;
  m->plan = p;
  m->rows = rows;
  m->cols = cols;
  m->ld = cols;
  cudaStream_t st = (cudaStream_t)stream;
  int rc = GRID_OK;
  if (is_crt(p)) {
    // the matrix mod each auxiliary prime, prepared (transformed) on its plan
    for (int j = 0; j < 3 && !rc; ++j) {
      grid_gpu_matrix* sub = new (std::nothrow) grid_gpu_matrix();
      if (!sub) {
        rc = GRID_ERR_OUT_OF_MEMORY;
        break;
      }
      m->crt[j] = sub;
      sub->plan = p->crt[j];
      sub->rows = rows;
      sub->cols = cols;
      sub->ld = cols;
      rc = prepare_evals(sub, A, false, st);
    }
  } else {
    rc = prepare_evals(m, A, a_is_evals != 0, st);
  }
  if (rc) {
    grid_gpu_matrix_destroy(m);
    return rc;
  }
  *out = m;
  return GRID_OK;
}

int grid_gpu_matrix_create(grid_gpu_plan* p, const uint32_t* A, size_t rows, size_t cols,
                           int a_is_evals, grid_gpu_matrix** out) {
  if (!p || !out || !A) return GRID_ERR_NULL_POINTER;
  *out = nullptr;
  if (!dims_ok(rows, cols, 1)) return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t bytes = rows * cols * p->d * 4;
  int rc = ensure_scratch(p, 6, bytes);
  if (rc) return rc;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, A, bytes, cudaMemcpyHostToDevice, p->stream));
  if (rc) return rc;
  rc = grid_gpu_matrix_create_dev(p, static_cast<uint32_t*>(p->scratch[6].ptr), rows, cols,
                                  a_is_evals, out, p->stream);
  const int fin = finish_host_call(p, p->stream);
  if (rc) return rc;
  if (fin && *out) {
    grid_gpu_matrix_destroy(*out);
    *out = nullptr;
  }
  return fin;
}

int grid_gpu_matrix_destroy(grid_gpu_matrix* m) {
  if (!m) return GRID_ERR_NULL_POINTER;
  for (grid_gpu_matrix* sub : m->crt)
    if (sub) grid_gpu_matrix_destroy(sub);
  if (m->owned && m->d_evals) cudaFree(m->d_evals);
  delete m;
  return GRID_OK;
}

int grid_gpu_matrix_view(const grid_gpu_matrix* parent, size_t cols, grid_gpu_matrix** out) {
  if (!parent || !out) return GRID_ERR_NULL_POINTER;
  *out = nullptr;
  if (cols == 0 || cols > parent->cols) return GRID_ERR_DIMENSION_MISMATCH;
  grid_gpu_matrix* m = new (std::nothrow) grid_gpu_matrix();
  if (!m) return GRID_ERR_OUT_OF_MEMORY;
  m->plan = parent->plan;
  m->rows = parent->rows;
  m->cols = cols;
  m->ld = parent->ld;
  m->d_evals = parent->d_evals;
  m->d_evals_pm = parent->d_evals_pm;
  m->ld_pm = parent->ld_pm;
  m->owned = false;
  for (int j = 0; j < 3; ++j)
    if (parent->crt[j]) {
      const int rc = grid_gpu_matrix_view(parent->crt[j], cols, &m->crt[j]);
      if (rc) {
        grid_gpu_matrix_destroy(m);
        return rc;
      }
    }
  *out = m;
  return GRID_OK;
}

int grid_gpu_matrix_shape(const grid_gpu_matrix* m, size_t* rows, size_t* cols) {
  if (!m || !rows || !cols) return GRID_ERR_NULL_POINTER;
  *rows = m->rows;
  *cols = m->cols;
  return GRID_OK;
}

int grid_gpu_matrix_device_evals(const grid_gpu_matrix* m, const uint32_t** evals) {
  if (!m || !evals) return GRID_ERR_NULL_POINTER;
  if (is_crt(m->plan)) return m->plan->ntt_status;  // no evaluation domain mod q
  *evals = m->d_evals;
  return GRID_OK;
}

/* ---- commitments ------------------------------------------------------- */

int grid_gpu_commit_workspace(const grid_gpu_matrix* A, size_t batch, size_t* bytes) {
  if (!A || !bytes) return GRID_ERR_NULL_POINTER;
  *bytes = commit_ws_bytes(A->plan, A->rows, A->cols, batch);
  return GRID_OK;
}

int grid_gpu_commit_dev(const grid_gpu_matrix* A, const uint32_t* s, size_t batch, uint32_t* t,
                        void* workspace, size_t workspace_bytes, void* stream) {
  if (!A || ((!s || !t) && batch)) return GRID_ERR_NULL_POINTER;
  if (batch == 0) return GRID_OK;
  if (!dims_ok(batch, A->rows, A->cols)) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(s) || !aligned16(t) || !aligned16(workspace)) return GRID_ERR_MISALIGNED;
  Carver cv(workspace, workspace_bytes);
  return commit_core(A, s, batch, t, cv, (cudaStream_t)stream);
}

int grid_gpu_commit(grid_gpu_matrix* A, const uint32_t* s, size_t batch, uint32_t* t) {
  if (!A || ((!s || !t) && batch)) return GRID_ERR_NULL_POINTER;
  if (batch == 0) return GRID_OK;
  if (!dims_ok(batch, A->rows, A->cols)) return GRID_ERR_INVALID_PARAMETERS;
  grid_gpu_plan* p = A->plan;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t s_bytes = batch * A->cols * p->d * 4, t_bytes = batch * A->rows * p->d * 4;
  const size_t ws = commit_ws_bytes(p, A->rows, A->cols, batch);
  int rc;
  if ((rc = ensure_scratch(p, 6, s_bytes)) || (rc = ensure_scratch(p, 7, t_bytes)) ||
      (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, s, s_bytes, cudaMemcpyHostToDevice, st));
  if (!rc) {
    Carver cv(p->scratch[8].ptr, ws);
    rc = commit_core(A, static_cast<uint32_t*>(p->scratch[6].ptr), batch,
                     static_cast<uint32_t*>(p->scratch[7].ptr), cv, st);
  }
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(t, p->scratch[7].ptr, t_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

int grid_gpu_linear_commit_workspace(const grid_gpu_matrix* A_msg, const grid_gpu_matrix* A_open,
                                     size_t batch, size_t* bytes) {
  if (!A_msg || !A_open || !bytes) return GRID_ERR_NULL_POINTER;
  const grid_gpu_plan* p = A_msg->plan;
  *bytes = linear_ws_bytes(A_msg, A_open, batch) + words_bytes(batch * A_open->rows * p->d);
  return GRID_OK;
}

int grid_gpu_linear_commit_dev(const grid_gpu_matrix* A_msg, const grid_gpu_matrix* A_open,
                               const uint32_t* m, const uint32_t* r, size_t batch, uint32_t* t,
                               void* workspace, size_t workspace_bytes, void* stream) {
  if (!A_msg || !A_open || ((!m || !r || !t) && batch)) return GRID_ERR_NULL_POINTER;
  if (A_msg->plan != A_open->plan) return GRID_ERR_INVALID_PARAMETERS;
  if (A_msg->rows != A_open->rows) return GRID_ERR_DIMENSION_MISMATCH;
  if (batch == 0) return GRID_OK;
  if (!dims_ok(batch, A_msg->rows, A_msg->cols) || !dims_ok(batch, A_open->rows, A_open->cols))
    return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(m) || !aligned16(r) || !aligned16(t) || !aligned16(workspace))
    return GRID_ERR_MISALIGNED;
  const grid_gpu_plan* p = A_msg->plan;
  cudaStream_t st = (cudaStream_t)stream;
  Carver cv(workspace, workspace_bytes);
  uint32_t* t2 = cv.take<uint32_t>(batch * A_open->rows * p->d);
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  return linear_core(A_msg, A_open, m, r, batch, t, t2, cv, st);
}

int grid_gpu_linear_commit(grid_gpu_matrix* A_msg, grid_gpu_matrix* A_open, const uint32_t* m,
                           const uint32_t* r, size_t batch, uint32_t* t) {
  if (!A_msg || !A_open || ((!m || !r || !t) && batch)) return GRID_ERR_NULL_POINTER;
  if (A_msg->plan != A_open->plan) return GRID_ERR_INVALID_PARAMETERS;
  if (A_msg->rows != A_open->rows) return GRID_ERR_DIMENSION_MISMATCH;
  if (batch == 0) return GRID_OK;
  grid_gpu_plan* p = A_msg->plan;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t rows = A_msg->rows, d = p->d;
  const size_t m_bytes = batch * A_msg->cols * d * 4, r_bytes = batch * A_open->cols * d * 4;
  const size_t t_bytes = batch * rows * d * 4;
  const size_t ws = linear_ws_bytes(A_msg, A_open, batch);
  int rc;
  if ((rc = ensure_scratch(p, 6, m_bytes)) || (rc = ensure_scratch(p, 7, r_bytes)) ||
      (rc = ensure_scratch(p, 9, t_bytes)) || (rc = ensure_scratch(p, 10, t_bytes)) ||
      (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  uint32_t* dm = static_cast<uint32_t*>(p->scratch[6].ptr);
  uint32_t* dr = static_cast<uint32_t*>(p->scratch[7].ptr);
  uint32_t* t1 = static_cast<uint32_t*>(p->scratch[9].ptr);
  uint32_t* t2 = static_cast<uint32_t*>(p->scratch[10].ptr);
  rc = cuda_status(cudaMemcpyAsync(dm, m, m_bytes, cudaMemcpyHostToDevice, st));
  if (!rc) rc = cuda_status(cudaMemcpyAsync(dr, r, r_bytes, cudaMemcpyHostToDevice, st));
  if (!rc) {
    Carver cv(p->scratch[8].ptr, ws);
    rc = linear_core(A_msg, A_open, dm, dr, batch, t1, t2, cv, st);
  }
  if (!rc) rc = cuda_status(cudaMemcpyAsync(t, t1, t_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- BDLOP parts: u = A_mask * r, v = A_msg * m + A_open * r ---------- */

int grid_gpu_bdlop_workspace(const grid_gpu_matrix* A_mask, const grid_gpu_matrix* A_msg,
                             const grid_gpu_matrix* A_open, size_t batch, size_t* bytes) {
  if (!A_mask || !A_msg || !A_open || !bytes) return GRID_ERR_NULL_POINTER;
  const grid_gpu_plan* p = A_msg->plan;
  *bytes = commit_ws_bytes(p, A_mask->rows, A_mask->cols, batch) +
           linear_ws_bytes(A_msg, A_open, batch) + words_bytes(batch * A_open->rows * p->d);
  return GRID_OK;
}

int grid_gpu_bdlop_commit_dev(const grid_gpu_matrix* A_mask, const grid_gpu_matrix* A_msg,
                              const grid_gpu_matrix* A_open, const uint32_t* m, const uint32_t* r,
                              size_t batch, uint32_t* u, uint32_t* v, void* workspace,
                              size_t workspace_bytes, void* stream) {
  if (!A_mask || !A_msg || !A_open || ((!m || !r || !u || !v) && batch))
    return GRID_ERR_NULL_POINTER;
  if (A_mask->plan != A_msg->plan || A_open->plan != A_msg->plan)
    return GRID_ERR_INVALID_PARAMETERS;
  // the mask and the opening part multiply the same randomness
  if (A_msg->rows != A_open->rows || A_mask->cols != A_open->cols)
    return GRID_ERR_DIMENSION_MISMATCH;
  if (batch == 0) return GRID_OK;
  if (!dims_ok(batch, A_msg->rows, A_msg->cols) || !dims_ok(batch, A_mask->rows, A_mask->cols))
    return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(m) || !aligned16(r) || !aligned16(u) || !aligned16(v) || !aligned16(workspace))
    return GRID_ERR_MISALIGNED;
  const grid_gpu_plan* p = A_msg->plan;
  cudaStream_t st = (cudaStream_t)stream;
  Carver cv(workspace, workspace_bytes);
  uint32_t* t2 = cv.take<uint32_t>(batch * A_open->rows * p->d);
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  const Carver given = cv;
  int rc = commit_core(A_mask, r, batch, u, cv, st);
  cv = given;
  if (!rc) rc = linear_core(A_msg, A_open, m, r, batch, v, t2, cv, st);
  return rc;
}

int grid_gpu_bdlop_commit(grid_gpu_matrix* A_mask, grid_gpu_matrix* A_msg, grid_gpu_matrix* A_open,
                          const uint32_t* m, const uint32_t* r, size_t batch, uint32_t* u,
                          uint32_t* v) {
  if (!A_mask || !A_msg || !A_open || ((!m || !r || !u || !v) && batch))
    return GRID_ERR_NULL_POINTER;
  if (A_mask->plan != A_msg->plan || A_open->plan != A_msg->plan)
    return GRID_ERR_INVALID_PARAMETERS;
  if (A_msg->rows != A_open->rows || A_mask->cols != A_open->cols)
    return GRID_ERR_DIMENSION_MISMATCH;
  if (batch == 0) return GRID_OK;
  grid_gpu_plan* p = A_msg->plan;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t d = p->d;
  const size_t m_bytes = batch * A_msg->cols * d * 4, r_bytes = batch * A_open->cols * d * 4;
  const size_t u_bytes = batch * A_mask->rows * d * 4, v_bytes = batch * A_msg->rows * d * 4;
  size_t ws = 0;
  int rc = grid_gpu_bdlop_workspace(A_mask, A_msg, A_open, batch, &ws);
  if (rc || (rc = ensure_scratch(p, 6, m_bytes)) || (rc = ensure_scratch(p, 7, r_bytes)) ||
      (rc = ensure_scratch(p, 9, v_bytes)) || (rc = ensure_scratch(p, 10, u_bytes)) ||
      (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, m, m_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(p->scratch[7].ptr, r, r_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = grid_gpu_bdlop_commit_dev(A_mask, A_msg, A_open,
                                   static_cast<uint32_t*>(p->scratch[6].ptr),
                                   static_cast<uint32_t*>(p->scratch[7].ptr), batch,
                                   static_cast<uint32_t*>(p->scratch[10].ptr),
                                   static_cast<uint32_t*>(p->scratch[9].ptr), p->scratch[8].ptr,
                                   ws, st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(u, p->scratch[10].ptr, u_bytes, cudaMemcpyDeviceToHost, st));
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(v, p->scratch[9].ptr, v_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- Gram matrix (garbage g) ------------------------------------------- */

int grid_gpu_gram_workspace(const grid_gpu_plan* p, size_t r, size_t n, size_t* bytes) {
  if (!p || !bytes) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  *bytes = gram_ws_bytes(p, r, n, true);
  return GRID_OK;
}

int grid_gpu_gram_dev(const grid_gpu_plan* p, const uint32_t* S, size_t r, size_t n,
                      uint32_t* G, void* workspace, size_t workspace_bytes, void* stream) {
  if (!p || !S || !G) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(S) || !aligned16(G) || !aligned16(workspace)) return GRID_ERR_MISALIGNED;
  cudaStream_t st = (cudaStream_t)stream;
  if (is_crt(p) && !crt_bound_ok(p, n)) return GRID_ERR_INVALID_PARAMETERS;
  const size_t gw = r * (r + 1) / 2 * p->d;
  const bool pm = gram_pm(p, r, n) && workspace_bytes >= gram_ws_bytes(p, r, n, true);
  const EvalsLayout l(residue_plan(p), pm, n);
  const size_t ldx = l.stride;
  Carver cv(workspace, workspace_bytes);
  uint32_t* s_hat = cv.take<uint32_t>(r * ldx * p->d);
  const size_t ew = l.work(r, r, n, EMM_UPPER);
  uint32_t* work = ew ? cv.take<uint32_t>(ew) : nullptr;
  uint32_t* gj[3] = {};
  if (is_crt(p))
    for (auto& x : gj) x = cv.take<uint32_t>(gw);
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  int rc = GRID_OK;
  for (int j = 0; j < (is_crt(p) ? 3 : 1) && !rc; ++j) {
    const grid_gpu_plan* q = is_crt(p) ? p->crt[j] : p;
    uint32_t* out = is_crt(p) ? gj[j] : G;
    if (pm) {
      rc = launch_ntt_tc_pm(q, S, r, n, s_hat, st);
      if (!rc)
        rc = launch_emm_pm(q, s_hat, s_hat, (int)r, (int)r, (int)n, (int)ldx, (int)ldx, EMM_UPPER,
                           false, out, LimbSpec(), work, st);
      continue;
    }
    rc = launch_ntt(q, MODE_FWD, S, nullptr, s_hat, r * n, st);
    if (!rc)
      rc = launch_emm(q, s_hat, s_hat, (int)r, (int)r, (int)n, (int)n, EMM_UPPER, out, work, st);
    if (!rc) rc = launch_ntt(q, MODE_INV, out, nullptr, out, r * (r + 1) / 2, st);
  }
  if (!rc && is_crt(p)) rc = crt_combine(p, gj[0], gj[1], gj[2], gw, G, st);
  return rc;
}

int grid_gpu_gram(grid_gpu_plan* p, const uint32_t* S, size_t r, size_t n, uint32_t* G) {
  if (!p || !S || !G) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t s_bytes = r * n * p->d * 4, g_bytes = r * (r + 1) / 2 * p->d * 4;
  const size_t ws = gram_ws_bytes(p, r, n, true);
  int rc;
  if ((rc = ensure_scratch(p, 6, s_bytes)) || (rc = ensure_scratch(p, 7, g_bytes)) ||
      (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, S, s_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = grid_gpu_gram_dev(p, static_cast<uint32_t*>(p->scratch[6].ptr), r, n,
                           static_cast<uint32_t*>(p->scratch[7].ptr), p->scratch[8].ptr, ws, st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(G, p->scratch[7].ptr, g_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- garbage h and the amortized witness -------------------------------- */

int grid_gpu_garbage_h_workspace(const grid_gpu_plan* p, size_t r, size_t n, size_t* bytes) {
  if (!p || !bytes) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  *bytes = garbage_h_ws_bytes(p, r, n, true);
  return GRID_OK;
}

int grid_gpu_garbage_h_dev(const grid_gpu_plan* p, const uint32_t* S, const uint32_t* Phi,
                           size_t r, size_t n, uint32_t* H, void* workspace,
                           size_t workspace_bytes, void* stream) {
  if (!p || !S || !Phi || !H) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(S) || !aligned16(Phi) || !aligned16(H) || !aligned16(workspace))
    return GRID_ERR_MISALIGNED;
  cudaStream_t st = (cudaStream_t)stream;
  Carver cv(workspace, workspace_bytes);
  const bool pm = garbage_h_pm(p, r, n) && workspace_bytes >= garbage_h_ws_bytes(p, r, n, true);
  const EvalsLayout l(residue_plan(p), pm, n);
  const size_t ldx = l.stride;
  uint32_t* s_hat = cv.take<uint32_t>(r * ldx * p->d);
  uint32_t* phi_hat = cv.take<uint32_t>(r * ldx * p->d);
  uint32_t* cross = cv.take<uint32_t>(r * r * p->d);
  const size_t ew = l.work(r, r, n, EMM_DENSE);
  uint32_t* work = ew ? cv.take<uint32_t>(ew) : nullptr;
  uint32_t* cj[3] = {};
  if (is_crt(p)) {
    if (!crt_bound_ok(p, n)) return GRID_ERR_INVALID_PARAMETERS;
    for (auto& x : cj) x = cv.take<uint32_t>(r * r * p->d);
  }
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  // point-major: <phi_i, s_j> through to coefficients, symmetrised if sym
  auto cross_pm = [&](const grid_gpu_plan* q, bool sym, uint32_t* out) {
    int rc = launch_ntt_tc_pm(q, S, r, n, s_hat, st);
    if (!rc) rc = launch_ntt_tc_pm(q, Phi, r, n, phi_hat, st);
    if (!rc)
      rc = launch_emm_pm(q, phi_hat, s_hat, (int)r, (int)r, (int)n, (int)ldx, (int)ldx, EMM_DENSE,
                         sym, out, LimbSpec(), work, st);
    return rc;
  };
  // poly-major: out[i][j] = <phi_i, s_j> in plan q's evaluation domain
  auto cross_evals = [&](const grid_gpu_plan* q, uint32_t* out) {
    int rc = launch_ntt(q, MODE_FWD, S, nullptr, s_hat, r * n, st);
    if (!rc) rc = launch_ntt(q, MODE_FWD, Phi, nullptr, phi_hat, r * n, st);
    if (!rc)
      rc = launch_emm(q, phi_hat, s_hat, (int)r, (int)r, (int)n, (int)n, EMM_DENSE, out, work, st);
    return rc;
  };
  if (!is_crt(p)) {
    if (pm) return cross_pm(p, true, H);
    int rc = cross_evals(p, cross);
    if (!rc) rc = launch_symmetrize_half(p, cross, (int)r, H, st);
    if (rc) return rc;
    return launch_ntt(p, MODE_INV, H, nullptr, H, r * (r + 1) / 2, st);
  }
  // ring plan without an NTT for q: the cross products per auxiliary prime,
  // back to coefficients, reconstructed mod q; then the (linear) symmetrisation
  int rc = GRID_OK;
  for (int j = 0; j < 3 && !rc; ++j) {
    if (pm) {
      rc = cross_pm(p->crt[j], false, cj[j]);
    } else {
      rc = cross_evals(p->crt[j], cj[j]);
      if (!rc) rc = launch_ntt(p->crt[j], MODE_INV, cj[j], nullptr, cj[j], r * r, st);
    }
  }
  if (!rc) rc = crt_combine(p, cj[0], cj[1], cj[2], r * r * p->d, cross, st);
  if (!rc) rc = launch_symmetrize_half(p, cross, (int)r, H, st);
  return rc;
}

int grid_gpu_garbage_h(grid_gpu_plan* p, const uint32_t* S, const uint32_t* Phi, size_t r,
                       size_t n, uint32_t* H) {
  if (!p || !S || !Phi || !H) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t s_bytes = r * n * p->d * 4, h_bytes = r * (r + 1) / 2 * p->d * 4;
  const size_t ws = garbage_h_ws_bytes(p, r, n, true);
  int rc;
  if ((rc = ensure_scratch(p, 6, s_bytes)) || (rc = ensure_scratch(p, 9, s_bytes)) ||
      (rc = ensure_scratch(p, 7, h_bytes)) || (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, S, s_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(p->scratch[9].ptr, Phi, s_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = grid_gpu_garbage_h_dev(p, static_cast<uint32_t*>(p->scratch[6].ptr),
                                static_cast<uint32_t*>(p->scratch[9].ptr), r, n,
                                static_cast<uint32_t*>(p->scratch[7].ptr), p->scratch[8].ptr, ws,
                                st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(H, p->scratch[7].ptr, h_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

int grid_gpu_amortize_workspace(const grid_gpu_plan* p, size_t r, size_t n, size_t* bytes) {
  if (!p || !bytes) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  *bytes = amortize_ws_bytes(p, r, n);
  return GRID_OK;
}

int grid_gpu_amortize_dev(const grid_gpu_plan* p, const uint32_t* S, const uint32_t* c, size_t r,
                          size_t n, uint32_t* z, void* workspace, size_t workspace_bytes,
                          void* stream) {
  if (!p || !S || !c || !z) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(S) || !aligned16(c) || !aligned16(z) || !aligned16(workspace))
    return GRID_ERR_MISALIGNED;
  cudaStream_t st = (cudaStream_t)stream;
  Carver cv(workspace, workspace_bytes);
  uint32_t* s_hat = cv.take<uint32_t>(r * n * p->d);
  uint32_t* c_hat = cv.take<uint32_t>(r * p->d);
  if (!is_crt(p)) {
    if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
    if (amortize_tc_fits(p, r, n)) return launch_amortize_tc(p, S, c, r, n, z, s_hat, st);
    int rc = launch_ntt(p, MODE_FWD, S, nullptr, s_hat, r * n, st);
    if (!rc) rc = launch_ntt(p, MODE_FWD, c, nullptr, c_hat, r, st);
    if (!rc) rc = launch_amortize(p, c_hat, s_hat, (int)r, n, z, st);
    if (rc) return rc;
    return launch_ntt(p, MODE_INV, z, nullptr, z, n, st);
  }
  // ring plan without an NTT for q: z[k] = sum_i c_i s_i[k] sums r * d products
  if (!crt_bound_ok(p, r)) return GRID_ERR_INVALID_PARAMETERS;
  const size_t zw = n * p->d;
  uint32_t* zj[3] = {cv.take<uint32_t>(zw), cv.take<uint32_t>(zw), cv.take<uint32_t>(zw)};
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  int rc = GRID_OK;
  for (int j = 0; j < 3 && !rc; ++j) {
    const grid_gpu_plan* q = p->crt[j];
    if (amortize_tc_fits(q, r, n)) {
      rc = launch_amortize_tc(q, S, c, r, n, zj[j], s_hat, st);
      continue;
    }
    rc = launch_ntt(q, MODE_FWD, S, nullptr, s_hat, r * n, st);
    if (!rc) rc = launch_ntt(q, MODE_FWD, c, nullptr, c_hat, r, st);
    if (!rc) rc = launch_amortize(q, c_hat, s_hat, (int)r, n, zj[j], st);
    if (!rc) rc = launch_ntt(q, MODE_INV, zj[j], nullptr, zj[j], n, st);
  }
  if (rc) return rc;
  return crt_combine(p, zj[0], zj[1], zj[2], zw, z, st);
}

int grid_gpu_amortize(grid_gpu_plan* p, const uint32_t* S, const uint32_t* c, size_t r, size_t n,
                      uint32_t* z) {
  if (!p || !S || !c || !z) return GRID_ERR_NULL_POINTER;
  if (!square_dims_ok(p, r, n)) return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t s_bytes = r * n * p->d * 4, c_bytes = r * p->d * 4, z_bytes = n * p->d * 4;
  const size_t ws = amortize_ws_bytes(p, r, n);
  int rc;
  if ((rc = ensure_scratch(p, 6, s_bytes)) || (rc = ensure_scratch(p, 9, c_bytes)) ||
      (rc = ensure_scratch(p, 7, z_bytes)) || (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, S, s_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(p->scratch[9].ptr, c, c_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = grid_gpu_amortize_dev(p, static_cast<uint32_t*>(p->scratch[6].ptr),
                               static_cast<uint32_t*>(p->scratch[9].ptr), r, n,
                               static_cast<uint32_t*>(p->scratch[7].ptr), p->scratch[8].ptr, ws,
                               st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(z, p->scratch[7].ptr, z_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- JL projection ------------------------------------------------------ */

int grid_gpu_jl_workspace(size_t rows, size_t* bytes) {
  if (!bytes) return GRID_ERR_NULL_POINTER;
  *bytes = round_up(jl_scratch_bytes(rows), 256);
  return GRID_OK;
}

int grid_gpu_jl_project_dev(const grid_gpu_plan* p, const uint8_t* seed, size_t rows,
                            const uint32_t* parts, size_t num_parts, size_t cols, size_t d,
                            uint32_t* p_out, int8_t* flat_out, void* workspace,
                            size_t workspace_bytes, void* stream) {
  if (!p || !seed || !p_out || (!parts && cols && num_parts)) return GRID_ERR_NULL_POINTER;
  if (!aligned16(workspace)) return GRID_ERR_MISALIGNED;
  return launch_jl_project(p->f, seed, rows, parts, num_parts, cols, d, p_out, flat_out,
                           workspace, workspace_bytes, p->num_sms, p->d_err, (cudaStream_t)stream);
}

int grid_gpu_jl_project(grid_gpu_plan* p, const uint8_t* seed, size_t rows,
                        const uint32_t* parts, size_t num_parts, size_t cols, size_t d,
                        uint32_t* p_out, int8_t* flat_out) {
  if (!p || !seed || !p_out || (!parts && cols && num_parts)) return GRID_ERR_NULL_POINTER;
  if (rows == 0 || rows > 256 || d == 0 || cols % d) return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t in_bytes = num_parts * cols * 4, flat_bytes = flat_out ? rows * num_parts * cols : 0;
  const size_t ws = round_up(jl_scratch_bytes(rows), 256);
  int rc;
  if ((rc = ensure_scratch(p, 6, in_bytes ? in_bytes : 16)) ||
      (rc = ensure_scratch(p, 7, rows * 4)) || (rc = ensure_scratch(p, 8, ws)) ||
      (flat_bytes && (rc = ensure_scratch(p, 11, flat_bytes))))
    return rc;
  cudaStream_t st = p->stream;
  if (in_bytes)
    rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, parts, in_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = launch_jl_project(p->f, seed, rows, static_cast<uint32_t*>(p->scratch[6].ptr), num_parts,
                           cols, d, static_cast<uint32_t*>(p->scratch[7].ptr),
                           flat_bytes ? static_cast<int8_t*>(p->scratch[11].ptr) : nullptr,
                           p->scratch[8].ptr, ws, p->num_sms, p->d_err, st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(p_out, p->scratch[7].ptr, rows * 4, cudaMemcpyDeviceToHost, st));
  if (!rc && flat_bytes)
    rc = cuda_status(cudaMemcpyAsync(flat_out, p->scratch[11].ptr, flat_bytes,
                                     cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- JL evaluations (aggregation side) --------------------------------- */

int grid_gpu_jl_evals_workspace(size_t* bytes) {
  if (!bytes) return GRID_ERR_NULL_POINTER;
  *bytes = round_up(jl_evals_scratch_bytes(), 256);
  return GRID_OK;
}

int grid_gpu_jl_evals_dev(const grid_gpu_plan* p, const uint8_t* seed, size_t rows,
                          const uint32_t* parts, size_t num_parts, size_t cols, size_t d,
                          uint32_t* evals, void* workspace, size_t workspace_bytes, void* stream) {
  if (!p || !seed || !evals || !parts) return GRID_ERR_NULL_POINTER;
  if (d != p->d) return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(workspace)) return GRID_ERR_MISALIGNED;
  return launch_jl_evals(p->f, seed, rows, parts, num_parts, cols, d, evals, workspace,
                         workspace_bytes, p->num_sms, p->d_err, (cudaStream_t)stream);
}

int grid_gpu_jl_evals(grid_gpu_plan* p, const uint8_t* seed, size_t rows, const uint32_t* parts,
                      size_t num_parts, size_t cols, size_t d, uint32_t* evals) {
  if (!p || !seed || !evals || !parts) return GRID_ERR_NULL_POINTER;
  if (d != p->d || d == 0 || cols == 0 || cols % d || num_parts == 0)
    return GRID_ERR_INVALID_PARAMETERS;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t in_bytes = num_parts * cols * 4, out_bytes = rows * d * 4;
  const size_t ws = round_up(jl_evals_scratch_bytes(), 256);
  int rc;
  if ((rc = ensure_scratch(p, 6, in_bytes)) || (rc = ensure_scratch(p, 7, out_bytes)) ||
      (rc = ensure_scratch(p, 8, ws)))
    return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, parts, in_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = launch_jl_evals(p->f, seed, rows, static_cast<uint32_t*>(p->scratch[6].ptr), num_parts,
                         cols, d, static_cast<uint32_t*>(p->scratch[7].ptr), p->scratch[8].ptr, ws,
                         p->num_sms, p->d_err, st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(evals, p->scratch[7].ptr, out_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- uniform ring elements (seeded commitment-key expansion) ----------- */

int grid_gpu_sample_uniform_polys_workspace(const grid_gpu_plan* p, size_t npolys,
                                            uint64_t accept_max, size_t* bytes) {
  if (!p || !bytes) return GRID_ERR_NULL_POINTER;
  *bytes = round_up(sample_uniform_workspace_bytes(p->f.q, (unsigned long long)npolys * p->d,
                                                   accept_max),
                    256);
  return GRID_OK;
}

int grid_gpu_sample_uniform_polys_dev(const grid_gpu_plan* p, const uint8_t* seed, size_t npolys,
                                      uint64_t accept_max, uint32_t* out, void* workspace,
                                      size_t workspace_bytes, void* stream) {
  if (!p || !seed || (!out && npolys)) return GRID_ERR_NULL_POINTER;
  if (!aligned16(workspace)) return GRID_ERR_MISALIGNED;
  return launch_sample_uniform(p, seed, (unsigned long long)npolys * p->d, accept_max, out,
                               workspace, workspace_bytes, (cudaStream_t)stream);
}

int grid_gpu_sample_uniform_polys(grid_gpu_plan* p, const uint8_t* seed, size_t npolys,
                                  uint64_t accept_max, uint32_t* out) {
  if (!p || !seed || (!out && npolys)) return GRID_ERR_NULL_POINTER;
  if (npolys == 0) return GRID_OK;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t out_bytes = npolys * p->d * 4;
  const size_t ws = round_up(
      sample_uniform_workspace_bytes(p->f.q, (unsigned long long)npolys * p->d, accept_max), 256);
  int rc;
  if ((rc = ensure_scratch(p, 7, out_bytes)) || (rc = ensure_scratch(p, 8, ws))) return rc;
  cudaStream_t st = p->stream;
  rc = launch_sample_uniform(p, seed, (unsigned long long)npolys * p->d, accept_max,
                             static_cast<uint32_t*>(p->scratch[7].ptr), p->scratch[8].ptr, ws, st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(out, p->scratch[7].ptr, out_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- decompositions ---------------------------------------------------- */

int grid_gpu_decompose_balanced_dev(const grid_gpu_plan* p, const uint32_t* polys, size_t npolys,
                                    uint64_t base, size_t num_limbs, uint32_t* out, void* stream) {
  if (!p || ((!polys || !out) && npolys)) return GRID_ERR_NULL_POINTER;
  return launch_decompose_balanced(p, polys, npolys, base, num_limbs, out, (cudaStream_t)stream);
}

int grid_gpu_decompose_balanced(grid_gpu_plan* p, const uint32_t* polys, size_t npolys,
                                uint64_t base, size_t num_limbs, uint32_t* out) {
  if (!p || ((!polys || !out) && npolys)) return GRID_ERR_NULL_POINTER;
  if (base < 2 || num_limbs == 0 || num_limbs > 64) return GRID_ERR_INVALID_PARAMETERS;
  if (npolys == 0) return GRID_OK;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t in_bytes = npolys * p->d * 4, out_bytes = in_bytes * num_limbs;
  int rc;
  if ((rc = ensure_scratch(p, 6, in_bytes)) || (rc = ensure_scratch(p, 7, out_bytes))) return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, polys, in_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = launch_decompose_balanced(p, static_cast<uint32_t*>(p->scratch[6].ptr), npolys, base,
                                   num_limbs, static_cast<uint32_t*>(p->scratch[7].ptr), st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(out, p->scratch[7].ptr, out_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

int grid_gpu_gadget_digits(uint64_t q, uint64_t base, size_t* digits) {
  if (!digits) return GRID_ERR_NULL_POINTER;
  if (base < 2 || q < 3) return GRID_ERR_INVALID_PARAMETERS;
  *digits = gadget_digit_count(q, base);
  return GRID_OK;
}

int grid_gpu_gadget_decompose_dev(const grid_gpu_plan* p, const uint32_t* x, size_t len,
                                  uint64_t base, int digit_major, uint32_t* out, void* stream) {
  if (!p || ((!x || !out) && len)) return GRID_ERR_NULL_POINTER;
  if (base < 2) return GRID_ERR_INVALID_PARAMETERS;
  if (!digit_major && len % p->d) return GRID_ERR_LENGTH_MISMATCH;
  return launch_gadget_decompose(p, x, len, base, gadget_digit_count(p->q, base), digit_major,
                                 out, (cudaStream_t)stream);
}

int grid_gpu_gadget_decompose(grid_gpu_plan* p, const uint32_t* x, size_t len, uint64_t base,
                              int digit_major, uint32_t* out) {
  if (!p || ((!x || !out) && len)) return GRID_ERR_NULL_POINTER;
  if (base < 2) return GRID_ERR_INVALID_PARAMETERS;
  if (!digit_major && len % p->d) return GRID_ERR_LENGTH_MISMATCH;
  if (len == 0) return GRID_OK;
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t k = gadget_digit_count(p->q, base);
  const size_t in_bytes = len * 4, out_bytes = in_bytes * k;
  int rc;
  if ((rc = ensure_scratch(p, 6, in_bytes)) || (rc = ensure_scratch(p, 7, out_bytes))) return rc;
  cudaStream_t st = p->stream;
  rc = cuda_status(cudaMemcpyAsync(p->scratch[6].ptr, x, in_bytes, cudaMemcpyHostToDevice, st));
  if (!rc)
    rc = launch_gadget_decompose(p, static_cast<uint32_t*>(p->scratch[6].ptr), len, base, k,
                                 digit_major, static_cast<uint32_t*>(p->scratch[7].ptr), st);
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(out, p->scratch[7].ptr, out_bytes, cudaMemcpyDeviceToHost, st));
  const int fin = finish_host_call(p, st);
  return rc ? rc : fin;
}

/* ---- fused LaBRADOR prover round ---------------------------------------- */

int grid_gpu_prover_round_workspace(const grid_gpu_matrix* A, size_t r, size_t jl_rows,
                                    size_t* bytes) {
  if (!A || !bytes) return GRID_ERR_NULL_POINTER;
  const grid_gpu_plan* p = A->plan;
  const size_t n = A->cols, kappa = A->rows, d = p->d;
  if (!dims_ok(r, n, kappa) || !square_dims_ok(p, r, n) || !words_fit(r, kappa, d))
    return GRID_ERR_INVALID_PARAMETERS;
  *bytes = round_ws_bytes(p, r, n, kappa, jl_rows, true);
  return GRID_OK;
}

int grid_gpu_prover_round_dev(const grid_gpu_matrix* A, const uint32_t* S, size_t r,
                              uint64_t b1, size_t t1, uint64_t b2, size_t t2,
                              const uint8_t* jl_seed, size_t jl_rows, uint32_t* t_limbs,
                              uint32_t* g, uint32_t* g_limbs, uint32_t* p_out, int8_t* jl_flat,
                              void* workspace, size_t workspace_bytes, void* stream) {
  if (!A || !S || !t_limbs || !g) return GRID_ERR_NULL_POINTER;
  const grid_gpu_plan* p = A->plan;
  const size_t n = A->cols, kappa = A->rows, d = p->d;
  if (!dims_ok(r, n, kappa) || !square_dims_ok(p, r, n) || !words_fit(r, kappa, d))
    return GRID_ERR_INVALID_PARAMETERS;
  if (!aligned16(S) || !aligned16(g) || !aligned16(workspace)) return GRID_ERR_MISALIGNED;
  if (is_crt(p) && !crt_bound_ok(p, n)) return GRID_ERR_INVALID_PARAMETERS;
  cudaStream_t st = (cudaStream_t)stream;
  const bool pm = round_pm(p, r, n, kappa) &&
                  workspace_bytes >= round_ws_bytes(p, r, n, kappa, jl_rows, true);
  const EvalsLayout l(residue_plan(p), pm, n);
  Carver cv(workspace, workspace_bytes);
  const size_t ldx = l.stride;
  uint32_t* s_hat = cv.take<uint32_t>(r * ldx * d);
  const size_t ew = round_work(l, r, n, kappa);
  uint32_t* work = ew ? cv.take<uint32_t>(ew) : nullptr;
  uint32_t* t = cv.take<uint32_t>(r * kappa * d);
  void* jl_ws = cv.take<char>(jl_scratch_bytes(jl_rows ? jl_rows : 1));
  // ring plan without an NTT for q: t and g per auxiliary prime
  const size_t tw = r * kappa * d, gw = r * (r + 1) / 2 * d;
  uint32_t *tj[3] = {}, *gj[3] = {};
  if (is_crt(p))
    for (int j = 0; j < 3; ++j) {
      tj[j] = cv.take<uint32_t>(tw);
      gj[j] = cv.take<uint32_t>(gw);
    }
  if (!cv.ok) return GRID_ERR_INVALID_PARAMETERS;
  // inner commitments and the Gram over the witness's evaluations (one
  // transform shared by both) on plan q into tt / gg, or their limbs (tt unwritten then)
  auto contract = [&](const grid_gpu_plan* q, const grid_gpu_matrix* Aq, uint32_t* tt,
                      uint32_t* gg, const LimbSpec& tl, const LimbSpec& gl, cudaStream_t cs) {
    if (pm && Aq->d_evals_pm) {
      // point-major evaluations: both products load their operands with TMA
      int rc = launch_ntt_tc_pm(q, S, r, n, s_hat, cs);
      if (!rc)
        rc = launch_emm_pm(q, s_hat, Aq->d_evals_pm, (int)r, (int)kappa, (int)n, (int)ldx,
                           (int)Aq->ld_pm, EMM_DENSE, false, tl.out ? nullptr : tt, tl, work, cs,
                           true);
      if (!rc)
        rc = launch_emm_pm(q, s_hat, s_hat, (int)r, (int)r, (int)n, (int)ldx, (int)ldx, EMM_UPPER,
                           false, gg, gl, work, cs, true);
      return rc;
    }
    int rc = launch_ntt(q, MODE_FWD, S, nullptr, s_hat, r * n, cs);
    if (!rc)
      rc = launch_emm(q, s_hat, Aq->d_evals, (int)r, (int)kappa, (int)n, (int)Aq->ld, EMM_DENSE,
                      tt, work, cs);
    if (!rc) rc = launch_ntt(q, MODE_INV, tt, nullptr, tt, r * kappa, cs);
    if (!rc)
      rc = launch_emm(q, s_hat, s_hat, (int)r, (int)r, (int)n, (int)n, EMM_UPPER, gg, work, cs);
    if (!rc) rc = launch_ntt(q, MODE_INV, gg, nullptr, gg, r * (r + 1) / 2, cs);
    return rc;
  };
  // The JL projection reads only S and shares nothing with the commitment and
  // Gram chain: fork both off the caller's stream (chain on the high-priority
  // stream, JL on the low-priority one, so the JL's CTAs fill the SMs the
  // chain leaves idle) and join them back before returning.
  const bool jl = jl_seed && p_out;
  cudaStream_t hi = p->fork_hi, lo = p->fork_lo;
  cudaEvent_t ev[3] = {};
  int rc = GRID_OK;
  for (int i = 0; i < 3 && !rc; ++i)
    rc = cuda_status(cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming));
  if (!rc) rc = cuda_status(cudaEventRecord(ev[0], st));
  if (!rc) rc = cuda_status(cudaStreamWaitEvent(hi, ev[0], 0));
  if (!rc && jl) rc = cuda_status(cudaStreamWaitEvent(lo, ev[0], 0));
  int rc_chain = rc, rc_jl = rc;
  if (!rc) {
    // 3. JL projection of the coefficient vectors (one part per witness vector)
    if (jl)
      rc_jl = launch_jl_project(p->f, jl_seed, jl_rows, S, r, n * d, d, p_out, jl_flat, jl_ws,
                                jl_scratch_bytes(jl_rows), p->num_sms, p->d_err, lo);
    // 1. inner commitments t_i = A s_i and 2. garbage g_ij = <s_i, s_j>, i <= j, with
    // the balanced limbs of both (inner_commit_decomposed, decompose_polys)
    auto spec = [](uint32_t* out, uint64_t base, size_t limbs) {
      return out && aligned16(out) && limbs_ok(base, limbs) ? limb_spec(out, base, limbs)
                                                            : LimbSpec();
    };
    LimbSpec tl = spec(t_limbs, b1, t1), gl = spec(g_limbs, b2, t2);
    if (!is_crt(p)) {
      if (!pm || !A->d_evals_pm) tl = gl = LimbSpec();  // gathering products: a pass of its own
      rc_chain = contract(p, A, t, g, tl, gl, hi);
    } else {
      for (int j = 0; j < 3 && !rc_chain; ++j)
        rc_chain = contract(p->crt[j], A->crt[j], tj[j], gj[j], LimbSpec(), LimbSpec(), hi);
      if (!rc_chain)
        rc_chain = crt_combine(p, tj[0], tj[1], tj[2], tw, tl.out ? nullptr : t, hi, tl);
      if (!rc_chain) rc_chain = crt_combine(p, gj[0], gj[1], gj[2], gw, g, hi, gl);
    }
    if (!rc_chain && !tl.out)
      rc_chain = launch_decompose_balanced(p, t, r * kappa, b1, t1, t_limbs, hi);
    if (!rc_chain && g_limbs && !gl.out)
      rc_chain = launch_decompose_balanced(p, g, r * (r + 1) / 2, b2, t2, g_limbs, hi);
    // join: the caller's stream waits for both forks (also after a failed launch)
    int rj = cuda_status(cudaEventRecord(ev[1], hi));
    if (!rj) rj = cuda_status(cudaStreamWaitEvent(st, ev[1], 0));
    if (!rj && jl) rj = cuda_status(cudaEventRecord(ev[2], lo));
    if (!rj && jl) rj = cuda_status(cudaStreamWaitEvent(st, ev[2], 0));
    rc = rc_chain ? rc_chain : rc_jl ? rc_jl : rj;
  }
  for (cudaEvent_t e : ev)
    if (e) cudaEventDestroy(e);
  return rc;
}

}  // extern "C"
