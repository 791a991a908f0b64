// elm.cu -- the ELM assembly interface of the reference
// (src/felmsolver/cel_elmsolver_module.f90) on one GPU: row-wise insertion of
// 1-based entries, MatrixCompleted (sort, CSR, Jacobi, optional diagonal
// scaling and JAD), DoIt/ReDoIt with a host right-hand side, CollectSolution
// into a caller-owned buffer.  Single sub-domain only: the MPI gather onto
// reduce-masters (:299-345) has nothing to do on one rank.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "celg_internal.h"

struct Elm {
  int n_total = 0, n_local = 0, row_low = 1;
  std::vector<int> rows, cols;
  std::vector<double> vals;
  std::vector<long long> diag_idx;
  int cur_row = -1;
  // Rows that arrive whole, in order and with ascending columns need no sort:
  // as long as all do (direct), celg_elm_insert_rows copies the caller's
  // columns and values straight into the arrays of the matrix to be (dmat,
  // columns 1-based until it is completed) and keeps the row pointer here;
  // pieces of a few rows are held here until there are enough for a copy.
  // Any other insertion moves the entries to rows/cols/vals above.
  bool direct = true;
  bool lost = false;       // a CUDA error while completing them: nothing is left to retry with
  std::vector<int> rp;     // one entry per row begun, and the end
  celg_mat* dmat = nullptr;
  size_t dcap = 0;         // entries dmat has room for
  size_t sent = 0;         // entries it has; the held ones follow
  std::vector<int> held_cols;
  std::vector<double> held_vals;
  size_t hint = 0;
  celg_mat* mat = nullptr;
  bool completed = false;
  int solver = CELG_SOLVER_GMRES;
  celg_params params;
  int diag_scaling = 1;
  double* b_d = nullptr;
  double* x_d = nullptr;
  bool solved = false;
};

using namespace celg;

extern "C" int celg_elm_destroy(celg_handle* h) {
  if (!h || !h->elm) return CELG_OK;
  Elm* e = h->elm;
  cudaSetDevice(h->device);
  cudaStreamSynchronize(h->stream);
  if (e->mat) celg_mat_destroy(e->mat);
  if (e->dmat) celg_mat_destroy(e->dmat);
  dev_free(h, e->b_d);  // x_d is a part of its block
  delete e;
  h->elm = nullptr;
  return CELG_OK;
}

// Defaults of cel_elmSolverInitialization (:134-151): GMRES with restart
// 4-1 = 3, Jacobi, diagonal scaling, eps 1e-8 (absolute), iter_max 5000,
// CSR, x0 = 1 as in the solvers.
extern "C" int celg_elm_init(celg_handle* h, int n_total, int n_local, int row_low,
                             const int nnz_hint[2]) {
  if (!h || n_total < 0 || n_local < 0) return CELG_ERR_ARG;
  if (n_local != n_total || row_low != 1) return CELG_ERR_ARG;  // one sub-domain
  celg_elm_destroy(h);
  Elm* e = new Elm();
  e->n_total = n_total;
  e->n_local = n_local;
  e->row_low = row_low;
  long long hint = nnz_hint ? (long long)(nnz_hint[0] + nnz_hint[1]) * n_local : 0;
  if (hint > 0 && hint < (1LL << 31)) e->hint = (size_t)hint;
  e->diag_idx.assign((size_t)n_local, -1);
  celg_params_default(&e->params);
  e->params.x0_mode = CELG_X0_REF_ONES;
  e->params.eps_abs = 1e-8;
  e->params.eps_rel = 0.0;
  e->params.iter_max = 5000;
  e->params.restart = 3;
  e->solver = CELG_SOLVER_GMRES;
  e->diag_scaling = 1;
  h->elm = e;
  return CELG_OK;
}

extern "C" int celg_elm_set_solver(celg_handle* h, int solver, const celg_params* p,
                                   int diag_scaling) {
  if (!h || !h->elm || !p) return CELG_ERR_STATE;
  if (solver < CELG_SOLVER_PCG || solver > CELG_SOLVER_GMRES) return CELG_ERR_ARG;
  Elm* e = h->elm;
  if (e->completed && (diag_scaling != 0) != (e->diag_scaling != 0)) return CELG_ERR_STATE;
  e->solver = solver;
  e->params = *p;
  e->diag_scaling = diag_scaling != 0;
  return CELG_OK;
}

extern "C" int celg_elm_row_start(celg_handle* h, int row) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (e->completed) return CELG_ERR_STATE;
  if (row < e->row_low || row >= e->row_low + e->n_local) return CELG_ERR_ARG;
  e->cur_row = row;
  return CELG_OK;
}

// Leaves the direct mode: the rows so far (`sent` of their entries in dmat, the
// columns there from col_base; the rest held here) become triplets on the
// host, in the order they were inserted.  vals_d: their values, null when
// e->vals has them.
static int elm_to_triplets(celg_handle* h, Elm* e, const double* vals_d, int col_base) {
  const size_t nnz = e->rp.empty() ? 0 : (size_t)e->rp.back();
  const size_t room = std::max(nnz, e->hint);
  e->rows.reserve(room);
  e->cols.reserve(room);
  e->vals.reserve(room);
  if (nnz) {
    e->cols.resize(nnz);
    e->vals.resize(nnz);
    if (e->sent) {
      CELG_CUDA(cudaMemcpyAsync(e->cols.data(), e->dmat->csr.ci, sizeof(int) * e->sent, cudaMemcpyDeviceToHost, h->stream));
      if (vals_d)
        CELG_CUDA(cudaMemcpyAsync(e->vals.data(), vals_d, sizeof(double) * e->sent, cudaMemcpyDeviceToHost, h->stream));
      CELG_CUDA(cudaStreamSynchronize(h->stream));
      if (col_base != 1)
        for (size_t k = 0; k < e->sent; ++k) e->cols[k] += 1 - col_base;
    }
    std::copy(e->held_cols.begin(), e->held_cols.end(), e->cols.begin() + (long)e->sent);
    std::copy(e->held_vals.begin(), e->held_vals.end(), e->vals.begin() + (long)e->sent);
    for (size_t r = 0; r + 1 < e->rp.size(); ++r) {
      const int row = e->row_low + (int)r;
      e->rows.insert(e->rows.end(), (size_t)(e->rp[r + 1] - e->rp[r]), row);
      for (int k = e->rp[r]; k < e->rp[r + 1]; ++k)
        if (e->cols[(size_t)k] == row) e->diag_idx[r] = k;
    }
  }
  if (e->dmat) celg_mat_destroy(e->dmat);
  e->dmat = nullptr;
  e->rp.clear();
  e->held_cols.clear();
  e->held_vals.clear();
  e->direct = false;
  return CELG_OK;
}

static int elm_undirect(celg_handle* h, Elm* e) {
  if (!e->direct) return CELG_OK;
  return e->lost ? CELG_ERR_STATE : elm_to_triplets(h, e, e->dmat ? e->dmat->csr.v : nullptr, 1);
}

// Copies total entries (columns, values) behind those that dmat has; *room =
// false (and nothing done) when there is no device memory for them.
static int elm_send(celg_handle* h, Elm* e, const int* cols, const double* vals, size_t total, bool* room) {
  *room = true;
  const size_t need = e->sent + total;
  if (need > e->dcap || !e->dmat) {
    celg_mat* m = new celg_mat();
    m->h = h;
    // (a hint is taken up to twice what is there: it may be far too large, and
    // the room stays with the matrix)
    const size_t room_for = std::max(std::max(need, std::min(e->hint, 2 * need)), e->dmat ? 2 * e->dcap : 0);
    size_t cap = std::min(room_for, ((size_t)1 << 31) - 1);
    cudaError_t ce = alloc_csr_room(m, e->n_local, cap, e->n_local);
    if (ce == cudaErrorMemoryAllocation && cap > need) {
      (void)cudaGetLastError();
      cap = need;
      ce = alloc_csr_room(m, e->n_local, cap, e->n_local);
    }
    if (ce != cudaSuccess) {
      delete m;
      *room = !out_of_memory(ce);
      return *room ? cuda_status(ce, "ELM rows") : CELG_OK;
    }
    if (e->sent) {
      CELG_CUDA(cudaMemcpyAsync(m->csr.ci, e->dmat->csr.ci, sizeof(int) * e->sent, cudaMemcpyDeviceToDevice, h->stream));
      CELG_CUDA(cudaMemcpyAsync(m->csr.v, e->dmat->csr.v, sizeof(double) * e->sent, cudaMemcpyDeviceToDevice, h->stream));
    }
    if (e->dmat) celg_mat_destroy(e->dmat);
    e->dmat = m;
    e->dcap = cap;
  }
  if (total) {
    // (from pageable memory these return when the caller's arrays are read)
    CELG_CUDA(cudaMemcpyAsync(e->dmat->csr.ci + e->sent, cols, sizeof(int) * total, cudaMemcpyHostToDevice, h->stream));
    CELG_CUDA(cudaMemcpyAsync(e->dmat->csr.v + e->sent, vals, sizeof(double) * total, cudaMemcpyHostToDevice, h->stream));
    CELG_CUDA(cudaStreamSynchronize(h->stream));
  }
  e->sent = need;
  return CELG_OK;
}

static int elm_send_held(celg_handle* h, Elm* e, bool* room) {
  const int st = elm_send(h, e, e->held_cols.data(), e->held_vals.data(), e->held_vals.size(), room);
  if (st || !*room) return st;
  e->held_cols.clear();
  e->held_vals.clear();
  return CELG_OK;
}

// Whole rows in order with ascending columns, appended to dmat; *taken is
// false (and nothing done) when the rows are not of that kind, or the device
// has no room for them.  Copies of
// their own cost about 25 us a call, so short pieces are held on the host
// until kElmHold entries are together.
constexpr size_t kElmHold = 4096;
static int elm_append_rows(celg_handle* h, Elm* e, int first_row, int nrows, const int* row_ptr, const int* cols,
                           const double* vals, bool* taken) {
  *taken = nrows == 0;
  if (*taken) return CELG_OK;
  const int base = row_ptr[0];
  const size_t total = (size_t)(row_ptr[nrows] - base);
  const int r0 = first_row - e->row_low;
  const size_t done = e->rp.empty() ? 0 : e->rp.size() - 1;  // rows begun so far
  const size_t at = e->rp.empty() ? 0 : (size_t)e->rp.back();
  if (r0 < (int)done || at + total >= (size_t)1 << 31 || (total > 0 && (!cols || !vals))) return CELG_OK;
  for (int i = 0; i < nrows; ++i)
    if (row_ptr[i + 1] < row_ptr[i]) return CELG_OK;
  bool bad = false;
  for (int i = 0; i < nrows; ++i) {
    const int b = row_ptr[i] - base, end = row_ptr[i + 1] - base;
    if (b == end) continue;
    bad |= cols[b] < 1 || cols[end - 1] > e->n_total;
    for (int k = b + 1; k < end; ++k) bad |= cols[k] < cols[k - 1];
  }
  if (bad) return CELG_OK;
  const size_t held = e->held_vals.size();
  int st = CELG_OK;
  bool room = true;
  if (total < kElmHold) {
    e->held_cols.insert(e->held_cols.end(), cols, cols + total);
    e->held_vals.insert(e->held_vals.end(), vals, vals + total);
    if (held + total >= kElmHold) st = elm_send_held(h, e, &room);
    if (st || !room) {
      e->held_cols.resize(held);
      e->held_vals.resize(held);
    }
  } else {
    if (held) st = elm_send_held(h, e, &room);
    if (!st && room) st = elm_send(h, e, cols, vals, total, &room);
  }
  if (st || !room) return st;
  if (e->rp.empty()) e->rp.push_back(0);
  e->rp.resize((size_t)r0 + 1, (int)at);  // rows left out are empty
  for (int i = 0; i < nrows; ++i) e->rp.push_back((int)at + row_ptr[i + 1] - base);
  *taken = true;
  return CELG_OK;
}

extern "C" int celg_elm_insert(celg_handle* h, int col, double value) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (e->completed || e->cur_row < 0) return CELG_ERR_STATE;
  if (col < 1 || col > e->n_total) return CELG_ERR_ARG;
  if (const int st = elm_undirect(h, e)) return st;
  e->rows.push_back(e->cur_row);
  e->cols.push_back(col);
  e->vals.push_back(value);
  if (col == e->cur_row) e->diag_idx[(size_t)(e->cur_row - e->row_low)] = (long long)e->vals.size() - 1;
  return CELG_OK;
}

// Only the diagonal can be re-inserted; the reference stops with an error
// for off-diagonal entries (:180-184).
extern "C" int celg_elm_reinsert(celg_handle* h, int col, double value) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (e->completed || e->cur_row < 0) return CELG_ERR_STATE;
  if (col != e->cur_row) return CELG_ERR_ARG;
  if (const int st = elm_undirect(h, e)) return st;
  const long long k = e->diag_idx[(size_t)(e->cur_row - e->row_low)];
  if (k < 0) return CELG_ERR_ARG;
  e->vals[(size_t)k] = value;
  return CELG_OK;
}

extern "C" int celg_elm_row_completed(celg_handle* h) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  return CELG_OK;
}

extern "C" int celg_elm_insert_rows(celg_handle* h, int first_row, int nrows, const int* row_ptr,
                                    const int* cols, const double* vals) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (e->completed) return CELG_ERR_STATE;
  if (nrows < 0 || !row_ptr || first_row < e->row_low ||
      first_row + nrows > e->row_low + e->n_local)
    return CELG_ERR_ARG;
  const int base = row_ptr[0];
  const long long total = (long long)row_ptr[nrows] - base;
  if (total < 0) return CELG_ERR_ARG;
  if (e->direct) {
    cudaSetDevice(h->device);
    bool taken = false;
    if (const int st = elm_append_rows(h, e, first_row, nrows, row_ptr, cols, vals, &taken)) return st;
    if (taken) {
      e->cur_row = first_row + nrows - 1;
      return CELG_OK;
    }
    if (const int st = elm_undirect(h, e)) return st;
  }
  e->rows.reserve(e->rows.size() + (size_t)total);
  e->cols.reserve(e->cols.size() + (size_t)total);
  e->vals.reserve(e->vals.size() + (size_t)total);
  for (int i = 0; i < nrows; ++i) {
    const int row = first_row + i;
    if (row_ptr[i + 1] < row_ptr[i]) return CELG_ERR_ARG;
    for (int k = row_ptr[i] - base; k < row_ptr[i + 1] - base; ++k) {
      const int c = cols[k];
      if (c < 1 || c > e->n_total) return CELG_ERR_ARG;
      e->rows.push_back(row);
      e->cols.push_back(c);
      e->vals.push_back(vals[k]);
      if (c == row) e->diag_idx[(size_t)(row - e->row_low)] = (long long)e->vals.size() - 1;
    }
  }
  e->cur_row = first_row + nrows - 1;
  return CELG_OK;
}

// the triplets go to the device as inserted; the stable (row, column) sort
// and the row pointer are built there (assemble.cu)
static int elm_complete_triplets(celg_handle* h, Elm* e, celg_mat** m) {
  const size_t nnz = e->vals.size();
  if (nnz >= (size_t)1 << 31) return CELG_ERR_ARG;
  const size_t nz = std::max<size_t>(nnz, 1);
  int *r_d = nullptr, *c_d = nullptr;
  double* v_d = nullptr;
  cudaError_t ce = raw_alloc(h, &r_d, sizeof(int) * nz);
  if (ce == cudaSuccess) ce = raw_alloc(h, &c_d, sizeof(int) * nz);
  if (ce == cudaSuccess) ce = raw_alloc(h, &v_d, sizeof(double) * nz);
  if (ce == cudaSuccess && nnz)
    ce = cudaMemcpyAsync(r_d, e->rows.data(), sizeof(int) * nnz, cudaMemcpyHostToDevice, h->stream);
  if (ce == cudaSuccess && nnz)
    ce = cudaMemcpyAsync(c_d, e->cols.data(), sizeof(int) * nnz, cudaMemcpyHostToDevice, h->stream);
  if (ce == cudaSuccess && nnz)
    ce = cudaMemcpyAsync(v_d, e->vals.data(), sizeof(double) * nnz, cudaMemcpyHostToDevice, h->stream);
  int st = ce == cudaSuccess ? coo_to_mat_device(h, e->n_local, e->n_local, (int)nnz, r_d, c_d, v_d,
                                                 e->row_low, 1, m)
                             : cuda_status(ce, "ELM triplet upload");
  cudaStreamSynchronize(h->stream);
  cudaFree(r_d);
  cudaFree(c_d);
  cudaFree(v_d);
  return st;
}

// the rows are in place: their pointer follows (without room for the last of
// them they become triplets)
static int elm_complete_direct(celg_handle* h, Elm* e) {
  const int nnz = e->rp.back();
  e->rp.resize((size_t)e->n_local + 1, nnz);
  bool room = true;
  int st = elm_send_held(h, e, &room);
  if (!st && !room) st = elm_undirect(h, e);
  if (st || !room) return st;
  celg_mat* d = e->dmat;
  st = set_csr_entries(d, nnz);
  if (st) return st;
  e->lost = true;  // until the columns, 0-based from here on, are known to be whole
  // (the row pointer is 1-based like the columns, for one conversion)
  for (int& v : e->rp) v += 1;
  const cudaError_t ce =
      cudaMemcpyAsync(d->csr.rp, e->rp.data(), sizeof(int) * e->rp.size(), cudaMemcpyHostToDevice, h->stream);
  st = ce == cudaSuccess ? finish_csr(h, d, 1) : cuda_status(ce, "ELM row pointer");
  for (int& v : e->rp) v -= 1;
  if (!st) e->lost = false;
  return st;
}

// Scaling overwrites the values that direct rows have on the device alone: a
// copy of them for the forms whose set-up after it can run out of memory.
static int elm_keep_values(celg_handle* h, Elm* e, const celg_mat* m, double** plain) {
  const size_t bytes = sizeof(double) * (size_t)m->csr.nnz;
  if (dev_alloc(h, plain, bytes) == cudaSuccess) {
    CELG_CUDA(cudaMemcpyAsync(*plain, m->csr.v, bytes, cudaMemcpyDeviceToDevice, h->stream));
    return CELG_OK;
  }
  (void)cudaGetLastError();
  e->vals.resize((size_t)m->csr.nnz);
  CELG_CUDA(cudaMemcpyAsync(e->vals.data(), m->csr.v, bytes, cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  return CELG_OK;
}

// cel_elmSolverMatrixCompleted (:193-439) for one rank: entries sorted by
// row, then column (cel_sp_mat_format_sparse_31_sort,
// src/fspmt/cel_sp_mat_module.f90:518-585; equal keys keep insertion order)
// and the CSR row pointer (cel_sp_mat_to_csr, :430-456), both on the device;
// then Jacobi, optional diagonal scaling (:375-388 of the ELM module), JAD
// when selected.  When a step fails (no memory left) the entries are kept, so
// that the call can be repeated.
extern "C" int celg_elm_matrix_completed(celg_handle* h) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (e->completed || e->lost) return CELG_ERR_STATE;
  int st = e->direct && !e->rp.empty() ? elm_complete_direct(h, e) : CELG_OK;
  if (st) return st;
  const bool direct = e->direct && !e->rp.empty();
  celg_mat* m = direct ? e->dmat : nullptr;
  if (!direct && (st = elm_complete_triplets(h, e, &m))) return st;
  const size_t n = ((size_t)std::max(1, e->n_local) + 31) & ~(size_t)31;
  const bool jad = e->params.fmt == CELG_FMT_JAD, fp32 = e->params.precision == CELG_PREC_FP32_IR;
  double* plain = nullptr;
  st = celg_mat_jacobi(m);
  if (!st && !e->b_d && dev_alloc(h, &e->b_d, sizeof(double) * 2 * n) != cudaSuccess) {
    (void)cudaGetLastError();
    st = CELG_ERR_CUDA;
  }
  e->x_d = e->b_d + n;
  if (!st && direct && e->diag_scaling && (jad || fp32)) st = elm_keep_values(h, e, m, &plain);
  auto forms = [&]() -> int {
    int s = e->diag_scaling ? celg_mat_scale_diagonal(m) : CELG_OK;
    if (!s && jad) s = celg_mat_to_jad(m, nullptr);
    if (!s && fp32) s = celg_mat_make_fp32(m);
    return s;
  };
  if (!st) st = forms();
  if (st && plain) {
    // the copy may be what there was no room beside: to the host with it
    e->vals.resize((size_t)m->csr.nnz);
    if (cudaMemcpyAsync(e->vals.data(), plain, sizeof(double) * e->vals.size(), cudaMemcpyDeviceToHost, h->stream) ==
            cudaSuccess &&
        cudaStreamSynchronize(h->stream) == cudaSuccess) {
      dev_free(h, plain, false);
      plain = nullptr;
      st = forms();
    }
  }
  dev_free(h, plain);
  if (st) {
    if (!direct) {
      celg_mat_destroy(m);
    } else if (m->scaled && e->vals.empty()) {
      e->lost = true;
    } else {
      e->lost = elm_to_triplets(h, e, m->scaled ? nullptr : m->csr.v, 0) != CELG_OK;
    }
    return st;
  }
  e->mat = m;
  e->dmat = nullptr;
  e->completed = true;
  std::vector<int>().swap(e->rp);
  std::vector<int>().swap(e->rows);
  std::vector<int>().swap(e->cols);
  std::vector<double>().swap(e->vals);
  return CELG_OK;
}

// cel_elmSolverDoIt (:441-651): b copied from the host, divided by sqrt|d|
// when the matrix is scaled (cel_sp_mat_distr_boundary_diag_scale), solved;
// iierr is the status (0 = converged), niter the iteration count of the
// solver (outer iterations for GMRES) and ftol its final residual norm.
extern "C" int celg_elm_doit(celg_handle* h, const double* b, int* iierr, int* niter,
                             double* ftol) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (!e->completed) return CELG_ERR_STATE;
  if (!b && e->n_local > 0) return CELG_ERR_ARG;
  cudaSetDevice(h->device);
  const size_t n = (size_t)e->n_local;
  CELG_CUDA(cudaMemcpyAsync(e->b_d, b, sizeof(double) * n, cudaMemcpyHostToDevice, h->stream));
  int st = CELG_OK;
  if (e->diag_scaling) st = launch_scale_vec(h, (long)n, e->b_d, e->mat->scale, e->b_d, 1);
  if (st) return st;
  celg_result res;
  std::memset(&res, 0, sizeof(res));
  celg_params p = e->params;
  int ret;
  if (e->solver == CELG_SOLVER_PCG) ret = celg_pcg_jacobi(h, e->mat, e->b_d, e->x_d, &p, &res);
  else if (e->solver == CELG_SOLVER_CG) ret = cg_solve(h, e->mat, e->b_d, e->x_d, &p, &res);
  else ret = gmres_solve(h, e->mat, e->b_d, e->x_d, &p, &res);
  e->solved = ret == CELG_OK || ret == CELG_ERR_NOCONV;
  if (iierr) *iierr = ret;
  if (niter) *niter = res.iter_done;
  if (ftol) *ftol = res.final_norm2;
  return ret;
}

extern "C" int celg_elm_redoit(celg_handle* h, const double* b, int* iierr, int* niter,
                               double* ftol) {
  return celg_elm_doit(h, b, iierr, niter, ftol);
}

extern "C" int celg_elm_collect_solution(celg_handle* h, double* x) {
  if (!h || !h->elm) return CELG_ERR_STATE;
  Elm* e = h->elm;
  if (!e->solved) return CELG_ERR_STATE;
  if (!x && e->n_local > 0) return CELG_ERR_ARG;
  CELG_CUDA(cudaMemcpyAsync(x, e->x_d, sizeof(double) * (size_t)e->n_local, cudaMemcpyDeviceToHost,
                            h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  return CELG_OK;
}

extern "C" int celg_elm_performance(celg_handle* h, double* solve_ms, int* iters,
                                    double* bytes_per_iter) {
  if (!h) return CELG_ERR_ARG;
  if (solve_ms) *solve_ms = h->last_ms;
  if (iters) *iters = h->last_iters;
  if (bytes_per_iter) *bytes_per_iter = h->last_bytes_per_iter;
  return CELG_OK;
}
