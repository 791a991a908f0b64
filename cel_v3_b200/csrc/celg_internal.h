// celg_internal.h -- host-side objects of libcelgpu.so (not part of the ABI).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/celgpu.h"

namespace celg {

// Device copy of a CSR matrix, 0-based.  row_ptr has n+1+4 entries and
// cols/vals nnz+4 (tails filled with nnz / 0) so that the 16-byte rounded
// bulk copies of the SpMV pipeline never leave the allocation.
// Runs of x that a tile needs for the column offsets of a row table
// (csr_win_kernel).
constexpr int kWinSegs = 8;
struct WinPlan {
  int nseg = 0;          // 0: no plan (too many runs or too much to stage)
  int total = 0;         // staged elements of a tile
  int start[kWinSegs];   // first offset of the run from the tile's first row, a multiple of 4
  int len[kWinSegs];     // elements, a multiple of 4
  int base[kWinSegs];    // position in the stage
};

struct CsrDev {
  int n = 0;
  int nnz = 0;
  int ncols = 0;          // n, or more for a row block with halo columns

  int* rp = nullptr;
  int* ci = nullptr;
  double* v = nullptr;
  float* v32 = nullptr;   // FP32 copy (refinement inner solve), nnz+32
  int cap = 0;            // staged entries per 256-row sub-tile
  // column indices as 1-byte indices into a dictionary of column offsets
  // (col - row), when the matrix has at most 256 of them (FP32 copy and
  // the FP64 PCG sweeps)
  uint8_t* ci8 = nullptr; // nnz+32
  int* dict = nullptr;    // ndict offsets, ascending
  int ndict = 0;
  int cap_dict = 0;       // staging capacity with 16-entry alignment
  // row patterns (row_forms.cu): one pattern index per row (n + 16 bytes)
  // and the pattern table (npat x 8 column offsets; the arrays after pat are
  // parts of its allocation)
  uint8_t* pid = nullptr;
  int* pat = nullptr;
  int npat = 0;
  int* plen = nullptr;       // entries of each pattern
  int* prep = nullptr;       // a row of each pattern
  // row table: the values too are those of the pattern index (npat x 8)
  double* rowv = nullptr;
  float* rowv32 = nullptr;
  WinPlan win;
  // Jacobi value of each pattern index, when all its rows have the same
  double* jtab = nullptr;
  float* jtab32 = nullptr;
  bool jtab_ok = false;
  bool juni = false;         // one value for all rows
  double jval = 0.0;
  // copy in slices of 32 rows for the one-kernel solve (pcg_onchip.cu)
  double* sell_v = nullptr;
  float* sell_v32 = nullptr;
  int* sell_c = nullptr;     // columns (no row patterns)
  int* sell_base = nullptr;  // first entry / 32 of each slice (no row patterns)
  long sell_total = -1;      // entries; -1: not looked at yet, 0: not worth it
};

struct JadDev {
  int mmax = -1;          // -1: not built
  int* begin = nullptr;   // mmax+1
  int* ci = nullptr;      // nnz
  double* v = nullptr;    // nnz
  int* perm = nullptr;    // n
  uint8_t* pid = nullptr; // pattern index of each permuted row (n + 16), with row patterns
};

struct PcgState;  // device scalar state of one solve (pcg_internal.cuh)

struct GraphEntry {
  std::string key;
  cudaGraph_t graph;
  cudaGraphExec_t exec;
};

}  // namespace celg

struct celg_handle {
  int device = 0;
  cudaStream_t stream = nullptr;      // work stream (owned, or the caller's)
  bool own_stream = false;
  cudaStream_t cap_stream = nullptr;  // private stream used only to capture graphs
  int sms = 148;
  // reduction scratch: partials (2 rows of max tiles) and a completion ticket
  double* partials = nullptr;
  size_t partials_cap = 0;   // doubles
  unsigned* ticket = nullptr;
  int* err_d = nullptr;      // device error word (bounded waits)
  double* scal_d = nullptr;  // small device scalars for blas1 results
  double* scal_h = nullptr;  // pinned mirror
  // row-form search (row_forms.cu): its sets on the device and a pinned copy
  void* rows_d = nullptr;
  void* rows_h = nullptr;
  // PCG work vectors
  double* wr = nullptr;
  double* wp = nullptr;
  double* wv = nullptr;
  double* wq = nullptr;  // second PCG direction (paired K3)
  size_t wcap = 0;           // elements
  double* wz = nullptr;      // z = M r of block-Jacobi solves (wzcap elements)
  size_t wzcap = 0;
  celg::PcgState* state_d = nullptr;
  celg::PcgState* state_h = nullptr;  // pinned
  void* ru_state_d = nullptr;         // reliable-update solver state
  void* ru_state_h = nullptr;         // pinned
  // cached solve graphs (keyed by matrix, vectors and parameters)
  std::vector<celg::GraphEntry> graphs;
  double* hist_d = nullptr;
  int hist_cap = 0;
  // largest cooperative grid known to be accepted, smallest known to be
  // refused (coop_fits; 0: none yet)
  int coop_ok = 0, coop_no = 0;
  // exchange slots of the one-kernel solve (oc_cap doubles)
  double* oc_slots = nullptr;
  size_t oc_cap = 0;
  // the same for many systems side by side: work vectors, pinned states, and
  // the streams and events of its lanes (lane 0 is the handle's stream)
  double* oc_work = nullptr;
  size_t oc_work_cap = 0;
  celg::PcgState* oc_states = nullptr;
  int oc_states_cap = 0;
  cudaStream_t oc_lane[8] = {};
  cudaEvent_t oc_event[8] = {};
  int batch_path = -1;  // of the last batched solve: CELG_BATCH_SWEEPS or CELG_BATCH_KERNELS, -1 before the first
  // host-buffer solve staging (stable pointers keep cached graphs valid)
  double* sb = nullptr;
  double* sx = nullptr;
  size_t scap = 0;
  // FP32 refinement work vectors
  float* f32 = nullptr;   // 6 vectors of f32cap floats
  size_t f32cap = 0;
  double* ir_d = nullptr; // FP64 correction / residual
  size_t ircap = 0;
  // ELM assembly state
  struct Elm* elm = nullptr;
  // concatenated systems of the last batched solve
  struct Batch* batch = nullptr;
  // work vectors and per-column state of multi-right-hand-side solves
  struct Multi* multi = nullptr;
  // GMRES(m) work space (V, Z, H) and device state, kept between solves
  double* gm_work = nullptr;
  size_t gm_cap = 0;          // doubles
  void* gm_state_d = nullptr;
  void* gm_state_h = nullptr; // pinned
  void* gm_exch = nullptr;    // exchange words of its one-kernel orthogonalisation
  // last solve timing
  float last_ms = 0.f;
  int last_iters = 0;
  double last_bytes_per_iter = 0.0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // tile order of the next sweep (RedCtx::sweep bit 0)
  int sweep_rev = 0;
  // blocks of dev_alloc in use, and given back ones kept for the next request
  struct DevBlock {
    void* p;
    size_t bytes;
  };
  std::vector<DevBlock> blocks, spare;
  size_t spare_bytes = 0;
};

struct celg_mat {
  celg_handle* h = nullptr;
  celg::CsrDev csr;
  celg::JadDev jad;
  double* diag = nullptr;     // n
  double* jacobi = nullptr;   // n
  float* jacobi32 = nullptr;  // n
  double* scale = nullptr;    // sqrt|d| when row-scaled, else null
  double* bjinv = nullptr;    // n x bj_bs inverse diagonal blocks (block Jacobi)
  bool dict_tried = false;    // the offset dictionary was attempted (csr.ci8 set if it fits)
  int bj_bs = 0;
  bool scaled = false;
  // 1 when a stream that is not its handle's may hold work on the arrays:
  // another handle multiplied with it, or a call was captured into a graph
  // that runs wherever the caller launches it (note_use)
  mutable int elsewhere = 0;
};

namespace celg {

int cuda_status(cudaError_t e, const char* what);
#define CELG_CUDA(call)                                       \
  do {                                                        \
    cudaError_t e_ = (call);                                  \
    if (e_ != cudaSuccess) return ::celg::cuda_status(e_, #call); \
  } while (0)

// e says that there was no memory (the error is cleared): what is only kept
// for speed is then left out.
bool out_of_memory(cudaError_t e);

// Device memory of the handle's matrices.  Blocks given back are kept for
// later requests on the handle, in the order of its stream, up to
// kSpareBytes in all (getting and returning a block costs 0.1-0.2 ms each,
// at times milliseconds); celg_destroy frees them, and so does any allocation
// of the handle that finds no other memory.  keep = false: the block
// goes back to the device, which waits for all work on it, on every stream.
constexpr size_t kSpareBlock = (size_t)32 << 20, kSpareBytes = (size_t)96 << 20;
cudaError_t dev_alloc_bytes(celg_handle* h, void** p, size_t bytes);
void dev_free(celg_handle* h, void* p, bool keep = true);
void dev_free_spare(celg_handle* h);
template <typename T>
cudaError_t dev_alloc(celg_handle* h, T** p, size_t bytes) {
  void* q = nullptr;
  const cudaError_t e = dev_alloc_bytes(h, &q, bytes);
  *p = static_cast<T*>(q);
  return e;
}
// cudaMalloc for everything else of a handle (given back with cudaFree): the
// spare blocks make room when there is none left.
cudaError_t raw_alloc_bytes(celg_handle* h, void** p, size_t bytes);
template <typename T>
cudaError_t raw_alloc(celg_handle* h, T** p, size_t bytes) {
  void* q = nullptr;
  const cudaError_t e = raw_alloc_bytes(h, &q, bytes);
  *p = static_cast<T*>(q);
  return e;
}
int ensure_partials(celg_handle* h, long ntiles, int nred);
void graph_cache_clear(celg_handle* h);
void graph_cache_drop_matrix(celg_handle* h, const void* m);
int ensure_work(celg_handle* h, size_t n);
long ntiles_of(long n);
int grid_for_tiles(celg_handle* h, long ntiles, int blocks_per_sm);

// spmv.cu
int launch_spmv_csr(celg_handle* h, const CsrDev& A, const double* x, double* y, int accumulate);
int launch_spmv_csr_f32(celg_handle* h, const CsrDev& A, const float* x, float* y, int accumulate);
int launch_spmv_jad(celg_handle* h, const CsrDev& A, const JadDev& J, const double* x, double* y);
int csr_compute_cap(celg_handle* h, CsrDev& A);
int csr_span_launch(celg_handle* h, const CsrDev& A, int* out);
void csr_set_cap(CsrDev& A, int span);

// blas1.cu
int launch_dot(celg_handle* h, long n, const double* a, const double* b, double* out_d, int take_sqrt);
int launch_axpy(celg_handle* h, long n, double alpha, const double* x, double* y);
int launch_xpby(celg_handle* h, long n, const double* x, double beta, double* y);
int launch_mul(celg_handle* h, long n, const double* a, const double* b, double* z);
int launch_residual(celg_handle* h, celg_mat* m, int fmt, const double* b, const double* x,
                    double* r, double* norm_out_d);
int launch_jacobi_setup(celg_handle* h, celg_mat* m);
int launch_row_scale(celg_handle* h, celg_mat* m);
int launch_to_f32(celg_handle* h, long n, const double* a, float* b);
int launch_scale_vec(celg_handle* h, long n, const double* a, const double* s, double* out, int divide);

// pcg.cu / gmres.cu / ir.cu
int pcg_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
              celg_result* res);
int cg_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
             celg_result* res);
int gmres_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
                celg_result* res);
int ir_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
             celg_result* res);
int ru_solve(celg_handle* h, celg_mat* m, const double* b, double* x, const celg_params* p,
             celg_result* res);
int ensure_f32(celg_handle* h, size_t n);
// api.cu: matrix storage (alloc_csr leaves row_ptr/cols/vals for the caller
// to fill; finish_csr shifts to 0-based, validates and sets the staging cap)
// Build the 1-byte column offsets of the matrix once (no-op when built,
// attempted before, or the matrix has more than 256 column offsets).
int ensure_offset_dict(celg_handle* h, celg_mat* m);
// the same for any CSR array set (left unset beyond 256 distinct offsets)
int build_offset_dict_csr(celg_handle* h, CsrDev& A);
// pcg_onchip.cu: whether the driver accepts a cooperative grid of that many
// CTAs, one per SM, on the handle's stream.
int coop_fits(celg_handle* h, int grid, bool* fits);
// pcg_onchip.cu: drop the sliced copy (the values changed, or the matrix goes)
void sell_free(celg_handle* h, CsrDev& A);
// row_forms.cu
size_t row_sets_bytes();
int row_forms_search(celg_handle* h, const CsrDev& A, bool with_values, const int* bad);
int row_forms_build(celg_handle* h, CsrDev& A, bool with_values);
int row_forms_jacobi(celg_handle* h, CsrDev& A, const double* J);
void row_forms_free(celg_handle* h, CsrDev& A, bool keep = true);
int alloc_csr(celg_mat* m, int n, int nnz, int ncols);
cudaError_t alloc_csr_room(celg_mat* m, int n, size_t nnz_cap, int ncols);
int set_csr_entries(celg_mat* m, int nnz);
int finish_csr(celg_handle* h, celg_mat* m, int base);
void free_mat_arrays(celg_mat* m);
// An operator that queues work on m and returns, on h's stream.
void note_use(celg_handle* h, const celg_mat* m);
// assemble.cu: COO (device arrays, row and column bases) -> CSR matrix
int coo_to_mat_device(celg_handle* h, int n, int ncols, int nnz, const int* rows_d,
                      const int* cols_d, const double* vals_d, int row_base, int col_base,
                      celg_mat** out);
// dist.cu / dist_solve.cu: the one-call distributed solve's data on a celg_dist
int dist_internals(celg_dist* d, celg_handle** h, int* n, int* ncols, void*** solve_slot);
void dist_solve_free(void* solve);
// pcg.cu: bytes of the matrix that one sweep reads, values of vt bytes: in the
// most compact form it has, or (table = false) without the row table, or
// (compact = false) with its int32 columns.
double matrix_sweep_bytes(const CsrDev& A, int vt, bool compact = true, bool table = true);
// pcg.cu: bytes of J that K2 and K3 of an iteration do not read
double jacobi_saved_bytes(const CsrDev& A, int vt);
void batch_free(::Batch* b);
void multi_free(::Multi* m);
void multi_forget_matrix(::Multi* m, const void* mat);
int multi_tuned_cfg(::Multi* m);  // the SpMM variant the tuner picked, -1 if none
int multi_tuned_cfg32(::Multi* m);  // the FP32 SpMM shape the tuner picked, -1 if none

}  // namespace celg
