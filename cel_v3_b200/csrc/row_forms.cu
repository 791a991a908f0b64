// row_forms.cu -- compact forms of a CSR matrix, found when it is uploaded:
//
//   row patterns   the rows use at most kPatMax distinct sequences of column
//                  offsets col - row, none longer than kPatLen (a
//                  structured-grid stencil has a few dozen): one byte per
//                  row indexes the table of sequences;
//   row table      the rows' values repeat too, at most kPatMax distinct
//                  (offsets, values) rows in all (a constant-coefficient
//                  stencil: 27): the byte then indexes a table of whole
//                  rows, and a sweep reads one byte per row for the matrix
//                  instead of 8 per entry and 5 per row;
//   Jacobi table   the diagonal scaling is the same for all rows of an
//                  index: the vector sweeps read it through the byte too.
//
// One pass hashes each row's offsets, and its values while they still repeat,
// into two small sets; a second assigns the bytes and compares every row with
// its set's representative bit by bit, so that the tables are exact whatever
// the hash does.  A set that overflows ends its part of the pass at once: a
// matrix whose values do not repeat costs one look at its columns.
#include <algorithm>
#include <cstring>
#include <vector>

#include "tile_kernels.cuh"

namespace celg {

constexpr int kRowSlots = 1024;

struct RowSets {
  unsigned long long key[2][kRowSlots];  // 0: empty
  int rep[2][kRowSlots];
  int count[2];
  int over[2];
  int mismatch;
  int pad[3];
};

__device__ __forceinline__ unsigned long long hash_step(unsigned long long h, unsigned long long x) {
  h = (h ^ x) * 0xff51afd7ed558ccdull;
  return h ^ (h >> 32);
}

// hash of row i's offsets (and values); 0 is never returned
__device__ __forceinline__ unsigned long long row_hash(const int* __restrict__ ci, const double* __restrict__ v, int b,
                                                       int len, int i, unsigned long long* with_values) {
  unsigned long long h = 0x9e3779b97f4a7c15ull + (unsigned long long)len;
#pragma unroll
  for (int k = 0; k < kPatLen; ++k)
    if (k < len) h = hash_step(h, (unsigned)(ci[b + k] - i));
  if (with_values) {
    unsigned long long g = h;
#pragma unroll
    for (int k = 0; k < kPatLen; ++k)
      if (k < len) g = hash_step(g, (unsigned long long)__double_as_longlong(v[b + k]));
    *with_values = g ? g : 1;
  }
  return h ? h : 1;
}

__device__ __forceinline__ void set_insert(RowSets* s, int w, unsigned long long key, int row) {
  unsigned q = (unsigned)(key >> 40) & (kRowSlots - 1);
  for (int probe = 0; probe < kRowSlots; ++probe) {
    if (*(volatile int*)&s->over[w]) return;
    const unsigned long long cur = *(volatile unsigned long long*)&s->key[w][q];
    if (cur == key) return;
    if (cur == 0) {
      const unsigned long long prev = atomicCAS(&s->key[w][q], 0ull, key);
      if (prev == 0) {
        s->rep[w][q] = row;
        if (atomicAdd(&s->count[w], 1) >= kPatMax) atomicExch(&s->over[w], 1);
        return;
      }
      if (prev == key) return;
    }
    q = (q + 1) & (kRowSlots - 1);
  }
}

// bad: the upload's validation flags (a malformed row pointer is not followed)
__global__ void __launch_bounds__(256) row_sets_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                                       const double* __restrict__ v, const int* __restrict__ bad,
                                                       RowSets* s) {
  constexpr int kSeen = 128;  // keys this CTA has met, by their low bits
  __shared__ unsigned long long seen[2][kSeen];
  for (int q = threadIdx.x; q < 2 * kSeen; q += blockDim.x) (&seen[0][0])[q] = 0;
  __syncthreads();
  if (bad && (bad[0] || bad[1])) return;
  bool values = v != nullptr;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    if (*(volatile int*)&s->over[0]) return;
    if (values && *(volatile int*)&s->over[1]) values = false;
    const int b = rp[i], len = rp[i + 1] - b;
    if (len > kPatLen) {
      atomicExch(&s->over[0], 1);
      atomicExch(&s->over[1], 1);
      return;
    }
    unsigned long long key[2];
    key[0] = row_hash(ci, v, b, len, (int)i, values ? &key[1] : nullptr);
    for (int w = 0; w < (values ? 2 : 1); ++w) {
      volatile unsigned long long* c = &seen[w][key[w] & (kSeen - 1)];
      if (*c == key[w]) continue;
      set_insert(s, w, key[w], (int)i);
      *c = key[w];
    }
  }
}

// The byte of every row (the position of its key among the sorted keys) and
// the tables, each row compared with its representative.
template <bool VALUES>
__global__ void __launch_bounds__(256)
    row_ids_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                   const unsigned long long* __restrict__ keys, const int* __restrict__ reps, int nkeys,
                   uint8_t* __restrict__ pid, int* __restrict__ pat, int* __restrict__ plen,
                   double* __restrict__ rowv, float* __restrict__ rowv32, int* mismatch) {
  __shared__ unsigned long long s_key[kPatMax];
  __shared__ int s_rep[kPatMax];
  for (int q = threadIdx.x; q < nkeys; q += blockDim.x) {
    s_key[q] = keys[q];
    s_rep[q] = reps[q];
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int q = threadIdx.x; q < nkeys * kPatLen; q += blockDim.x) {
      const int r = s_rep[q / kPatLen], k = q % kPatLen, b = rp[r], len = rp[r + 1] - b;
      pat[q] = k < len ? ci[b + k] - r : 0;
      if (VALUES) {
        const double x = k < len ? v[b + k] : 0.0;
        rowv[q] = x;
        rowv32[q] = (float)x;
      }
      if (k == 0) plen[q / kPatLen] = len;
    }
  }
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const int b = rp[i], len = rp[i + 1] - b;
    unsigned long long kv = 0;
    unsigned long long key = row_hash(ci, v, b, len, (int)i, VALUES ? &kv : nullptr);
    if (VALUES) key = kv;
    int lo = 0, hi = nkeys - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_key[mid] < key) lo = mid + 1; else hi = mid;
    }
    const int r = s_rep[lo], rb = rp[r];
    bool same = rp[r + 1] - rb == len;
#pragma unroll
    for (int k = 0; k < kPatLen; ++k)
      if (k < len && same) {
        same = ci[b + k] - (int)i == ci[rb + k] - r;
        if (VALUES) same = same && __double_as_longlong(v[b + k]) == __double_as_longlong(v[rb + k]);
      }
    if (!same) *mismatch = 1;
    pid[i] = (uint8_t)lo;
  }
}

// the Jacobi value of each index, and whether every row has its index's
__global__ void __launch_bounds__(256)
    jacobi_table_kernel(int n, const uint8_t* __restrict__ pid, const int* __restrict__ reps, int npat,
                        const double* __restrict__ J, double* __restrict__ tab, float* __restrict__ tab32,
                        int* mismatch) {
  __shared__ double s_j[kPatMax];
  for (int q = threadIdx.x; q < npat; q += blockDim.x) {
    const double x = J[reps[q]];
    s_j[q] = x;
    if (blockIdx.x == 0) {
      tab[q] = x;
      tab32[q] = (float)x;
    }
  }
  __syncthreads();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    if (__double_as_longlong(J[i]) != __double_as_longlong(s_j[pid[i]])) *mismatch = 1;
}

// The runs of x a tile needs for the offsets in pat (sorted, clusters nearer
// than a tile merged: a run of its own costs kTile elements).  Offset 0 is
// always covered.
static WinPlan plan_window(const int* pat, int count) {
  std::vector<long> off(pat, pat + count);
  off.push_back(0);
  std::sort(off.begin(), off.end());
  WinPlan w;
  for (size_t k = 0; k < off.size();) {
    size_t m = k;
    while (m + 1 < off.size() && off[m + 1] - off[m] < kTile) ++m;
    if (w.nseg == kWinSegs || off[m] - off[k] > 8 * kTile) return WinPlan();
    const int start = (int)(off[k] & ~3L);
    w.start[w.nseg] = start;
    w.len[w.nseg] = (int)((off[m] - start + kTile + 3) & ~3L);
    w.base[w.nseg] = w.total;
    w.total += w.len[w.nseg++];
    k = m + 1;
  }
  return w;
}

void row_forms_free(celg_handle* h, CsrDev& A, bool keep) {
  dev_free(h, A.pat, keep);  // the other arrays are parts of its block
  A.pid = nullptr;
  A.pat = nullptr;
  A.npat = 0;
  A.plen = A.prep = nullptr;
  A.rowv = nullptr;
  A.rowv32 = nullptr;
  A.win = WinPlan();
  A.jtab = nullptr;
  A.jtab32 = nullptr;
  A.jtab_ok = A.juni = false;
}

size_t row_sets_bytes() { return sizeof(RowSets); }

// Queues the search on the stream (results in h->rows_d).
int row_forms_search(celg_handle* h, const CsrDev& A, bool with_values, const int* bad) {
  RowSets* s = static_cast<RowSets*>(h->rows_d);
  CELG_CUDA(cudaMemsetAsync(s, 0, sizeof(RowSets), h->stream));
  if (A.n == 0 || A.nnz == 0) return CELG_OK;
  const int grid = (int)std::max(1L, std::min(((long)A.n + 255) / 256, (long)h->sms * 8));
  row_sets_kernel<<<grid, 256, 0, h->stream>>>(A.n, A.rp, A.ci, with_values ? A.v : nullptr, bad, s);
  CELG_CUDA(cudaGetLastError());
  CELG_CUDA(cudaMemcpyAsync(h->rows_h, s, sizeof(RowSets), cudaMemcpyDeviceToHost, h->stream));
  return CELG_OK;
}

// Builds the forms the search found (the stream has been waited for).  Without
// memory for them the matrix keeps its plain columns.
int row_forms_build(celg_handle* h, CsrDev& A, bool with_values) {
  row_forms_free(h, A);
  if (A.n == 0 || A.nnz == 0) return CELG_OK;
  const RowSets* found = static_cast<const RowSets*>(h->rows_h);
  std::vector<RowSets> keep(1, *found);
  const RowSets& s = keep[0];
  for (int w = with_values ? 1 : 0; w >= 0; --w) {
    if (s.over[w] || s.count[w] > kPatMax || s.count[w] < 1) continue;
    std::vector<std::pair<unsigned long long, int>> rows;
    for (int q = 0; q < kRowSlots; ++q)
      if (s.key[w][q]) rows.emplace_back(s.key[w][q], s.rep[w][q]);
    std::sort(rows.begin(), rows.end());
    const int np = (int)rows.size();
    // one block: pat, plen, reps (ints), the tables of 8-byte values, the bytes
    const size_t ints = (size_t)np * (kPatLen + 2);
    const size_t tab = ((ints * sizeof(int) + 15) & ~(size_t)15);
    const size_t bytes = (tab + (size_t)np * (kPatLen * 12) + kPatMax * 12 + (size_t)np * 8 + 64 + 255) & ~(size_t)255;
    const cudaError_t em = dev_alloc(h, &A.pat, bytes + (size_t)A.n + 16);
    if (out_of_memory(em)) return CELG_OK;
    CELG_CUDA(em);
    A.pid = reinterpret_cast<uint8_t*>(A.pat) + bytes;
    A.npat = np;
    A.plen = A.pat + (size_t)np * kPatLen;
    A.prep = A.plen + np;
    unsigned char* q = reinterpret_cast<unsigned char*>(A.pat) + tab;
    double* rowv = reinterpret_cast<double*>(q);
    double* jtab = rowv + (size_t)np * kPatLen;
    unsigned long long* keys_d = reinterpret_cast<unsigned long long*>(jtab + kPatMax);
    float* rowv32 = reinterpret_cast<float*>(keys_d + np + (np & 1));
    float* jtab32 = rowv32 + (size_t)np * kPatLen;
    // keys and representatives through the pinned block (its contents are in `keep`)
    unsigned long long* kh = static_cast<unsigned long long*>(h->rows_h);
    int* rh = reinterpret_cast<int*>(kh + np);
    for (int k = 0; k < np; ++k) {
      kh[k] = rows[(size_t)k].first;
      rh[k] = rows[(size_t)k].second;
    }
    int* mis = &static_cast<RowSets*>(h->rows_d)->mismatch;
    cudaError_t e = cudaMemcpyAsync(keys_d, kh, sizeof(unsigned long long) * np, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(A.prep, rh, sizeof(int) * np, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(A.pid + A.n, 0, 16, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(mis, 0, sizeof(int), h->stream);
    if (e == cudaSuccess) {
      const int grid = (int)std::max(1L, std::min(((long)A.n + 255) / 256, (long)h->sms * 8));
      if (w)
        row_ids_kernel<true><<<grid, 256, 0, h->stream>>>(A.n, A.rp, A.ci, A.v, keys_d, A.prep, np, A.pid, A.pat,
                                                         A.plen, rowv, rowv32, mis);
      else
        row_ids_kernel<false><<<grid, 256, 0, h->stream>>>(A.n, A.rp, A.ci, nullptr, keys_d, A.prep, np, A.pid, A.pat,
                                                          A.plen, rowv, rowv32, mis);
      e = cudaGetLastError();
    }
    int* mis_h = rh + np;
    int* pat_h = mis_h + 1;
    if (e == cudaSuccess) e = cudaMemcpyAsync(mis_h, mis, sizeof(int), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess && w)
      e = cudaMemcpyAsync(pat_h, A.pat, sizeof(int) * (size_t)np * kPatLen, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
      row_forms_free(h, A);
      return cuda_status(e, "row forms");
    }
    if (*mis_h) {  // two different rows with one hash
      row_forms_free(h, A);
      continue;
    }
    if (w) {
      A.rowv = rowv;
      A.rowv32 = rowv32;
      A.win = plan_window(pat_h, np * kPatLen);
      A.jtab = jtab;
      A.jtab32 = jtab32;
    }
    return CELG_OK;
  }
  return CELG_OK;
}

int row_forms_jacobi(celg_handle* h, CsrDev& A, const double* J) {
  A.jtab_ok = A.juni = false;
  if (!A.rowv || A.n == 0) return CELG_OK;
  int* mis = &static_cast<RowSets*>(h->rows_d)->mismatch;
  CELG_CUDA(cudaMemsetAsync(mis, 0, sizeof(int), h->stream));
  const int grid = (int)std::max(1L, std::min(((long)A.n + 255) / 256, (long)h->sms * 8));
  jacobi_table_kernel<<<grid, 256, 0, h->stream>>>(A.n, A.pid, A.prep, A.npat, J, A.jtab, A.jtab32, mis);
  CELG_CUDA(cudaGetLastError());
  double* th = static_cast<double*>(h->rows_h);
  int* mh = reinterpret_cast<int*>(th + kPatMax);
  CELG_CUDA(cudaMemcpyAsync(th, A.jtab, sizeof(double) * (size_t)A.npat, cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaMemcpyAsync(mh, mis, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  A.jtab_ok = *mh == 0;
  A.juni = A.jtab_ok;
  for (int k = 1; k < A.npat && A.juni; ++k) A.juni = std::memcmp(th + k, th, sizeof(double)) == 0;
  A.jval = th[0];
  return CELG_OK;
}

}  // namespace celg
