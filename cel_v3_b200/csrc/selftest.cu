// selftest.cu -- check of the bounded device waits.
//
// Every spin-wait of the library's kernels (the mbarrier waits of the bulk-copy
// pipelines, the polls of words in global memory of the one-kernel solves and
// of the GMRES orthogonalisation) gives up after a time limit, records
// CELG_ERR_TIMEOUT and returns, so that a wait which can never end turns into
// an error status instead of a hung GPU.  celg_check_bounded_wait runs those
// same waits on an mbarrier that nothing ever arrives on and on a word that
// nothing publishes, with a short limit, and reports the status the host reads
// back when both gave up; the context stays usable afterwards.
#include "tile_kernels.cuh"

namespace celg {

// CTA 0 waits on an mbarrier (err[0]), the warps of CTA 1 on a word (err[1]):
// the first to give up makes the others of its CTA give up.
__global__ void bounded_wait_probe_kernel(int* err, const unsigned long long* word, unsigned long long limit_ns) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int abort_;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);  // expects one arrival; none will come
    fence_mbar_init();
    abort_ = 0;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) (void)mbar_wait_bounded(&bar, 0u, err, limit_ns);
    return;
  }
  unsigned long long t0 = 0;
  for (unsigned i = 0; *(volatile const unsigned long long*)word == ~0ull && poll_more(i, t0, &abort_, limit_ns); ++i) {
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_) atomicExch(err + 1, kErrTimeout);
}

}  // namespace celg

extern "C" int celg_check_bounded_wait(celg_handle* h, int limit_ms, int* status) {
  if (!h || !status || limit_ms <= 0 || limit_ms > 10000) return CELG_ERR_ARG;
  CELG_CUDA(cudaSetDevice(h->device));
  // err_d: the two error words, and at 8 the word that is not published
  int* word = h->err_d + 8;
  CELG_CUDA(cudaMemsetAsync(h->err_d, 0, 2 * sizeof(int), h->stream));
  CELG_CUDA(cudaMemsetAsync(word, 0xff, sizeof(unsigned long long), h->stream));
  celg::bounded_wait_probe_kernel<<<2, 64, 0, h->stream>>>(
      h->err_d, reinterpret_cast<const unsigned long long*>(word), (unsigned long long)limit_ms * 1000000ull);
  CELG_CUDA(cudaGetLastError());
  int got[2] = {0, 0};
  CELG_CUDA(cudaMemcpyAsync(got, h->err_d, sizeof(got), cudaMemcpyDeviceToHost, h->stream));
  CELG_CUDA(cudaStreamSynchronize(h->stream));
  CELG_CUDA(cudaMemsetAsync(h->err_d, 0, 2 * sizeof(int), h->stream));
  *status = got[0] == got[1] ? got[0] : CELG_OK;
  return CELG_OK;
}
