// Internal declarations shared by the translation units of libibem_gb300.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>

#include "../../include/ibem_gb300.h"

namespace ibem {

// Record a failure message for ibem_last_error() and return `st`.
ibem_status fail(ibem_status st, const std::string& msg);
ibem_status cuda_fail(cudaError_t e, const char* where);

#define IBEM_CUDA(call)                                        \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return ::ibem::cuda_fail(e_, #call); \
  } while (0)

#define IBEM_LAUNCH_CHECK(where)                                \
  do {                                                          \
    cudaError_t e_ = cudaGetLastError();                        \
    if (e_ != cudaSuccess) return ::ibem::cuda_fail(e_, where); \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// What the library sets up once, on first use, must not end a stream capture that this or another
// thread has under way: calls that the runtime counts as unsafe there are made inside one of these.
struct CaptureSafe {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  CaptureSafe() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~CaptureSafe() { cudaThreadExchangeStreamCaptureMode(&mode); }
  CaptureSafe(const CaptureSafe&) = delete;
  CaptureSafe& operator=(const CaptureSafe&) = delete;
};

// Stream-ordered device memory for the library's buffers and workspaces, from a pool of its own
// (one per device, made on first use): allocation and release are queued on the stream, safe
// from any thread and stream.  Between calls the pool keeps at most kPoolKeep bytes (what is
// beyond goes back at the next synchronisation), because mapping and unmapping memory on
// every call cost more than the small solves themselves (a training step: 0.4 of 1.3 ms; six
// ellipsoid realisations on four threads: 19 of 34 ms in cudaMalloc alone); an allocation that
// fails gives everything kept back and tries again.  pool_kept: bytes that the current device's
// pool holds unused; pool_trim gives them back.
constexpr size_t kPoolKeep = (size_t)1 << 30;
cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t st);
void pool_free(void* p, cudaStream_t st);
size_t pool_kept();
cudaError_t pool_trim();
template <class T>
cudaError_t pool_alloc(T** p, size_t bytes, cudaStream_t st) {
  return pool_alloc(reinterpret_cast<void**>(p), bytes, st);
}

// Counts kernel launches of this library (read through ibem_kernel_launches); every
// launch site is written `::ibem::count_launch(), kernel<<<...>>>(...)`.
int count_launch();
long long launches_so_far();

// ---- sphere kernels (sphere24.cu / sphere60.cu / sphere78.cu) ----
struct SphLaunch {
  const double* cen;
  const double* rad;
  int num;
  double E0, nu0, E1, nu1;
};
ibem_status launch_pair24(const SphLaunch& p, double* A, int64_t lda, int64_t row0, int64_t col0, cudaStream_t st);
ibem_status launch_pair60(const SphLaunch& p, double* A, int64_t lda, int64_t row0, int64_t col0, cudaStream_t st);
ibem_status launch_pair78(const SphLaunch& p, double* A, int64_t lda, int64_t row0, int64_t col0, cudaStream_t st);
ibem_status launch_node24(const SphLaunch& p, const double* nodes, int NN, double* H, int64_t ldh, int64_t row0, int64_t col0, cudaStream_t st);
ibem_status launch_node60(const SphLaunch& p, const double* nodes, int NN, double* H, int64_t ldh, int64_t row0, int64_t col0, cudaStream_t st);
ibem_status launch_node78(const SphLaunch& p, const double* nodes, int NN, double* H, int64_t ldh, int64_t row0, int64_t col0, cudaStream_t st);
// particle part of the stress at points; sbase (nump x 6) holds the boundary or
// remote stress on entry and the total stress on exit
ibem_status launch_field24(const SphLaunch& p, const double* pts, int nump, const double* E, double* stress, cudaStream_t st);
ibem_status launch_field24_df(const SphLaunch& p, const double* pts, int nump, const double* E, double* stress,
                              cudaStream_t st);
ibem_status launch_field60(const SphLaunch& p, const double* pts, int nump, const double* E, double* stress, cudaStream_t st);
ibem_status launch_field78(const SphLaunch& p, const double* pts, int nump, const double* E, double* stress, cudaStream_t st);

// ---- boundary kernels (bem.cu) ----
ibem_status bem_hg(const double* nodes, int NN, const int* conn, int NE, const ibem_material& m,
                   double* H, int64_t ldh, int64_t hrow0, int64_t hcol0, double* G, int64_t ldg,
                   int64_t grow0, int64_t gcol0, cudaStream_t st);
ibem_status bem_to_incl(const double* nodes, int NN, const int* conn, int NE, const double* cen,
                        int num, const ibem_material& m, int layout, double* H, int64_t ldh,
                        int64_t hcol0, double* G, int64_t ldg, int64_t gcol0, int64_t row0,
                        cudaStream_t st);
ibem_status bem_post(const double* pts, int nump, const double* nodes, int NN, const int* conn,
                     int NE, const ibem_material& m, const double* U, const double* T,
                     double* stress, cudaStream_t st, bool mixed = false);

}  // namespace ibem
