// The host code that builds a domain's [line][k] twiddle tables
// (csrc/launch_pass.cuh) on a CUDA runtime that the tests fake: device memory
// is host memory, allocations can be refused, a copy from pageable memory is
// only under way when it returns, and another stream is being captured: a call
// that the capture's mode forbids breaks it.
//   model limit   an allocation above `limit` bytes is refused
// Prints one line for what went wrong; exit status 0 if nothing did.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

static size_t g_limit = 0;
static int g_pending = 0;  // copies under way

static int g_broken = 0;   // calls that broke the capture
static cudaStreamCaptureMode g_mode = cudaStreamCaptureModeGlobal;  // of the thread
static int g_stream;       // the one non-blocking stream a call may create

static void unsafe() { g_broken += g_mode != cudaStreamCaptureModeRelaxed; }
static cudaError_t fake_exchange(cudaStreamCaptureMode* m) {
  const cudaStreamCaptureMode was = g_mode;
  g_mode = *m;
  *m = was;
  return cudaSuccess;
}
static cudaError_t fake_malloc(void** p, size_t bytes) {
  unsafe();
  if (bytes > g_limit) return cudaErrorMemoryAllocation;
  *p = std::malloc(bytes);
  return cudaSuccess;
}
static cudaError_t fake_memcpy(void* dst, const void* src, size_t bytes, cudaMemcpyKind) {
  g_broken++;  // on the legacy stream, which the captured one may be ordered with
  std::memcpy(dst, src, bytes);
  g_pending++;
  return cudaSuccess;
}
static cudaError_t fake_create(cudaStream_t* s, unsigned flags) {
  unsafe();
  if (flags != cudaStreamNonBlocking) g_broken++;
  *s = reinterpret_cast<cudaStream_t>(&g_stream);
  return cudaSuccess;
}
static cudaError_t fake_memcpy_async(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t s) {
  unsafe();
  if (s != reinterpret_cast<cudaStream_t>(&g_stream)) g_broken++;
  std::memcpy(dst, src, bytes);
  g_pending++;
  return cudaSuccess;
}
static cudaError_t fake_synchronize(cudaStream_t) {
  unsafe();
  g_pending = 0;
  return cudaSuccess;
}
static cudaError_t fake_destroy(cudaStream_t) { return unsafe(), cudaSuccess; }
#define cudaThreadExchangeStreamCaptureMode fake_exchange
#define cudaMalloc fake_malloc
#define cudaMemcpy fake_memcpy
#define cudaStreamCreateWithFlags fake_create
#define cudaMemcpyAsync fake_memcpy_async
#define cudaStreamSynchronize fake_synchronize
#define cudaStreamDestroy fake_destroy
#include "launch_pass.cuh"

namespace omr {
int fail(int status, const std::string& msg) {
  std::printf("status %d: %s\n", status, msg.c_str());
  return status;
}
}  // namespace omr

using namespace omr;

template <class F>
static int check(bool refused) {
  omr_ntt_domain_s d;
  d.field = F::ID;
  d.log_n = 18;
  d.n = 1ull << 18;
  d.omega = root_of_unity_host<F>(18);
  const typename F::Tw* tab = nullptr;
  const int rc = line_twiddles<F>(&d, false, 6, 1, 4096, true, &tab);
  if (rc != OMR_NTT_OK) return 1;  // (fail has printed it)
  if (g_broken) return std::printf("a capture on another stream was broken\n"), 1;
  if (g_mode != cudaStreamCaptureModeGlobal) return std::printf("the thread's capture mode was changed\n"), 1;
  if (g_pending) return std::printf("the table's copy has not been waited for\n"), 1;
  if ((tab == nullptr) != refused) return std::printf("table %p\n", (const void*)tab), 1;
  if (refused) return d.line_tw.empty() ? 0 : (std::printf("a refused table was kept\n"), 1);
  uint64_t x = 1;  // omega^(4095 k)
  const uint64_t step = hpowmod(d.omega, 4095, F::p64());
  for (int k = 0; k < 64; k++, x = hmulmod(x, step, F::p64()))
    if (tab[4095 * 64 + k].w != F::make_tw(x).w) return std::printf("entry (4095, %d)\n", k), 1;
  return 0;
}

int main(int, char** argv) {
  g_limit = std::strtoull(argv[1], nullptr, 10);
  const bool refused = g_limit < 4096 * 64 * 8;
  return check<BabyBear>(refused) | check<Goldilocks>(refused);
}
