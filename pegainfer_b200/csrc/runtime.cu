// Per-thread runtime state: device binding, scratch, launch counter.
// Replaces csrc/linear.cu:7-42 of the reference (thread-local cuBLAS handles + workspace):
// same entry points, same "once per rank thread" contract, no cuBLAS.
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace pk {
ThreadState& tls() {
  static thread_local ThreadState s;
  return s;
}
int sm_count() {
  ThreadState& ts = tls();
  if (ts.sm_count == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&ts.sm_count, cudaDevAttrMultiProcessorCount, dev);
    ts.device = dev;
    if (ts.sm_count <= 0) ts.sm_count = 148;
  }
  return ts.sm_count;
}
static std::atomic<unsigned int*> g_wait_err{nullptr};
unsigned int* wait_err_word() { return g_wait_err.load(std::memory_order_acquire); }
static void make_wait_err_word() {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (wait_err_word()) return;
  void* p = nullptr;
  if (cudaHostAlloc(&p, 64, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  memset(p, 0, 64);
  g_wait_err.store(static_cast<unsigned int*>(p), std::memory_order_release);
}
// waits for a barrier that nothing completes, `spins` tries long
__global__ void wait_probe_kernel(uint32_t spins, unsigned int* err) {
  __shared__ uint64_t bar;
  __shared__ int flag;
  if (threadIdx.x != 0) return;
  flag = 0;
  mbar_init(&bar, 1);
  mbar_fence_init();
  mbar_wait_bounded(&bar, 0, &flag, spins);
  count_run_out(&flag, err);
}
}  // namespace pk

extern "C" {

int cuda_set_device(int device_ordinal) {
  pk::ThreadState& ts = pk::tls();
  ts.sm_count = 0;
  return static_cast<int>(cudaSetDevice(device_ordinal));
}

// Scratch for the internally split non-partition decode attention and the two-stage top-1.
static const size_t kScratchBytes = 16u << 20;

void cublas_init() {
  pk::ThreadState& ts = pk::tls();
  if (ts.scratch == nullptr) {
    if (cudaMalloc(&ts.scratch, kScratchBytes) == cudaSuccess) {
      ts.scratch_bytes = kScratchBytes;
      cudaMemset(ts.scratch, 0, kScratchBytes);
    } else {
      ts.scratch = nullptr;
      ts.scratch_bytes = 0;
    }
  }
  pk::make_wait_err_word();
  (void)pk::sm_count();
}

void cublas_destroy() {
  pk::ThreadState& ts = pk::tls();
  if (ts.scratch != nullptr) {
    cudaFree(ts.scratch);
    ts.scratch = nullptr;
    ts.scratch_bytes = 0;
  }
}

const char* pk_b200_version(void) {
  return "pegainfer-kernels-b200 0.1 (sm_100a; TMA-bulk GEMV, tcgen05 GEMM, no cuBLAS/FlashInfer)";
}

int64_t pk_b200_launch_count(int reset) {
  pk::ThreadState& ts = pk::tls();
  int64_t v = ts.launches;
  if (reset) ts.launches = 0;
  return v;
}

int pk_b200_wait_errors(void) {
  if (pk::wait_err_word() == nullptr || cudaDeviceSynchronize() != cudaSuccess) return -1;
  return (int)pk_b200_wait_errors_seen();
}

unsigned int pk_b200_wait_errors_seen(void) {
  const volatile unsigned int* w = pk::wait_err_word();
  return w ? *w : 0u;
}

int pk_b200_wait_probe(int spins, pk_stream stream) {
  if (spins <= 0 || spins > 1024 || pk::wait_err_word() == nullptr) return -1;
  return (int)pk::launch(pk::wait_probe_kernel, dim3(1), dim3(32), 0, stream, false, (uint32_t)spins, pk::wait_err_word());
}

void pk_b200_set_pdl(int enable) { pk::tls().pdl = enable != 0; }

}  // extern "C"
