// Device-side helpers of the GPU tests, compiled by tests/_device.py into a library of their own.
#include <cuda_runtime.h>

namespace {

// Holds its place on an SM for `ns` nanoseconds (at most `polls` looks at the clock).
__global__ void hold_kernel(unsigned int *started, unsigned long long ns, long long polls)
{
  extern __shared__ char room[];
  unsigned long long t0, t;
  if (threadIdx.x == 0) {
    room[0] = 0;
    __threadfence_system();
    atomicAdd_system(started, 1u);
  }
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  for (long long k = 0; k < polls; k++) {
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    if (t - t0 >= ns) break;
    __nanosleep(1000);
  }
}

struct Hold {
  cudaStream_t st = nullptr;
  cudaEvent_t done = nullptr;
  unsigned int *started = nullptr;
};

}  // namespace

// Fills `sms` SMs of the current device for `ms` milliseconds with CTAs of `threads` threads and
// `smem` bytes of shared memory each (more than half of an SM's, so that one fits); returns when all have started.
extern "C" void *hold_start(int sms, int threads, int smem, int ms)
{
  Hold *h = new Hold;
  const unsigned long long ns = 1000000ull * (unsigned long long)ms;
  bool ok = cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaEventCreateWithFlags(&h->done, cudaEventDisableTiming) == cudaSuccess &&
            cudaMallocHost(&h->started, sizeof(unsigned int)) == cudaSuccess &&
            cudaFuncSetAttribute(hold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
            // (an SM keeps its shared-memory carve-out while CTAs run on it: the largest, so that
            // what these leave is there for others)
            cudaFuncSetAttribute(hold_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared) == cudaSuccess;
  if (ok) {
    *h->started = 0;
    hold_kernel<<<sms, threads, smem, h->st>>>(h->started, ns, 4ll * ms * 1000);
    ok = cudaGetLastError() == cudaSuccess && cudaEventRecord(h->done, h->st) == cudaSuccess;
  }
  while (ok && cudaEventQuery(h->done) == cudaErrorNotReady &&
         *reinterpret_cast<volatile unsigned int *>(h->started) < (unsigned int)sms) {
  }
  return ok ? h : nullptr;
}

// 1 while the CTAs of hold_start are still running
extern "C" int hold_running(void *p) { return cudaEventQuery(static_cast<Hold *>(p)->done) == cudaErrorNotReady; }

extern "C" void hold_end(void *p)
{
  Hold *h = static_cast<Hold *>(p);
  cudaStreamSynchronize(h->st);
  cudaEventDestroy(h->done);
  cudaStreamDestroy(h->st);
  cudaFreeHost(h->started);
  delete h;
}
