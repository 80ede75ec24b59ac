// Device-side helpers of the GPU tests, compiled by tests/_device.py into a library of their own.
#include <cuda_runtime.h>
#include "mdg_mixed.cuh"

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

// out[k] = one of the sweeps' arithmetic helpers on (a[k], b[k]); the five-wide quotients take
// a[5 k .. 5 k + 4] over b[k].
template <typename T>
__global__ void form_kernel(int form, long long n, const T *a, const T *b, T *out)
{
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  if constexpr (sizeof(T) == 4) {
    out[k] = form == 0 ? mdg::quot(a[k], b[k]) : form == 1 ? mdg::root(a[k]) : mdg::pow_rarefaction(a[k], b[k]);
  } else {
    if (form < 3) {
      out[k] = form == 0 ? mdg::rcp64(a[k]) : form == 1 ? mdg::rsqrt64(a[k]) : mdg::sound_speed(a[k], b[k]);
      return;
    }
    double x[5], q[5];
    for (int v = 0; v < 5; v++) x[v] = a[5 * k + v];
    if (form == 3) mdg::quotients<5>(x, b[k], q);
    else mdg::quotients<5, true>(x, b[k], q);
    for (int v = 0; v < 5; v++) out[5 * k + v] = q[v];
  }
}

// Faces between the states st[k][2][3] = (rho, v, p) in a gamma-law gas: the mixed sweeps' HLLC
// and the plain FP64 one.  out[k] = {accepted, signal speed, FP64's, flux[5], FP64's}.
__global__ void face_kernel(long long n, double gam, const double *st, double *out)
{
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double w[2][7];
  for (int s = 0; s < 2; s++) {
    const double *q = st + 6 * k + 3 * s;
    const double x[7] = {q[0], q[2] / (gam - 1.0), q[1], 0.0, 0.0, q[2], gam};
    for (int v = 0; v < 7; v++) w[s][v] = x[v];
  }
  const mdg::FaceGeom<double> g{1.0, 1.0, 1.0, 1.0, 1.0};
  double f[5] = {0, 0, 0, 0, 0}, f64[5], s64;
  float sig = 0.0f;
  int shock;
  const bool ok = mdg::riemann_hllc_mixed<0>(w[0], w[1], g, mdg::gam_const<float>((float)gam), f, sig, shock);
  mdg::riemann_hllc<0, false, double>(w[0], w[1], g, mdg::gam_const(gam), f64, s64);
  double *o = out + 13 * k;
  o[0] = ok;
  o[1] = sig;
  o[2] = s64;
  for (int v = 0; v < 5; v++) { o[3 + v] = f[v]; o[8 + v] = f64[v]; }
}
extern "C" int faces(long long n, double gam, const double *st, double *out)
{
  double *d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * n * 19) != cudaSuccess) return 1;
  bool ok = cudaMemcpy(d, st, sizeof(double) * n * 6, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) face_kernel<<<(unsigned)((n + 127) / 128), 128>>>(n, gam, d, d + 6 * n);
  ok = ok && cudaMemcpy(out, d + 6 * n, sizeof(double) * n * 13, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? 0 : 1;
}

// Host arrays in and out; 0 on success.
template <typename T>
static int run_form(int form, long long n, const T *a, const T *b, T *out)
{
  const size_t wide = (sizeof(T) == 8 && form >= 3) ? 5 : 1;
  T *d = nullptr;
  if (cudaMalloc(&d, sizeof(T) * n * (2 * wide + 1)) != cudaSuccess) return 1;
  T *db = d + wide * n, *dout = db + n;
  bool ok = cudaMemcpy(d, a, sizeof(T) * wide * n, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(db, b, sizeof(T) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) form_kernel<T><<<(unsigned)((n + 255) / 256), 256>>>(form, n, d, db, dout);
  ok = ok && cudaMemcpy(out, dout, sizeof(T) * wide * n, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d);
  return ok ? 0 : 1;
}
extern "C" int form_f32(int form, long long n, const float *a, const float *b, float *out)
{
  return run_form(form, n, a, b, out);
}
extern "C" int form_f64(int form, long long n, const double *a, const double *b, double *out)
{
  return run_form(form, n, a, b, out);
}
