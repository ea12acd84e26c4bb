// Device functions and launchers of libhpgpu that no public entry point reaches by themselves, as C functions on host
// arrays for the tests (device_checks.py compiles and links this against the library).
#include <vector>

#include "hp_ff.cuh"
#include "hp_fp64.cuh"

namespace {

enum What { EXP64, DIV64, RSQRT64, CLIP01, BELOW, EXP_FF512, EXP_FF, RCP_SEED, RSQRT_SEED };

__global__ void k_eval(int what, int n, const double* x, const double* y, double* out, double* lo, const double* etab,
                       const float2* etabf) {
  __shared__ double tab[hp::kExpEntries];
  __shared__ float2 tabf[hp::kExpEntries], tab64[64];
  hp::f64::load_exp64(tab, etab);
  for (int i = threadIdx.x; i < hp::kExpEntries; i += blockDim.x) tabf[i] = etabf[i];
  for (int i = threadIdx.x; i < 64; i += blockDim.x) tab64[i] = etabf[i * (hp::kExpEntries / 64)];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const hp::ffa::f2 xf{(float)x[i], (float)y[i]};
  double v = 0.0, l = 0.0;
  switch (what) {
    case EXP64: v = hp::f64::exp64(x[i], tab); break;
    case DIV64: v = hp::f64::div64(x[i], y[i]); break;
    case RSQRT64: v = hp::f64::rsqrt64(x[i]); break;
    case CLIP01: v = hp::f64::clip01(x[i]); break;
    case BELOW: v = hp::f64::below(x[i], hp::f64::cutoff_of(y[i])) ? 1.0 : 0.0; break;
    case EXP_FF512: {
      const hp::ffa::f2 e = hp::ffa::exp_ff512(xf, tabf);
      v = e.hi, l = e.lo;
      break;
    }
    case EXP_FF: {
      const hp::ffa::f2 e = hp::ffa::exp_ff(xf, tab64);
      v = e.hi, l = e.lo;
      break;
    }
    case RCP_SEED: asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(v) : "d"(x[i])); break;
    case RSQRT_SEED: asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(v) : "d"(x[i])); break;
  }
  out[i] = v;
  lo[i] = l;
}

}  // namespace

extern "C" {

int dc_solve_capacity() { return hp::mbis_solve_capacity(); }

// out + lo = f(x, y) for n values, by the device function `what`.
int dc_eval(int what, int n, const double* x, const double* y, double* out, double* lo) {
  std::vector<double> d(hp::kExpEntries);
  std::vector<float2> f(hp::kExpEntries);
  hp::fill_exp_tables(d.data(), f.data());
  double* buf = nullptr;
  const size_t v = 8 * (size_t)n, t = 8 * (size_t)hp::kExpEntries;
  if (cudaMalloc(&buf, 4 * v + 2 * t) != cudaSuccess) return 1;
  double *dx = buf, *dy = dx + n, *dout = dy + n, *dlo = dout + n, *dtab = dlo + n;
  cudaMemcpy(dx, x, v, cudaMemcpyHostToDevice);
  cudaMemcpy(dy, y, v, cudaMemcpyHostToDevice);
  cudaMemcpy(dtab, d.data(), t, cudaMemcpyHostToDevice);
  cudaMemcpy(dtab + hp::kExpEntries, f.data(), t, cudaMemcpyHostToDevice);
  k_eval<<<(n + 255) / 256, 256>>>(what, n, dx, dy, dout, dlo, dtab,
                                   reinterpret_cast<const float2*>(dtab + hp::kExpEntries));
  cudaMemcpy(out, dout, v, cudaMemcpyDeviceToHost);
  cudaMemcpy(lo, dlo, v, cudaMemcpyDeviceToHost);
  cudaFree(buf);
  return cudaGetLastError() != cudaSuccess;
}

// Another stream of the process in capture, one that waits for the legacy stream.
static cudaStream_t capturing = nullptr;
int dc_capture_begin() {
  if (cudaStreamCreate(&capturing) != cudaSuccess) return 1;
  return cudaStreamBeginCapture(capturing, cudaStreamCaptureModeRelaxed) != cudaSuccess;
}
int dc_capture_end() {
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(capturing, &g);
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(capturing);
  cudaGetLastError();
  return e != cudaSuccess;
}

}  // extern "C"
