// FP64 building blocks of the per-point loops.
//
// GB300 issues FP64 at 2 lanes per clock and SM (1/64 of the FP32 rate), so
// a warp-wide FP64 instruction of any kind (FMA, add, compare, conversion)
// holds the pipe for 16 clocks and the FP64 kernels cost their instruction
// count; integer, FP32, shared-memory and HBM work beside it is nearly free
// (a stored FP64 value costs 1.2 ps of copy bandwidth, one FP64 instruction
// 1.6 ps). Hence: table lookups for polynomial terms, stored distances and
// pro-atoms instead of their recomputation, and sums that cross warps in
// shared memory before they cross lanes.
#pragma once

#include "hp_internal.cuh"

namespace hp {
namespace f64 {

// exp(x) by Tang's table-driven method (ACM TOMS 15(2), 1989): x = n ln2/512
// + f, |f| <= ln2/1024; exp(x) = 2^(n >> 9) T[n & 511] (1 + (e^f - 1)) with
// T[j] = 2^(j/512) and e^f - 1 by its Taylor polynomial of degree 4
// (truncation below 2e-18). Nine FP64 instructions; T[j] and the last
// operation are rounded, everything else is e^f - 1 <= 6.8e-4 times smaller:
// error below 1.02 ulp (largest of ten million: 1.008). tab: the table in
// shared memory (random 8-byte reads, which the FP64 pipe hides). |x| >= 708,
// infinities and NaN go to exp.
constexpr int kExpTab = 512;

static __device__ __noinline__ double exp_rare(double x) { return exp(x); }

__device__ __forceinline__ double exp64(double x, const double* tab) {
  const unsigned hx = (unsigned)__double2hiint(x);
  if ((hx & 0x7fffffffu) >= 0x40862000u) {  // |x| >= 708
    if (hx >= 0xc0875000u && hx < 0xfff00000u) return 0.0;  // x <= -746: below the subnormals
    return exp_rare(x);
  }
  const double kL = 0x1.71547652b82fep+9;                            // 512 / ln2
  const double kC1 = 0x1.62e42fefa39efp-10, kC2 = 0x1.abc9e3b39803fp-65;  // ln2 / 512
  const double kMagic = 6755399441055744.0;  // 1.5 * 2^52: round to nearest integer
  const double t = __fma_rn(x, kL, kMagic);
  const int n = __double2loint(t);
  const double nd = t - kMagic;
  double f = __fma_rn(nd, -kC1, x);
  f = __fma_rn(nd, -kC2, f);
  const double T = tab[n & (kExpTab - 1)];
  const double ts = __hiloint2double(__double2hiint(T) + ((n >> 9) << 20), __double2loint(T));
  double q = __fma_rn(f, 1.0 / 24.0, 1.0 / 6.0);
  q = __fma_rn(q, f, 0.5);
  q = __fma_rn(q, f * f, f);
  return __fma_rn(ts, q, ts);
}

// Block-local copy of the table; the caller synchronises before its use.
__device__ __forceinline__ void load_exp64(double* tab, const double* src) {
  for (int i = threadIdx.x; i < kExpTab; i += blockDim.x) tab[i] = src[i];
}

// a / d as a times the reciprocal: 1 / d = y / (1 - e) = y (1 + e + e^2 + ...)
// with e = 1 - d y, the geometric series cut after e^2 (the cubically
// convergent iteration of Altman, Pacific J. Math. 10, 1107 (1960), once). y:
// the hardware's approximation, |e| <= 1.0e-6 (every pattern of the upper 20
// mantissa bits, the rest zeros or ones), so that e^3 is 0.01 ulp. Five FP64
// instructions against the eight or more of a correctly rounded quotient; the
// reciprocal and the product are each rounded once, and half an ulp of the
// one is up to a whole ulp of the other: below 1.52 ulp (largest of ten
// million: 1.49). Divisors outside 2^-959 <= d < 2^961 (and zero, negative,
// infinite or NaN ones) are divided plainly.
// A residual correction (0.506 ulp) was measured: the 22-atom MBIS chain 1.4 %
// and the aLISA chain 2.8 % slower, with the same errors of the results
// against 64 bits (the quotient's rounding averages out over the points).
__device__ __forceinline__ double div64(double a, double d) {
  if ((unsigned)(__double2hiint(d) - 0x04000000) >= 0x78000000u) return a / d;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = __fma_rn(-d, y, 1.0);
  y = __fma_rn(y, __fma_rn(e, e, e), y);
  return a * y;
}

// 1 / sqrt(d) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2/8 + ...) with e = 1 - d y^2,
// the binomial series cut after e^2. y: the hardware's approximation, |e| <=
// 1.9e-6 (as above), so that 5 e^3/16 is 0.02 ulp; the rounding of d y is half
// of an ulp in e and a quarter to a half in the result, the last operation
// another half: below 1.03 ulp (largest of ten million: 0.993). d outside
// 2^-959 <= d < 2^961 by sqrt and a division. For the pivots of the FP64
// Cholesky factor, where each is a link of a serial chain.
__device__ __forceinline__ double rsqrt64(double d) {
  if ((unsigned)(__double2hiint(d) - 0x04000000) >= 0x78000000u) return 1.0 / sqrt(d);
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = __fma_rn(-d * y, y, 1.0);
  return __fma_rn(y * e, __fma_rn(0.375, e, 0.5), y);
}

// Distance from grid point p to atom a, in one fixed sequence of roundings:
// the stored value (JobDev::rd) and a recomputed one are the same bits.
__device__ __forceinline__ double dist64(const JobDev& J, int p, int a) {
  const double dx = J.px[p] - J.ax[a], dy = J.py[p] - J.ay[a], dz = J.pz[p] - J.az[a];
  return sqrt(__fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx)));
}

__device__ __forceinline__ double dist_of(const JobDev& J, const double* rd, int p, int a) {
  return rd ? rd[p] : dist64(J, p, a);
}

// Amplitude N S^3 / (8 pi) of an MBIS shell.
__device__ __forceinline__ double mbis_amp(double n, double s) { return n * (s * s * s) * kInv8PiD; }

// New (N, S) of an MBIS shell from the moments of its bare exponential: N = A
// m0, S = 3 m0 / m1 (mbis.py:150-156). The amplitude cancels in S, but a shell
// without one has S = 0 / 0 there, and the same here.
__device__ __forceinline__ void mbis_shell(double amp, double m0, double m1, double& n, double& s) {
  n = amp * m0;
  const bool none = (__double_as_longlong(amp) << 1) == 0;  // +-0, by integers
  s = none ? __longlong_as_double(0x7ff8000000000000ll) : 3.0 * m0 / m1;
}

// Pro-atom of n MBIS shells at distance r from amplitudes and exponents.
__device__ __forceinline__ double mbis_pro(const double* amp, const double* s, int stride, int n,
                                           double r, const double* tab) {
  double y = 0.0;
  for (int k = 0; k < n; ++k) y = __fma_rn(amp[k * stride], exp64(-s[k * stride] * r, tab), y);
  return y;
}

// The bound sum |N_k| S_k^3 / (8 pi) exp(-S_k r) of an MBIS pro-atom
// (N_k >= 0) at distance r >= 0, for the new and (po non-null) the old parameters together:
// one warp, a shell a lane. tab as exp64.
__device__ __forceinline__ double mbis_bound_warp(const double* pn, const double* po, int nsh,
                                                  double r, const double* tab) {
  const int lane = threadIdx.x & 31;
  const double* q = lane < 16 ? pn : po;
  const int k = lane & 15;
  double b = 0.0;
  if (k < nsh && q) b = mbis_amp(fabs(q[2 * k]), q[2 * k + 1]) * exp64(-q[2 * k + 1] * r, tab);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  return b;
}

// The bound sum_k |a_k - b_k| g_k(r) of a basis scheme (shells s0 .. s0 + nsh
// - 1, which decrease with r): one warp, a shell a lane.
__device__ __forceinline__ double basis_bound_warp(const JobDev& J, int s0, int nsh, const double* a,
                                                   const double* b, double r, const double* tab) {
  const int k = threadIdx.x & 31;
  double s = 0.0;
  if (k < nsh) {
    const double order = J.sh_order[s0 + k];
    const double rn = order == 2.0 ? r * r : order == 1.0 ? r : pow(r, order);
    s = fabs(a[k] - b[k]) * J.sh_pref[s0 + k] * exp64(-J.sh_alpha[s0 + k] * rn, tab);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// fmin(fmax(x, 0), 1) by integer comparisons (NaN gives 0, as fmax does).
__device__ __forceinline__ double clip01(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned)hi < 0x3ff00000u) return x;
  if (hi < 0) return 0.0;
  const long long b = __double_as_longlong(x);
  return b > 0x7ff0000000000000ll ? 0.0 : 1.0;
}

// x < cut by integer comparisons where cut > 0 (the FP64 pipe bounds the
// kernels that test each point): the bits of a positive x below those of cut,
// or the sign bit without a NaN. NaN is not below, as in the comparison.
struct Cutoff {
  double cut;
  unsigned long long bits;
  bool pos;
};
__device__ __forceinline__ Cutoff cutoff_of(double cut) {
  return {cut, (unsigned long long)__double_as_longlong(cut), cut > 0.0};
}
__device__ __forceinline__ bool below(double x, const Cutoff& c) {
  if (!c.pos) return x < c.cut;
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return u < c.bits || (u ^ 0x8000000000000000ull) <= 0x7ff0000000000000ull;
}

// Block sums of nq <= Q per-thread values: the warps' values of a lane are
// added first (from shared memory, warp q for quantity q), then the lanes,
// which takes 12 warp-wide additions a quantity instead of 48. put(q, sum)
// is called by lane 0 of a warp. red: Q * kThreads doubles. nw: warps that
// have values (the others' are left out).
template <int Q, typename Put>
__device__ __forceinline__ void block_sums(const double (&acc)[Q], int nq, double* red, Put put,
                                           int nw = kWarps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < nw) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (q < nq) red[q * kThreads + threadIdx.x] = acc[q];
  }
  __syncthreads();
  for (int q = warp; q < nq; q += kWarps) {
    double v = red[q * kThreads + lane];
#pragma unroll
    for (int w = 1; w < kWarps; ++w)
      if (w < nw) v += red[q * kThreads + 32 * w + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) put(q, v);
  }
}

}  // namespace f64

// One tile of the entropy integral sum w rho ln(rho / promol)
// (core/stockholder.py:145-151) into jpart, for jobs whose at_weights are not
// formed by k_atweights (atom grids, a stored G). red: kThreads doubles.
__device__ __forceinline__ void entropy_tile(const JobDev& J, int tile, double* red) {
  if (!J.local && !J.gmat) return;
  double acc[1] = {0.0};
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
    const double promol = J.promol[p], rho = J.rho[p];
    if (!((promol < J.density_cutoff) || (rho < J.density_cutoff)))
      acc[0] += J.w[p] * rho * log(rho / promol);
  }
  f64::block_sums<1>(acc, 1, red, [&](int, double v) {
    J.jpart[(size_t)QJ_ENTROPY * J.ntile + tile] = v;
  });
}

}  // namespace hp
