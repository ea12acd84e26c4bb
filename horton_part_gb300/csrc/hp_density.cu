// Density of contracted Gaussians on grid points (horton-part's density
// generator, scripts/generate_density.py:119-204: the basis functions on the
// points, then rho = einsum("ab,bp,ap->p", D, phi, phi) at :186-188), in
// FP64 on the GPU.
//
// One block per tile of T consecutive points (T chosen by the host so that
// the tile's basis values fit in shared memory, at most kDensTile; two blocks
// a tile where that leaves SMs idle, each with half of the tile's points and
// all of its significant shells):
//  1. the tile's bounding box; a shell is skipped for the whole tile when
//     a_min d_min^2 > kDensExpCut (a_min its smallest exponent, d_min the
//     distance from its centre to the box), i.e. every primitive is below
//     exp(-kDensExpCut) ~ 1e-26 of its peak there; the significant shells
//     are compacted in shell order (block prefix sum);
//  2. phi[f][p] for the significant functions: a warp takes 32 points and a
//     group of shells with one centre (the distance is formed once), the
//     contracted radial factor sum_k c_k exp(-a_k r^2) without the primitives
//     that are below 2^-70 of the shell's most diffuse one at the point
//     (rcut2), and the shell's Cartesian components
//     (file order), combined into pure functions with the shell's (2l+1) x
//     ncart matrix (constant memory, its zeros skipped);
//  3. rho(p) = sum_a phi_a (D_aa phi_a + 2 sum_{b<a} D_ab phi_b) for every
//     density matrix (total, spin, ...): the block's threads split as
//     (point, a-slice), rows a = slice, slice + S, ... in order, and the
//     slices' sums are added in a fixed tree.
// The arithmetic is FP64 throughout; the cost is the FP64 issue rate of
// phase 3 (n_sig^2 / 2 FMA per point and matrix, near the rate of a cuBLAS
// FP64 product) and of the exponentials (hp_fp64.cuh: 11 instructions a
// primitive; CUDA's exp and a distance per shell took 15 % of the time).
// 604,000 points, 190 functions: 15.0 -> 12.5 ms on a molecule of 6.2e9
// significant FMAs (9.8 ms of them); 1.22 to 1.30 times the FMAs' time on
// others (10.7 to 17.0 ms for 5.2e9 to 8.7e9).
//
// A low-rank factor D = L L^T (n_sig x n_occ products instead) was measured
// at 8.4 ms and not kept: it holds only for matrices formed from orbitals
// here, not for those read from a file with eight digits, and its error
// against 64 bits is 1.7 times the plain form's.
#include <math.h>

#include "hp_fp64.cuh"

namespace hp {

namespace {

constexpr int kDensThreads = 256;
constexpr int kDensThreadsMax = 1024;  // small point sets: more slices per tile
constexpr int kDensTile = 64;
constexpr double kDensExpCut = 60.0;

// (2l+1) x ncart matrices of the pure functions of l = 2, 3 (row-major, rows
// m = 0, +1, -1, ...), set from the host tables.
__constant__ double c_pure2[5 * 6];
__constant__ double c_pure3[7 * 10];

// Cartesian components of one point for angular momentum L in file order
// (s; x y z; xx yy zz xy xz yz; xxx yyy zzz xyy xxy xxz xzz yzz yyz xyz).
template <int L>
__device__ __forceinline__ void cart_values(double x, double y, double z, double* c) {
  if constexpr (L == 0) {
    c[0] = 1.0;
  } else if constexpr (L == 1) {
    c[0] = x;
    c[1] = y;
    c[2] = z;
  } else if constexpr (L == 2) {
    c[0] = x * x;
    c[1] = y * y;
    c[2] = z * z;
    c[3] = x * y;
    c[4] = x * z;
    c[5] = y * z;
  } else {
    c[0] = x * x * x;
    c[1] = y * y * y;
    c[2] = z * z * z;
    c[3] = x * y * y;
    c[4] = x * x * y;
    c[5] = x * x * z;
    c[6] = x * z * z;
    c[7] = y * z * z;
    c[8] = y * y * z;
    c[9] = x * y * z;
  }
}

// The functions of a shell at one point: rad times its components, at
// out[q * T] where `write`.
template <int L>
__device__ __forceinline__ void shell_out(bool pure, double rad, double x, double y, double z,
                                          double* out, int T, bool write) {
  constexpr int NC = (L + 1) * (L + 2) / 2;
  double c[NC];
  cart_values<L>(x, y, z, c);
  if (L < 2 || !pure) {
#pragma unroll
    for (int q = 0; q < NC; ++q)
      if (write) out[(size_t)q * T] = rad * c[q];
  } else if constexpr (L >= 2) {
    const double* tm = L == 2 ? c_pure2 : c_pure3;
    for (int m = 0; m < 2 * L + 1; ++m) {
      double v = 0.0;
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const double t = tm[m * NC + q];
        if (__double_as_longlong(t) << 1) v = __fma_rn(t, c[q], v);  // t != 0
      }
      if (write) out[(size_t)m * T] = rad * v;
    }
  }
}

// Basis values of one shell at one point (phase 2): x, y, z from its centre,
// r2 their squared length; zeros for a lane without a point (live false).
// All lanes of the warp, one shell. Not inlined: one copy of the exponential
// and of the components instead of one per call site keeps the kernel in the
// instruction cache (13.6 -> 12.5 ms on the 604,000 points above; on 4,500 points, where
// every line is fetched once, phase 2 takes 13 instead of 26 thousand cycles).
static __device__ __noinline__ void shell_values(const DensityArgs& a, int s, double x, double y, double z,
                                             double r2, float r2f, double* out, int T, const double* tab,
                                             bool live, bool write) {
  const int l = a.info[5 * s];
  const bool pure = a.info[5 * s + 1] != 0;
  const int nprim = a.info[5 * s + 2], k0 = a.info[5 * s + 3];
  double rad = 0.0;
  for (int k = 0; k < nprim; ++k) {
    const bool in = live && !(r2f > a.rcut2[k0 + k]);
    if (!__any_sync(0xffffffffu, in)) continue;
    const double v = __fma_rn(a.coefs[k0 + k], f64::exp64(-a.exps[k0 + k] * r2, tab), rad);
    if (in) rad = v;
  }
  switch (l) {
    case 0: shell_out<0>(false, rad, x, y, z, out, T, write); break;
    case 1: shell_out<1>(false, rad, x, y, z, out, T, write); break;
    case 2: shell_out<2>(pure, rad, x, y, z, out, T, write); break;
    default: shell_out<3>(pure, rad, x, y, z, out, T, write); break;
  }
}

// Shared memory: phi [nbasis][T] doubles, the slice sums (blockDim doubles),
// the exponential's table, then the significant functions' basis indices
// (nbasis ints) and every shell's first local function (nshell ints, -1: not
// significant).
__global__ void __launch_bounds__(kDensThreadsMax) k_density(DensityArgs a) {
  extern __shared__ double dsm[];
  __shared__ double box[6];
  __shared__ double pt[3 * kDensTile];  // the tile's points
  __shared__ int wcnt[kDensThreadsMax / 32], wfun[kDensThreadsMax / 32];
  // the block's points: one of the nsub parts of a tile
  const int T = a.tile / a.nsub;
  const int64_t q0 = (int64_t)(blockIdx.x / a.nsub) * a.tile;
  const int part = blockIdx.x % a.nsub;
  const int nq = (int)min((int64_t)a.tile, a.npoint - q0);
  const int64_t p0 = q0 + (int64_t)part * T;
  const int np = min(T, nq - part * T);
  if (np <= 0) return;
  const int NT = blockDim.x, NW = NT >> 5;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* phi = dsm;
  double* slice = phi + (size_t)a.nbasis * T;
  double* tab = slice + NT;
  int* fidx = reinterpret_cast<int*>(tab + f64::kExpTab);
  int* loc = fidx + a.nbasis;
  for (int i = threadIdx.x; i < 3 * nq; i += NT) pt[i] = a.points[q0 * 3 + i];
  f64::load_exp64(tab, a.etab);
  __syncthreads();
  // 1. bounding box of the tile (a warp per coordinate) and the significant
  // shells (in shell order)
  if (warp < 3) {
    double vmin = INFINITY, vmax = -INFINITY;
    for (int i = lane; i < nq; i += 32) {
      const double v = pt[3 * i + warp];
      vmin = fmin(vmin, v);
      vmax = fmax(vmax, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vmin = fmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
      vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if (lane == 0) {
      box[2 * warp] = vmin;
      box[2 * warp + 1] = vmax;
    }
  }
  __syncthreads();
  int ns = 0, nf = 0;
  for (int base = 0; base < a.nshell; base += NT) {
    const int s = base + threadIdx.x;
    bool sig = false;
    int nfs = 0;
    if (s < a.nshell) {
      double d2 = 0.0;
      for (int k = 0; k < 3; ++k) {
        const double c = a.centers[3 * s + k], lo = box[2 * k], hi = box[2 * k + 1];
        const double d = c < lo ? lo - c : (c > hi ? c - hi : 0.0);
        d2 += d * d;
      }
      sig = a.amin[s] * d2 <= kDensExpCut;
      const int l = a.info[5 * s], pure = a.info[5 * s + 1];
      nfs = sig ? (pure ? 2 * l + 1 : (l + 1) * (l + 2) / 2) : 0;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, sig);
    int fpre = nfs;  // inclusive prefix of the function counts within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, fpre, o);
      if (lane >= o) fpre += u;
    }
    if (lane == 31) {
      wcnt[warp] = __popc(bal);
      wfun[warp] = fpre;
    }
    __syncthreads();
    int fo = nf, st = ns, ft = nf;
    const int nw = min(NW, (a.nshell - base + 31) / 32);  // the warps with a shell
    for (int w = 0; w < nw; ++w) {
      if (w < warp) fo += wfun[w];
      st += wcnt[w];
      ft += wfun[w];
    }
    if (s < a.nshell) {
      const int f = fo + fpre - nfs;
      loc[s] = sig ? f : -1;
      const int f0 = a.info[5 * s + 4];
      for (int q = 0; q < nfs; ++q) fidx[f + q] = f0 + q;
    }
    __syncthreads();
    ns = st;
    nf = ft;
  }
  if (a.stats && threadIdx.x == 0 && part == 0) {
    const unsigned long long nn = (unsigned long long)nq;
    atomicAdd(&a.stats[0], (unsigned long long)ns);
    atomicAdd(&a.stats[1], (unsigned long long)nf * nn);
    atomicAdd(&a.stats[2], (unsigned long long)nf * (unsigned long long)(nf + 1) / 2ull * nn);
  }
  // 2. basis values of the significant shells (zero past the last point): a
  // warp per (group of shells with one centre, 32 points; fewer for a tile
  // of 8 or 16); per shell where the groups leave most warps idle
  const int npw = min(T, 32), nchunk = T / npw;
  const bool single = 2 * a.ngroup * nchunk <= NW;
  for (int e = warp; e < (single ? a.nshell : a.ngroup) * nchunk; e += NW) {
    const int g = e / nchunk, i = (e - g * nchunk) * npw + (lane & (npw - 1));
    const int sa = single ? g : a.groups[g], sb = single ? g + 1 : a.groups[g + 1];
    const double* pp = pt + 3 * (part * T + min(i, np - 1));
    const double x = pp[0] - a.centers[3 * sa];
    const double y = pp[1] - a.centers[3 * sa + 1];
    const double z = pp[2] - a.centers[3 * sa + 2];
    const double r2 = x * x + y * y + z * z;
    const float r2f = (float)r2;
    for (int s = sa; s < sb; ++s)
      if (loc[s] >= 0)
        shell_values(a, s, x, y, z, r2, r2f, phi + (size_t)loc[s] * T + i, T, tab, i < np, lane < npw);
  }
  __syncthreads();
  // 3. rho for every matrix: thread (point i, slice q)
  const int S = NT / T;  // T divides NT
  const int i = threadIdx.x % T, q = threadIdx.x / T;
  for (int mat = 0; mat < a.nmat; ++mat) {
    double acc = 0.0;
    const double* D = a.mats + (size_t)mat * a.nbasis * a.nbasis;
    for (int ra = q; ra < nf; ra += S) {
      const double* Drow = D + (size_t)fidx[ra] * a.nbasis;
      const double pa = phi[(size_t)ra * T + i];
      double y = 0.0;
      for (int rb = 0; rb < ra; ++rb) y += Drow[fidx[rb]] * phi[(size_t)rb * T + i];
      acc += pa * (Drow[fidx[ra]] * pa + 2.0 * y);
    }
    slice[threadIdx.x] = acc;
    __syncthreads();
    for (int h = S / 2; h > 0; h /= 2) {  // (S is a power of two)
      if (q < h) slice[threadIdx.x] += slice[threadIdx.x + h * T];
      __syncthreads();
    }
    if (q == 0 && i < np) a.out[(size_t)mat * a.npoint + p0 + i] = slice[i];
    __syncthreads();
  }
}

}  // namespace

size_t density_smem_bytes(int nbasis, int nshell, int tile, int threads) {
  return ((size_t)nbasis * tile + threads + f64::kExpTab) * sizeof(double) +
         sizeof(int) * ((size_t)nbasis + (size_t)nshell);
}

int density_tile(int nbasis, int nshell) {
  for (int t = kDensTile; t >= 8; t /= 2)
    if (density_smem_bytes(nbasis, nshell, t, kDensThreads) <= kDensSmemMax) return t;
  return 0;
}

int set_pure_tables(const double* pure2, const double* pure3) {
  if (cudaMemcpyToSymbol(c_pure2, pure2, sizeof(double) * 5 * 6) != cudaSuccess) return 1;
  if (cudaMemcpyToSymbol(c_pure3, pure3, sizeof(double) * 7 * 10) != cudaSuccess) return 1;
  return 0;
}

void launch_density(const DensityArgs& a, cudaStream_t st) {
  static int configured = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured != dev) {
    cudaFuncSetAttribute(k_density, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kDensSmemMax + 8 * kDensThreadsMax));
    configured = dev;
  }
  const int64_t nblk = (a.npoint + a.tile - 1) / a.tile;
  if (nblk <= 0) return;
  DensityArgs b = a;
  b.nsub = 2 * nblk <= 152 && a.tile == 64 ? 2 : 1;
  // fewer tiles than SMs: four times the slices, so that a tile's time is not
  // that of eight warps, and half a tile a block while all blocks have an SM
  // (water, 4,500 points: 35.4 -> 29.1 us by the halves, 23.5 with phase 2 out
  // of line)
  const int threads = nblk <= 152 ? kDensThreadsMax : kDensThreads;
  const size_t smem = density_smem_bytes(a.nbasis, a.nshell, a.tile / b.nsub, threads);
  k_density<<<(unsigned)(nblk * b.nsub), threads, smem, st>>>(b);
  ++g_launch_count;
}

}  // namespace hp
