// FP64 kernels of the basis schemes (GISA, aLISA, gLISA) over the stored
// basis matrix G (gmat [nshell][npoint], unit-population shells at the grid
// points; gisa.py:91-106, core/basis.py:161 of the reference). Bound by the
// FP64 pipe (one FMA per value and use) and HBM (8 bytes per value); see
// hp_fp64.cuh.
//
// A tight shell underflows to zero a few bohr from its atom. smask holds,
// per (atom, tile), one bit for each of the atom's shells that is nonzero
// somewhere on the tile; the kernels neither load nor multiply the others,
// which add exact zeros. About half the values go (20- and 30-atom chains,
// exponents 0.05 to 300).
#include <math.h>

#include <type_traits>

#include "hp_inner.cuh"

namespace hp {

namespace {

__device__ __forceinline__ const JobDev& decode_local_bs(const Batch& bt, int& local) {
  const int j = find_job(bt, blockIdx.x);
  local = blockIdx.x - bt.prefix[j];
  return bt.jobs[j];
}

__device__ __forceinline__ const JobDev& decode_at_bs(const Batch& bt, int& atom, int& tile) {
  int local;
  const JobDev& J = decode_local_bs(bt, local);
  atom = local / J.ntile;
  tile = local - atom * J.ntile;
  return J;
}

// The atom's shells from the first to the last active one on the tile
// (exponents are usually sorted, so there is no gap; a zero row between them
// adds zeros).
struct ActiveRange {
  int lo, n;
};

__device__ __forceinline__ ActiveRange active_range(unsigned mask) {
  if (!mask) return {0, 0};
  const int lo = __ffs((int)mask) - 1;
  return {lo, 32 - __clz((int)mask) - lo};
}

// f(integral_constant<int, n>) for 1 <= n <= 16.
template <int N, typename F>
__device__ __forceinline__ void with_rows_from(int n, F f) {
  if constexpr (N < kMaxShells) {
    if (n > N) return with_rows_from<N + 1>(n, f);
  }
  f(std::integral_constant<int, N>());
}
template <typename F>
__device__ __forceinline__ void with_rows(int n, F f) {
  switch (n) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    default: with_rows_from<11>(n, f); break;
  }
}

}  // namespace

// G and smask, one block per point tile, atoms outermost. exp by the table;
// order 2 from the squared distance (no root).
__global__ void __launch_bounds__(kThreads) k_basis64(Batch bt) {
  __shared__ double tab[f64::kExpTab];
  int tile;
  const JobDev& J = decode_local_bs(bt, tile);
  if (!J.gmat) return;
  f64::load_exp64(tab, J.etab);
  __syncthreads();
  const size_t N = J.npoint;
  const int p0 = tile * J.tile_points + threadIdx.x, p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int a = 0; a < J.natom; ++a) {
    const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
    const double ax = J.ax[a], ay = J.ay[a], az = J.az[a];
    unsigned mask = 0;
    for (int p = p0; p < p1; p += kThreads) {
      const double dx = J.px[p] - ax, dy = J.py[p] - ay, dz = J.pz[p] - az;
      const double d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx));
      for (int k = 0; k < nsh; ++k) {
        const int s = s0 + k;
        const double order = J.sh_order[s];
        const double rn = order == 2.0 ? d2 : order == 1.0 ? sqrt(d2) : pow(sqrt(d2), order);
        const double g = J.sh_pref[s] * f64::exp64(-J.sh_alpha[s] * rn, tab);
        J.gmat[s * N + p] = g;
        if (J.gmat32) J.gmat32[s * N + p] = (float)g;
        if (__double_as_longlong(g) != 0) mask |= 1u << k;
      }
    }
    mask = __reduce_or_sync(0xffffffffu, mask);
    if ((threadIdx.x & 31) == 0 && mask) atomicOr(&J.smask[(size_t)a * J.ntile + tile], mask);
  }
}

// Pro-atoms and promolecule (core/stockholder.py:153-175), one thread per
// point; a block's 256 points lie in one tile, so its masks are uniform. The
// rows of an atom go two at a time, their loads together (four or eight: 1.5
// and 4 % more of the GISA job, FP64 work on padding). The reference adds
// 1e-100 per atom: a sum of 1e-80 or more does not change by it, and the
// addition is left out there.
__global__ void __launch_bounds__(kThreads) k_promol_g64(Batch bt) {
  int blk;
  const JobDev& J = decode_local_bs(bt, blk);
  if (!J.gmat) return;
  const int p = blk * kThreads + threadIdx.x;
  if (p >= J.npoint) return;
  const int tile = blk / J.ppt;
  const size_t N = J.npoint;
  const double* __restrict__ G = J.gmat;
  const double* __restrict__ par = J.propars;
  double promol = 0.0;
  for (int a = 0; a < J.natom; ++a) {
    unsigned mask = J.smask[(size_t)a * J.ntile + tile];
    const int s0 = J.shell_off[a];
    const double* __restrict__ g0 = G + s0 * N + p;
    double pro = 0.0;
    while (mask) {
      constexpr int kU = 2;
      int k[kU];
      double c[kU], g[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        k[u] = mask ? __ffs((int)mask) - 1 : k[u > 0 ? u - 1 : 0];
        c[u] = mask ? par[s0 + k[u]] : 0.0;
        mask &= mask - 1;
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) g[u] = g0[k[u] * N];
#pragma unroll
      for (int u = 0; u < kU; ++u) pro = __fma_rn(c[u], g[u], pro);
    }
    J.rhoa[a * N + p] = pro;
    promol += pro;
    if ((unsigned)(__double2hiint(promol) - 0x2f600000) >= 0x50900000u) promol += 1e-100;
  }
  J.promol[p] = promol;
  J.invpro[p] = 1.0 / promol;
}

// GISA moments (gisa.py:257-279): at_weights, population sum w rho_a and
// q-vector sums sum w g_k rho_a of one (atom, tile), from the pro-atoms of
// k_promol_g64 (rhoa is not written back: GISA reads it nowhere else).
__global__ void __launch_bounds__(kThreads, 3) k_gisa_moments64(Batch bt) {
  __shared__ double red[(kMaxShells + 1) * kThreads];
  int a, tile;
  const JobDev& J = decode_at_bs(bt, a, tile);
  if (!J.gmat) return;
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const size_t N = J.npoint;
  ActiveRange act = active_range(J.smask[(size_t)a * J.ntile + tile]);
  if (act.n == 0) act.n = 1;  // the population sum is needed all the same
  const double* __restrict__ pro = J.rhoa + a * N;
  const double* __restrict__ inv = J.invpro;
  const double* __restrict__ rhov = J.rho;
  const double* __restrict__ wv = J.w;
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  double* out = J.apart + (size_t)a * J.qa * J.ntile + tile;
  const int nt = J.ntile;
  if (threadIdx.x < nsh) out[(size_t)(QA_INNER + threadIdx.x) * nt] = 0.0;  // the inactive shells
  __syncthreads();
  with_rows(act.n, [&](auto na) {
    constexpr int NA = decltype(na)::value;
    const double* __restrict__ g = J.gmat + (s0 + act.lo) * N;
    double acc[NA + 1];
#pragma unroll
    for (int j = 0; j <= NA; ++j) acc[j] = 0.0;
    for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
      double gv[NA];
#pragma unroll
      for (int j = 0; j < NA; ++j) gv[j] = g[j * N + p];
      const double wr = wv[p] * (f64::clip01(pro[p] * inv[p]) * rhov[p]);
#pragma unroll
      for (int j = 0; j < NA; ++j) acc[j] = __fma_rn(gv[j], wr, acc[j]);
      acc[NA] += wr;
    }
    f64::block_sums<NA + 1>(acc, NA + 1, red, [&](int q, double v) {
      out[(size_t)(q == NA ? (int)QA_POP : QA_INNER + act.lo + q) * nt] = v;
    });
  });
}

// aLISA self-consistent iteration (alisa.py:193-291), one (atom, tile): the
// moments sum w c_k g_k rho_a / pro and the change sum w (oldpro - pro)^2.
__global__ void __launch_bounds__(kThreads, 3) k_lisa_sc64(Batch bt) {
  constexpr int Q = kMaxShells + 1;
  __shared__ double red[Q * kThreads];
  __shared__ double tab[f64::kExpTab];
  __shared__ double c[kMaxShells];
  __shared__ int skip_s;
  inner_begin();
  int a, tile;
  const JobDev& J = decode_at_bs(bt, a, tile);
  if (!J.gmat || !J.active[a]) return;
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const double* pc = J.cur + s0;
  const double* pp = J.prev + s0;
  const bool first = J.inner_it[a] == 0;
  const size_t N = J.npoint;
  const int nt = J.ntile;
  double* out = J.apart + ((size_t)a * J.qa + QA_INNER) * nt + tile;
  const unsigned mask = J.smask[(size_t)a * nt + tile];
  bool skip = mask == 0;  // the pro-atom is zero on the whole tile
  if (J.tgeo && J.amax[(size_t)a * nt + tile] < (float)J.density_cutoff) {
    // per-atom cutoff (kSkipRel): zero moments, negligible change term
    f64::load_exp64(tab, J.etab);
    __syncthreads();
    if (threadIdx.x < 32) {
      const double b = first ? 0.0 : f64::basis_bound_warp(J, s0, nsh, pc, pp, tile_rmin(J, a, tile), tab);
      skip_s = tile_weight(J, tile) * b * b < kSkipRel * J.inner_threshold * J.inner_threshold;
    }
    __syncthreads();
    if (skip_s) {
      skip = true;
      if (threadIdx.x == 0) count_skipped(J, tile, 1.0);
    }
  }
  if (threadIdx.x < nsh) out[(size_t)threadIdx.x * nt] = 0.0;
  if (skip) {
    if (threadIdx.x == 0) {
      out[(size_t)(Q - 1) * nt] = 0.0;
      if (J.oldok) J.oldok[(size_t)a * nt + tile] = 0;
    }
    if (last_block_of(J, a)) lisa_sc_update(J, a);
    return;
  }
  const ActiveRange act = active_range(mask);
  if (threadIdx.x < act.n) c[threadIdx.x] = pc[act.lo + threadIdx.x];
  __syncthreads();
  const double* __restrict__ ra = J.rhoa + a * N;
  const double* __restrict__ wv = J.w;
  double* old = J.oldpro ? J.oldpro + a * N : nullptr;
  const bool stored = old && J.oldok[(size_t)a * nt + tile] != 0;
  const double cut = J.density_cutoff;
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  with_rows(act.n, [&](auto na) {
    constexpr int NA = decltype(na)::value;
    const double* __restrict__ g = J.gmat + (s0 + act.lo) * N;
    double acc[NA + 1];
#pragma unroll
    for (int j = 0; j <= NA; ++j) acc[j] = 0.0;
    for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
      double gv[NA], pro = 0.0;
#pragma unroll
      for (int j = 0; j < NA; ++j) gv[j] = g[j * N + p];
      const double rho = ra[p], w = wv[p];
      double op = stored && !first ? old[p] : 0.0;
#pragma unroll
      for (int j = 0; j < NA; ++j) pro = __fma_rn(c[j], gv[j], pro);
      const bool sick = (rho < cut) || (pro < cut);
      const double wr = sick ? 0.0 : w * f64::div64(rho, sick ? 1.0 : pro);
#pragma unroll
      for (int j = 0; j < NA; ++j) acc[j] = __fma_rn(gv[j], wr, acc[j]);
      if (old) old[p] = pro;
      if (first) continue;  // no change in the first iteration (the update takes 1e100)
      if (!stored) {
        for (int j = 0; j < NA; ++j) op = __fma_rn(pp[act.lo + j], g[j * N + p], op);
      }
      const double d = op - pro;
      acc[NA] = __fma_rn(w * d, d, acc[NA]);
    }
    f64::block_sums<NA + 1>(acc, NA + 1, red, [&](int q, double v) {
      if (q == NA) out[(size_t)(Q - 1) * nt] = v;
      else out[(size_t)(act.lo + q) * nt] = c[q] * v;
    });
  });
  if (old && threadIdx.x == 0) J.oldok[(size_t)a * nt + tile] = 1;
  if (last_block_of(J, a)) lisa_sc_update(J, a);
}

// Outer change sum w (sum_k (c - c_old)_k g_k)^2 (core/iterstock.py:32-45).
__global__ void __launch_bounds__(kThreads, 3) k_change_g64(Batch bt) {
  __shared__ double red[kThreads];
  __shared__ double tab[f64::kExpTab];
  __shared__ double c[kMaxShells];
  __shared__ int skip_s;
  int a, tile;
  const JobDev& J = decode_at_bs(bt, a, tile);
  if (!J.gmat) return;
  if (glisa_idle(J)) return;
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const double* pn = J.propars + s0;
  const double* po = J.propars_old + s0;
  const size_t N = J.npoint;
  double* out = J.apart + ((size_t)a * J.qa + QA_CHANGE) * J.ntile + tile;
  const unsigned mask = J.smask[(size_t)a * J.ntile + tile];
  bool skip = mask == 0;
  if (J.tgeo) {  // per-atom cutoff: bound of the pair's change term
    f64::load_exp64(tab, J.etab);
    __syncthreads();
    if (threadIdx.x < 32) {
      const double b = f64::basis_bound_warp(J, s0, nsh, pn, po, tile_rmin(J, a, tile), tab);
      skip_s = tile_weight(J, tile) * b * b < kSkipRel * J.threshold * J.threshold;
    }
    __syncthreads();
    if (skip_s) {
      skip = true;
      if (threadIdx.x == 0) count_skipped(J, tile, 2.0);
    }
  }
  if (skip) {
    if (threadIdx.x == 0) *out = 0.0;
    return;
  }
  const ActiveRange act = active_range(mask);
  if (threadIdx.x < act.n) c[threadIdx.x] = pn[act.lo + threadIdx.x] - po[act.lo + threadIdx.x];
  __syncthreads();
  const double* __restrict__ wv = J.w;
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  double acc[1] = {0.0};
  with_rows(act.n, [&](auto na) {
    constexpr int NA = decltype(na)::value;
    const double* __restrict__ g = J.gmat + (s0 + act.lo) * N;
    for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
      double gv[NA], d = 0.0;
#pragma unroll
      for (int j = 0; j < NA; ++j) gv[j] = g[j * N + p];
#pragma unroll
      for (int j = 0; j < NA; ++j) d = __fma_rn(c[j], gv[j], d);
      acc[0] = __fma_rn(wv[p] * d, d, acc[0]);
    }
  });
  f64::block_sums<1>(acc, 1, red, [&](int, double v) { *out = v; });
}

#define HP_LAUNCH_BS(kernel, kind, threads, ...)                                       \
  do {                                                                                 \
    if (hb.blocks[kind] > 0) {                                                         \
      kernel<<<hb.blocks[kind], threads, 0, st>>>(hb.b[kind], ##__VA_ARGS__);          \
      ++g_launch_count;                                                                \
    }                                                                                  \
  } while (0)

void launch_basis64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_basis64, K_POINT, kThreads); }
void launch_promol_g64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_promol_g64, K_POINT1, kThreads); }
void launch_gisa_moments64(const HostBatch& hb, cudaStream_t st) {
  HP_LAUNCH_BS(k_gisa_moments64, K_ATOM_TILE, kThreads);
}
void launch_lisa_sc64(const HostBatch& hb, cudaStream_t st) { launch_inner_kernel(k_lisa_sc64, hb, K_ATOM_TILE, st); }
void launch_change_g64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_change_g64, K_ATOM_TILE, kThreads); }

}  // namespace hp
