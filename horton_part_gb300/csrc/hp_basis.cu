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

#include <algorithm>
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
    // without a cutoff a zero row takes part: 0 times the quotient rho / 0 of a
    // point where every shell underflows
    if (!(J.density_cutoff > 0.0)) mask = (1u << nsh) - 1u;
    mask = __reduce_or_sync(0xffffffffu, mask);
    if ((threadIdx.x & 31) == 0 && mask) atomicOr(&J.smask[(size_t)a * J.ntile + tile], mask);
  }
}

// Pro-atoms and promolecule (core/stockholder.py:153-175), one thread per
// point; a block's 256 points lie in one tile, so its masks are uniform. An
// atom's active range is loaded at once and adds one FP64 instruction a row
// (two rows at a time from the mask bits: 208 -> 185 us on 20 atoms and 604k
// points, of which 150 us are FP64 issue). The reference adds 1e-100 per
// atom: a sum of 1e-80 or more does not change by it, and the addition is
// left out there.
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
    const ActiveRange act = active_range(J.smask[(size_t)a * J.ntile + tile]);
    if (act.n == 0) {
      J.rhoa[a * N + p] = 0.0;
    } else {
      const int s0 = J.shell_off[a] + act.lo;
      const double* __restrict__ g0 = G + s0 * N + p;
      with_rows(act.n, [&](auto na) {
        constexpr int NA = decltype(na)::value;
        double g[NA], pro = 0.0;
#pragma unroll
        for (int u = 0; u < NA; ++u) g[u] = g0[u * N];
#pragma unroll
        for (int u = 0; u < NA; ++u) pro = __fma_rn(par[s0 + u], g[u], pro);
        J.rhoa[a * N + p] = pro;
        promol += pro;
      });
    }
    if ((unsigned)(__double2hiint(promol) - 0x2f600000) >= 0x50900000u) promol += 1e-100;
  }
  J.promol[p] = promol;
  J.invpro[p] = 1.0 / promol;
}

// GISA moments (gisa.py:257-279): at_weights, population sum w rho_a and
// q-vector sums sum w g_k rho_a of one (atom, tile), from the pro-atoms of
// k_promol_g64 (rhoa is not written back: GISA reads it nowhere else). Three
// blocks an SM; 16 rows spill (168 bytes). 10 atoms, 145,500 points, five
// outer iterations: 2.30 -> 1.04 ms at 6 shells, 4.66 -> 2.32 at 16.
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
// Three blocks an SM; the forms of many active rows spill (552 bytes at 16).
// 10 atoms, 145,500 points, 40 iterations: 20.9 -> 3.7 ms at 6 shells,
// 38.6 -> 6.1 at 16.
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
  const f64::Cutoff cut = f64::cutoff_of(J.density_cutoff);
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
      const bool sick = f64::below(rho, cut) || f64::below(pro, cut);
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

// The tile's active rows with their coefficients in shared memory, for the
// passes that take every row at a point: eight rows' loads go together (with
// the bit masks read per point two were in flight and the pass took 1.5
// times as long). Zero weights pad the list to a multiple of eight.
constexpr int kListRows = 1024;
struct RowList {
  double c[kListRows];
  int row[kListRows];
  int n;
};

__device__ __forceinline__ void load_rows(const JobDev& J, int tile, const double* vec, RowList* L) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int n = 0;
    for (int a0 = 0; a0 < J.natom; a0 += 32) {
      const int a = a0 + lane;
      unsigned m = a < J.natom ? J.smask[(size_t)a * J.ntile + tile] : 0u;
      const int mine = __popc(m);
      int pos = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, pos, o);
        if (lane >= o) pos += x;
      }
      int at = n + pos - mine;
      for (; m; m &= m - 1) L->row[at++] = J.shell_off[a] + __ffs((int)m) - 1;
      n += __shfl_sync(0xffffffffu, pos, 31);
    }
    __syncwarp();
    const int n8 = (n + 7) & ~7;
    for (int i = n + lane; i < n8; i += 32) L->row[i] = n > 0 ? L->row[n - 1] : 0;
    if (lane == 0) L->n = n;
  }
  __syncthreads();
  const int n = L->n;
  for (int i = threadIdx.x; i < ((n + 7) & ~7); i += blockDim.x) L->c[i] = i < n ? vec[L->row[i]] : 0.0;
  __syncthreads();
}

// sum over the rows of the list of c G[row][p], even and odd rows in chains of
// their own.
__device__ __forceinline__ double dot_list(const JobDev& J, const RowList* L, int p) {
  const size_t N = J.npoint;
  const double* __restrict__ G = J.gmat + p;
  double y0 = 0.0, y1 = 0.0;
  for (int i = 0; i < L->n; i += 8) {
    double g[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) g[u] = G[L->row[i + u] * N];
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      y0 = __fma_rn(L->c[i + u], g[u], y0);
      y1 = __fma_rn(L->c[i + u + 1], g[u + 1], y1);
    }
  }
  return y0 + y1;
}

// The same without a list (jobs of more than kListRows shells).
__device__ __forceinline__ double dot_rows(const JobDev& J, int tile, int p, const double* __restrict__ vec) {
  const size_t N = J.npoint;
  double y = 0.0;
  for (int a = 0; a < J.natom; ++a) {
    const int s0 = J.shell_off[a];
    for (unsigned mask = J.smask[(size_t)a * J.ntile + tile]; mask; mask &= mask - 1) {
      const int m = s0 + __ffs((int)mask) - 1;
      y = __fma_rn(vec[m], J.gmat[m * N + p], y);
    }
  }
  return y;
}

// rho0 = G^T c (glisa.py:346-348); d1 = w rho/rho0, d2 = w rho/rho0^2 (0 where
// sick); entropy and negativity partials (glisa.py:441-450, 784).
__global__ void __launch_bounds__(kThreads) k_glisa_pro(Batch bt) {
  __shared__ double red[2 * kThreads];
  __shared__ RowList rows;
  int tile;
  const JobDev& J = decode_local_bs(bt, tile);
  if (glisa_idle(J)) return;
  const bool list = J.nshell <= kListRows;
  if (list) load_rows(J, tile, J.propars, &rows);
  double acc[2] = {0.0, 0.0};
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
    const double rho0 = list ? dot_list(J, &rows, p) : dot_rows(J, tile, p, J.propars);
    const double rho = J.rho[p];
    const double w = J.w[p];
    const bool sick = (rho < J.density_cutoff) || (rho0 < J.density_cutoff);
    const double inv = sick ? 0.0 : 1.0 / (sick ? 1.0 : rho0);
    const double ratio = rho * inv;
    const double d2 = w * ratio * inv;
    J.dvec1[p] = w * ratio;
    J.dvec2[p] = d2;
    J.rho0[p] = rho0;
    if (J.hess_s) J.hess_s[p] = sqrtf((float)d2);
    if (!sick) acc[0] += w * rho * log(ratio);
    if (rho0 < J.negative_cutoff) acc[1] += 1.0;
  }
  f64::block_sums<2>(acc, 2, red, [&](int q, double v) {
    J.jpart[(size_t)(q == 0 ? QJ_ENTROPY : QJ_NEG) * J.ntile + tile] = v;
  });
}

// gpart[m][tile] = sum_p G[m][p] v[p] with v = d1 (gradient) or v = hvec
// (Hessian-vector product of the refinement); a warp per shell, zero where
// the shell is inactive.
__global__ void __launch_bounds__(kThreads) k_glisa_grad(Batch bt, int use_hvec) {
  int tile;
  const JobDev& J = decode_local_bs(bt, tile);
  if (glisa_idle(J)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p0 = tile * J.tile_points;
  const int p1 = min(p0 + J.tile_points, J.npoint);
  const double* __restrict__ v = use_hvec ? J.hvec : J.dvec1;
  int a = 0, s1 = J.shell_off[1];  // the atom of shell m (m grows)
  for (int m = warp; m < J.nshell; m += kWarps) {
    while (m >= s1) s1 = J.shell_off[++a + 1];
    double s = 0.0;
    if ((J.smask[(size_t)a * J.ntile + tile] >> (m - J.shell_off[a])) & 1u) {
      const double* __restrict__ g = J.gmat + (size_t)m * J.npoint;
#pragma unroll 8
      for (int p = p0 + lane; p < p1; p += 32) s = __fma_rn(g[p], v[p], s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    if (lane == 0) J.gpart[(size_t)m * J.ntile + tile] = s;
  }
}

// Trial objective differences: tpart[t][tile] = this tile's part of
// f(c_t) - f(c), f(c) = sum over healthy points of w rho ln(rho / rho0(c)).
//   rho0_t = sum_m max(c_m + a_t delta_m, 0) g_m
//          = rho0 + a_t (G^T delta) + sum_{m clipped at t} -(c_m + a_t delta_m) g_m,
// one pass over G plus the few clipped shells. Where a point is healthy for
// both, its term is -w rho log1p((rho0_t - rho0) / rho0): the relative change
// is formed in FP64 and goes through the FP32 log1pf, which keeps each term
// (and the difference the Armijo test compares) accurate to ~1e-7 of itself
// without an FP64 log per trial; the few points whose sick status differs
// between rho0 and rho0_t take FP64 logs. Sums in float-float per thread.
__global__ void __launch_bounds__(kThreads) k_glisa_trials(Batch bt) {
  __shared__ double red[2 * kTrials * kThreads];
  __shared__ RowList rows;
  int tile;
  const JobDev& J = decode_local_bs(bt, tile);
  if (glisa_idle(J)) return;
  const bool list = J.nshell <= kListRows;
  if (list) load_rows(J, tile, J.delta, &rows);
  float ah[kTrials], al[kTrials], an[kTrials];
#pragma unroll
  for (int t = 0; t < kTrials; ++t) ah[t] = al[t] = an[t] = 0.0f;
  const int nclip = J.clip[J.nshell];
  const double cut = J.density_cutoff;
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
    const double u = list ? dot_list(J, &rows, p) : dot_rows(J, tile, p, J.delta);
    // corr_t = -sum_{m clipped at t} (c_m + 2^-t delta_m) g_m: the clipped
    // sets shrink as t grows, so walk the list (sorted by t_m, largest first)
    // once, keeping the running sums of c g and delta g
    double corr[kTrials];
    {
      double sc = 0.0, sd = 0.0;
      int k = 0;
#pragma unroll
      for (int t = kTrials - 1; t >= 0; --t) {
        for (; k < nclip && J.clip[J.nshell + 1 + k] > t; ++k) {
          const int m = J.clip[k];
          const double g = J.gmat[(size_t)m * J.npoint + p];
          sc = __fma_rn(J.propars[m], g, sc);
          sd = __fma_rn(J.delta[m], g, sd);
        }
        corr[t] = -__fma_rn(ldexp(1.0, -t), sd, sc);
      }
    }
    const double rho = J.rho[p], w = J.w[p], r0 = J.rho0[p];
    const bool rs = rho < cut;
    const bool h0 = !(rs || r0 < cut);
    const double inv = h0 ? 1.0 / (h0 ? r0 : 1.0) : 0.0;
    const float wr = (float)(w * rho);
#pragma unroll
    for (int t = 0; t < kTrials; ++t) {
      const double dr = __fma_rn(ldexp(1.0, -t), u, corr[t]);
      const double rt = r0 + dr;
      const bool ht = !(rs || rt < cut);
      float term = 0.0f;
      if (h0 && ht) {
        term = -wr * log1pf((float)(dr * inv));
        an[t] += fabsf(term);
      } else if (h0 || ht) {
        const double big = ht ? w * rho * log(rho / rt) : -(w * rho * log(rho / r0));
        const float bh = (float)big;
        term = bh;
        al[t] += (float)(big - (double)bh);
      }
      const float s = ah[t] + term;  // TwoSum into (ah, al)
      const float bb = s - ah[t];
      al[t] += (ah[t] - (s - bb)) + (term - bb);
      ah[t] = s;
    }
  }
  double acc[2 * kTrials];
#pragma unroll
  for (int t = 0; t < kTrials; ++t) {
    acc[t] = (double)ah[t] + (double)al[t];
    acc[kTrials + t] = (double)an[t];
  }
  f64::block_sums<2 * kTrials>(acc, 2 * kTrials, red,
                               [&](int q, double v) { J.tpart[(size_t)q * J.ntile + tile] = v; });
}

// ---------------------------------------------------------------------------
// gLISA Hessian H_ij = sum_p (w rho / rho0^2)(p) g_i(p) g_j(p) (glisa.py:457-470)
//
// FP64 FMAs on the lower triangle of the rows that are active on the tile:
// sum over tiles of points x nact (nact + 1) / 2, about a third of the full
// triangle (and a seventh of what padded 64 x 64 tiles of all rows issue).
// Bound by the FP64 pipe.
//
// One persistent block per SM and partial (hsched: units of hunit points of
// one tile, longest processing time first, ascending within a block). For a
// tile the active rows are compacted and their triangle is cut into 4 x 4
// register blocks dealt densely to the threads, so that no issue slot goes
// to inactive rows; when they fill less than half of the warps, groups of
// warps take the stage's points in turn (the FP64 pipes are per quarter of
// the SM, so 4 or 6 busy warps leave some idle); consecutive units of a tile keep the accumulators, which
// are added to the block's packed triangle in L2 when the tile changes (a
// few instructions per element against hundreds of points). Points pass
// through shared memory 16 at a time, rows scaled by w rho / rho0^2 beside
// the plain ones, two buffers.
//
// 20-atom molecule (604,000 points, 150 shells): 30.4 -> 5.5 ms; 10 atoms, 66,000
// points, 72 shells: 1520 -> 293 us.
// ---------------------------------------------------------------------------
constexpr int kH64Threads = 512;
constexpr int kH64K = 16;  // points per stage
constexpr int kH64Stage = kH64Rows * kH64K / kH64Threads;  // staged values per thread at most

__device__ __forceinline__ void tri_of(int e, int& i, int& j) {
  i = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
  while (i * (i + 1) / 2 > e) --i;
  while ((i + 1) * (i + 2) / 2 <= e) ++i;
  j = e - i * (i + 1) / 2;
}

__global__ void __launch_bounds__(kH64Threads, 1) k_glisa_hess64(Batch bt, int ld) {
  extern __shared__ double hsm[];  // [2 buffers][plain, scaled][kH64K][ld]
  __shared__ int row[kH64Rows];
  __shared__ int nact_s;
  int local;
  const JobDev& J = decode_local_bs(bt, local);
  if (!J.hsched || glisa_idle(J)) return;
  const int S = J.nshell;
  const size_t N = J.npoint;
  double* H = J.hpart + (size_t)local * (S * (S + 1) / 2);
  for (int e = threadIdx.x; e < S * (S + 1) / 2; e += kH64Threads) H[e] = 0.0;
  const int* units = J.hsched + J.hbuf + 1;
  const int upt = (J.tile_points + J.hunit - 1) / J.hunit;
  const int plane = kH64K * ld;
  double acc[2][16];
  int tile = -1, nact = 0, nb = 0, base = 0;
  int ngrp = 1, grp = 0;  // groups over the stage's points, this thread's one
  int bi[2], bj[2];
  auto flush = [&]() {
    // the groups' sums onto group 0's, group by group through shared memory
    // (the stage buffers are free: sweep ends at a barrier), then one read and
    // write per element, the reads together
    const int width = max(32, (nb + 31) & ~31);
    for (int g = 1; g < ngrp; ++g) {
      const int lane = (int)threadIdx.x - grp * width;
      if (grp == g) {
#pragma unroll
        for (int q = 0; q < 16; ++q) hsm[q * width + lane] = acc[0][q];
      }
      __syncthreads();
      if (grp == 0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) acc[0][q] += hsm[q * width + lane];
      }
      __syncthreads();
    }
    if (grp != 0) return;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (bi[t] < 0) continue;
      double h[16];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int i = 4 * bi[t] + u, j = 4 * bj[t] + v;
          h[4 * u + v] = i < nact && j <= i ? H[row[i] * (row[i] + 1) / 2 + row[j]] : 0.0;
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int i = 4 * bi[t] + u, j = 4 * bj[t] + v;
          if (i < nact && j <= i) H[row[i] * (row[i] + 1) / 2 + row[j]] = h[4 * u + v] + acc[t][4 * u + v];
        }
    }
  };
  auto assign = [&]() {  // this thread's 4 x 4 blocks of the pass that starts at block `base`
    const int width = max(32, (nb + 31) & ~31);
    ngrp = 1;
    while (2 * ngrp * width <= kH64Threads && ngrp < 8) ngrp *= 2;
    grp = ngrp > 1 ? (int)threadIdx.x / width : 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int e = base + t * kH64Threads + (int)threadIdx.x - grp * width;
      bi[t] = bj[t] = -1;
      if (e < nb && grp < ngrp && (ngrp == 1 || t == 0)) tri_of(e, bi[t], bj[t]);
#pragma unroll
      for (int q = 0; q < 16; ++q) acc[t][q] = 0.0;
    }
  };
  // the points [q0, q1) of the current tile into the accumulators
  auto sweep = [&](int q0, int q1) {
    const int rows4 = (nact + 3) & ~3;
    // thread: point sk of the stage, rows sr, sr + 32, ...
    const int sk = threadIdx.x % kH64K, sr = threadIdx.x / kH64K;
    double pre[kH64Stage], prd = 0.0;
    auto fetch = [&](int q) {
      const int p = q + sk;
      prd = p < q1 ? J.dvec2[p] : 0.0;
#pragma unroll
      for (int c = 0; c < kH64Stage; ++c) {
        const int r = sr + c * (kH64Threads / kH64K);
        pre[c] = r < nact && p < q1 ? J.gmat[row[r] * N + p] : 0.0;
      }
    };
    auto store = [&](int b) {
      double* X = hsm + b * 2 * plane + sk * ld;
#pragma unroll
      for (int c = 0; c < kH64Stage; ++c) {
        const int r = sr + c * (kH64Threads / kH64K);
        if (r < rows4) {
          X[r] = pre[c];
          X[plane + r] = pre[c] * prd;
        }
      }
    };
    fetch(q0);
    store(0);
    __syncthreads();
    int b = 0;
    const bool two = nb - base > kH64Threads;
    for (int q = q0; q < q1; q += kH64K) {
      const bool more = q + kH64K < q1;
      if (more) fetch(q + kH64K);
      const double* X = hsm + b * 2 * plane;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (t == 1 && !two) break;
        if (bi[t] < 0) continue;
        const double* xa = X + 4 * bi[t];
        const double* xb = X + plane + 4 * bj[t];
#pragma unroll 2
        for (int k = grp; k < kH64K; k += ngrp) {
          const double2 a0 = *reinterpret_cast<const double2*>(xa + k * ld);
          const double2 a1 = *reinterpret_cast<const double2*>(xa + k * ld + 2);
          const double2 b0 = *reinterpret_cast<const double2*>(xb + k * ld);
          const double2 b1 = *reinterpret_cast<const double2*>(xb + k * ld + 2);
          const double av[4] = {a0.x, a0.y, a1.x, a1.y}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[t][4 * u + v] = __fma_rn(av[u], bv[v], acc[t][4 * u + v]);
        }
      }
      if (more) store(b ^ 1);
      __syncthreads();
      b ^= 1;
    }
  };
  for (int k = J.hsched[local]; k < J.hsched[local + 1]; ++k) {
    const int u = units[k];
    const int t = u / upt;
    if (t != tile) {
      if (tile >= 0 && nb <= 2 * kH64Threads) flush();
      __syncthreads();  // row is read by flush; H by the block's other threads
      tile = t;
      if (threadIdx.x < 32) {  // compact the active rows, atom by atom
        int n = 0;
        for (int a0 = 0; a0 < J.natom; a0 += 32) {
          const int a = a0 + threadIdx.x;
          unsigned m = a < J.natom ? J.smask[(size_t)a * J.ntile + tile] : 0u;
          int pos = __popc(m);
          for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, pos, o);
            if ((int)threadIdx.x >= o) pos += x;
          }
          const int total = __shfl_sync(0xffffffffu, pos, 31);
          int at = n + pos - __popc(m);
          for (; m; m &= m - 1) row[at++] = J.shell_off[a] + __ffs((int)m) - 1;
          n += total;
        }
        if (threadIdx.x == 0) nact_s = n;
      }
      __syncthreads();
      nact = nact_s;
      const int nq = (nact + 3) >> 2;
      nb = nq * (nq + 1) / 2;
      base = 0;
      assign();
    }
    const int q0 = tile * J.tile_points + (u - t * upt) * J.hunit;
    const int q1 = min(min(q0 + J.hunit, (tile + 1) * J.tile_points), J.npoint);
    if (nact == 0 || q0 >= q1) continue;
    if (nb <= 2 * kH64Threads) {
      sweep(q0, q1);
    } else {  // more blocks than the accumulators hold: passes over the unit
      for (base = 0; base < nb; base += 2 * kH64Threads) {
        assign();
        sweep(q0, q1);
        flush();
      }
      base = 0;
      __syncthreads();
    }
  }
  if (tile >= 0 && nb <= 2 * kH64Threads) flush();
}

#define HP_LAUNCH_BS(kernel, kind, threads, ...)                                       \
  do {                                                                                 \
    if (hb.blocks[kind] > 0) {                                                         \
      kernel<<<hb.blocks[kind], threads, 0, st>>>(hb.b[kind], ##__VA_ARGS__);          \
      ++g_launch_count;                                                                \
    }                                                                                  \
  } while (0)

void launch_glisa_pro(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_glisa_pro, K_POINT, kThreads); }
void launch_glisa_grad(const HostBatch& hb, cudaStream_t st, int use_hvec) {
  HP_LAUNCH_BS(k_glisa_grad, K_POINT, kThreads, use_hvec);
}
void launch_glisa_trials64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_glisa_trials, K_POINT, kThreads); }
void launch_basis64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_basis64, K_POINT, kThreads); }
void launch_promol_g64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_promol_g64, K_POINT1, kThreads); }
void launch_gisa_moments64(const HostBatch& hb, cudaStream_t st) {
  HP_LAUNCH_BS(k_gisa_moments64, K_ATOM_TILE, kThreads);
}
void launch_lisa_sc64(const HostBatch& hb, cudaStream_t st) { launch_inner_kernel(k_lisa_sc64, hb, K_ATOM_TILE, st); }
// rows: most shells of a job of the batch that takes the kernel (0: none).
void launch_glisa_hess64(const HostBatch& hb, cudaStream_t st, int rows) {
  if (rows <= 0 || hb.blocks[K_HESS] <= 0) return;
  // an even row stride, 2 mod 4: 16-byte loads, the staging's columns spread
  // over the banks. The groups' sums (flush) take 16 values for each of nb
  // threads rounded up to 32, nb = nq (nq + 1) / 2 with nq = ceil(nact / 4):
  // at most 4 ld of them, from ld = 10 on
  const int ld = std::max(10, ((rows + 3) & ~3) + 2);
  const size_t smem = sizeof(double) * 4 * kH64K * (size_t)ld;
  static int configured = -1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured != dev) {
    cudaFuncSetAttribute(k_glisa_hess64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(double) * 4 * kH64K * (kH64Rows + 2)));
    configured = dev;
  }
  k_glisa_hess64<<<hb.blocks[K_HESS], kH64Threads, smem, st>>>(hb.b[K_HESS], ld);
  ++g_launch_count;
}
void launch_change_g64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_BS(k_change_g64, K_ATOM_TILE, kThreads); }

}  // namespace hp
