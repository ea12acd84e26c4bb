// MBIS kernels in FP64 (the default precision), mbis.py:81-163 and
// core/stockholder.py:153-175 of the reference. All are bound by the FP64
// pipe (2 lanes per clock and SM), so they are written for few FP64
// instructions per (point, atom) pair: see hp_fp64.cuh. Shells enter as
// amplitude A = N S^3 / (8 pi) and exponent S; JobDev::keep holds the
// amplitudes of the parameters a pass evaluates (k_copy_old, the inner
// update), at the slot of N.
//
// Per job, where they take at most half of the remaining budget, the
// distances of all pairs (rd) and the pro-atoms of the last inner iteration
// (oldpro, valid on the (atom, tile) pairs flagged in oldok) are kept; jobs
// without them recompute the same bits.
#include <math.h>

#include <atomic>

#include "hp_inner.cuh"

namespace hp {

namespace {

constexpr int kQ = 2 * kMbisMaxShell + 1;

__device__ __forceinline__ const JobDev& decode_local_mb(const Batch& bt, int& local) {
  const int j = find_job(bt, blockIdx.x);
  local = blockIdx.x - bt.prefix[j];
  return bt.jobs[j];
}

__device__ __forceinline__ const JobDev& decode_at_mb(const Batch& bt, int& atom, int& tile) {
  int local;
  const JobDev& J = decode_local_mb(bt, local);
  atom = local / J.ntile;
  tile = local - atom * J.ntile;
  return J;
}

__device__ __forceinline__ const double* rd_row(const JobDev& J, int a) {
  return J.rd ? J.rd + (size_t)a * J.npoint : nullptr;
}

}  // namespace

// Distances of every (atom, point) pair, once per job initialisation.
__global__ void __launch_bounds__(kThreads) k_rdist64(Batch bt) {
  int blk;
  const JobDev& J = decode_local_mb(bt, blk);
  if (!J.rd) return;
  const int p = blk * kThreads + threadIdx.x;
  if (p >= J.npoint) return;
  for (int a = 0; a < J.natom; ++a) J.rd[(size_t)a * J.npoint + p] = f64::dist64(J, p, a);
}

// Pro-atoms and promolecule, one thread per point.
__global__ void __launch_bounds__(kThreads) k_promol64(Batch bt) {
  __shared__ double tab[f64::kExpTab];
  int blk;
  const JobDev& J = decode_local_mb(bt, blk);
  f64::load_exp64(tab, J.etab);
  __syncthreads();
  const int p = blk * kThreads + threadIdx.x;
  if (p >= J.npoint) return;
  double promol = 0.0;
  for (int a = 0; a < J.natom; ++a) {
    const int s0 = J.shell_off[a], n = J.shell_off[a + 1] - s0;
    const double r = f64::dist_of(J, rd_row(J, a), p, a);
    const double pro = f64::mbis_pro(J.keep + 2 * s0, J.propars + 2 * s0 + 1, 2, n, r, tab);
    J.rhoa[(size_t)a * J.npoint + p] = pro;
    promol += pro;
    promol += 1e-100;
  }
  J.promol[p] = promol;
  J.invpro[p] = 1.0 / promol;
}

// One (atom, tile) of an inner iteration with NSH shells: the moments
// sum w e_k rho_a / pro and sum w e_k r rho_a / pro of the bare exponentials
// e_k (the update multiplies by A_k) and the change sum w (oldpro - pro)^2.
// Per pair 12 FP64 instructions a shell (9 of the exponential) and 13 more.
// amp[2 k], cur[2 k + 1], prev[2 k], prev[2 k + 1]: the atom's amplitudes,
// exponents and previous parameters; put(slot, v) stores the tile's partials
// (slots 0 .. 2 NSH - 1 the moments, kQ - 1 the change).
template <int NSH, typename Put>
__device__ __forceinline__ void mbis_tile(const JobDev& J, int a, int tile, bool first,
                                          const double* amp, const double* cur, const double* prev,
                                          const double* tab, double* red, Put put) {
  constexpr int NQ = 2 * NSH + 1;
  double A[NSH], S[NSH], acc[NQ];
#pragma unroll
  for (int k = 0; k < NSH; ++k) {
    A[k] = amp[2 * k];
    S[k] = -cur[2 * k + 1];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) acc[q] = 0.0;
  const size_t row = (size_t)a * J.npoint;
  const double* __restrict__ ra = J.rhoa + row;
  const double* __restrict__ wv = J.w;
  const double* rd = rd_row(J, a);
  double* old = J.oldpro ? J.oldpro + row : nullptr;
  const bool stored = old && J.oldok[a * J.ntile + tile] != 0;
  const f64::Cutoff cut = f64::cutoff_of(J.density_cutoff);
  const int p0 = tile * J.tile_points + threadIdx.x;
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  // the next point's values are loaded while the current one is worked on
  double rn = 0.0, rhon = 0.0, wn = 0.0, on = 0.0;
  auto load = [&](int p) {
    if (p < p1) {
      rhon = ra[p];
      wn = wv[p];
      if (rd) rn = rd[p];
      if (stored && !first) on = old[p];
    }
  };
  load(p0);
  for (int p = p0; p < p1; p += kThreads) {
    const double r = rd ? rn : f64::dist64(J, p, a);
    const double rho = rhon, w = wn, oldv = on;
    load(p + kThreads);
    double e[NSH], pro = 0.0;
#pragma unroll
    for (int k = 0; k < NSH; ++k) {
      e[k] = f64::exp64(S[k] * r, tab);
      pro = __fma_rn(A[k], e[k], pro);
    }
    const bool sick = f64::below(rho, cut) || f64::below(pro, cut);
    // (no quotient where sick: far from the atom pro underflows, and a zero
    // divisor takes the divide's slow path)
    const double wr = sick ? 0.0 : w * f64::div64(rho, sick ? 1.0 : pro);
    const double wrr = wr * r;
#pragma unroll
    for (int k = 0; k < NSH; ++k) {
      acc[2 * k] = __fma_rn(e[k], wr, acc[2 * k]);
      acc[2 * k + 1] = __fma_rn(e[k], wrr, acc[2 * k + 1]);
    }
    if (old) old[p] = pro;
    if (first) continue;  // no change in the first iteration (the update takes 1e100)
    double op = oldv;
    if (!stored) {
      op = 0.0;
      for (int k = 0; k < NSH; ++k) {
        const double n = prev[2 * k], s = prev[2 * k + 1];
        op = __fma_rn(f64::mbis_amp(n, s), f64::exp64(-s * r, tab), op);
      }
    }
    const double d = op - pro;
    acc[NQ - 1] = __fma_rn(w * d, d, acc[NQ - 1]);
  }
  f64::block_sums<NQ>(acc, NQ, red, [&](int q, double v) { put(q == NQ - 1 ? kQ - 1 : q, v); });
  if (old && threadIdx.x == 0) J.oldok[a * J.ntile + tile] = 1;
}

template <typename Put>
__device__ __forceinline__ void mbis_tile_n(int nsh, const JobDev& J, int a, int tile, bool first,
                                            const double* amp, const double* cur, const double* prev,
                                            const double* tab, double* red, Put put) {
  switch (nsh) {
    case 1: mbis_tile<1>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    case 2: mbis_tile<2>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    case 3: mbis_tile<3>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    case 4: mbis_tile<4>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    case 5: mbis_tile<5>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    case 6: mbis_tile<6>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
    default: mbis_tile<7>(J, a, tile, first, amp, cur, prev, tab, red, put); break;
  }
}

// The per-atom cutoff of an inner iteration: rho_a below the cutoff on the
// whole tile (the moments are exact zeros) and a negligible change term. The
// tile's partials are zeroed and it is counted. One warp forms the bound: in
// every thread it costs as much of the FP64 pipe as the tile itself. Uniform
// over the block; skip_s: one int of shared memory.
template <typename Put>
__device__ __forceinline__ bool mbis_skip(const JobDev& J, int a, int tile, int nsh, bool first,
                                          const double* cur, const double* prev, const double* tab,
                                          Put put, int* skip_s) {
  if (!J.tgeo || !(J.amax[(size_t)a * J.ntile + tile] < (float)J.density_cutoff)) return false;
  if (threadIdx.x < 32) {
    const double b = f64::mbis_bound_warp(cur, first ? nullptr : prev, nsh, tile_rmin(J, a, tile), tab);
    *skip_s = tile_weight(J, tile) * b * b < kSkipRel * J.inner_threshold * J.inner_threshold;
  }
  __syncthreads();
  const bool skip = *skip_s != 0;
  __syncthreads();
  if (!skip) return false;
  if (threadIdx.x < 2 * nsh) put((int)threadIdx.x, 0.0);
  if (threadIdx.x == 0) {
    put(kQ - 1, 0.0);
    if (J.oldok) J.oldok[a * J.ntile + tile] = 0;
    count_skipped(J, tile, 1.0);
  }
  return true;
}

// MBIS inner iteration, one block per (atom, tile). Bound by the FP64 pipe:
// about 30 FP64 instructions a pair at 1.5 shells, against ~150 when the
// distance, the old pro-atom's exponentials, CUDA's exp and divide and the
// sums of seven shells were all formed per pair. Two outer iterations of a
// 22-atom chain of 320k points: 116.7 -> 29.6 ms (85 % of the FP64 issue).
// Three blocks an SM: best at one and two shells; from four on the registers
// spill (516 bytes at seven), and it is still 3.9 times as fast as the kernel
// before (10 atoms, 145,500 points, 40 iterations: 34.3 -> 8.6 ms at 4
// shells, 49.6 -> 12.7 at 7).
__global__ void __launch_bounds__(kThreads, 3) k_mbis_inner64(Batch bt) {
  __shared__ double tab[f64::kExpTab];
  __shared__ double red[kQ * kThreads];
  __shared__ int skip_s;
  int a, tile;
  const JobDev& J = decode_at_mb(bt, a, tile);
  f64::load_exp64(tab, J.etab);
  inner_begin();
  if (!J.active[a]) return;
  __syncthreads();  // the table
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const bool first = J.inner_it[a] == 0;
  const double *amp = J.keep + 2 * s0, *cur = J.cur + 2 * s0, *prev = J.prev + 2 * s0;
  double* out = J.apart + ((size_t)a * J.qa + QA_INNER) * J.ntile + tile;
  const int nt = J.ntile;
  auto put = [&](int slot, double v) { out[(size_t)slot * nt] = v; };
  if (!mbis_skip(J, a, tile, nsh, first, cur, prev, tab, put, &skip_s))
    mbis_tile_n(nsh, J, a, tile, first, amp, cur, prev, tab, red, put);
  if (last_block_of(J, a)) mbis_update(J, a);
}

// The whole inner solve of every atom in one launch, for batches small enough
// that all blocks are resident (a cooperative launch): atom a's blocks (T
// consecutive tiles each) go through its iterations together; each of them
// sums the atom's partials in the order of warp_tile_sum and forms the same
// new parameters, so nothing is handed back. Bits as k_mbis_inner64.
//
// Latency-bound: the partials travel as 16-byte packets (value, tag), written
// and read as one access each, and a reader polls the packets themselves: one
// L2 round trip an iteration instead of the four of a fence, a counter, its
// poll and the partials, and no acquire that empties the L1 cache the tiles'
// values are read from. The tag holds the launch's number and the iteration.
// The packets alternate between two buffers: a block writes iteration i + 2
// when it has read all packets of i + 1, whose writers had read those of i.
//
// FP64 issue is shared by the blocks of an SM, and the atoms with most shells
// iterate longest: their blocks come last in the grid, where each has an SM
// with a lighter one (first, the few SMs that are filled first held two of
// the heaviest blocks, and every iteration waited for them).
// Water (3 atoms, 291 blocks) through the class: 14.0 -> 11.4 ms
// (counter and 512-point tiles before; 21.1 with a launch per iteration).
//
// The wait is bounded: a block that runs out of polls sets E_TIMEOUT and
// ends, and so do the others, each by its own bound (max_polls; kSolvePolls is
// most of a second).

__device__ __forceinline__ void put_packet(ulonglong2* p, double v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}

__device__ __forceinline__ double get_packet(const ulonglong2* p, unsigned long long& tag) {
  long long v;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
      : "=l"(v), "=l"(tag)
      : "l"(p)
      : "memory");
  return __longlong_as_double(v);
}

// The warp's sum of ntile packets of this tag, in the order of
// warp_tile_sum_of; waits for them (*late is set where they do not come).
__device__ __forceinline__ double packet_sum(const ulonglong2* pk, int ntile, unsigned long long tag,
                                             int max_polls, int* late) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int t = threadIdx.x & 31; t < ntile; t += 256) {
    double v[8];
    int polls = 0;
    bool ok;
    do {
      ok = true;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        v[u] = 0.0;
        if (t + 32 * u < ntile) {
          unsigned long long g;
          v[u] = get_packet(pk + t + 32 * u, g);
          ok &= g == tag;
        }
      }
    } while (!ok && ++polls < max_polls);
    if (!ok) *late = 1;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      if (t + 32 * h + 96 < ntile) {
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += v[h + u];
      } else {  // the last up to three
        s[0] = ((s[0] + v[h]) + v[h + 1]) + v[h + 2];
      }
    }
  }
  __syncwarp();
  double y = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
  return y;
}

__global__ void __launch_bounds__(kThreads, 2) k_mbis_solve64(Batch bt, int T, unsigned seq, int max_polls) {
  __shared__ double tab[f64::kExpTab];
  __shared__ double red[kQ * kThreads];
  __shared__ double amp[2 * kMbisMaxShell], cur[2 * kMbisMaxShell], prev[2 * kMbisMaxShell];
  __shared__ double m[kQ];
  __shared__ int skip_s, late_s, state_s, atom_s;
  int local;
  const JobDev& J = decode_local_mb(bt, local);
  f64::load_exp64(tab, J.etab);
  const int nt = J.ntile, natom = J.natom;
  const int nb = (nt + T - 1) / T;  // blocks of an atom
  const int b = local % nb;
  {  // the (local / nb)-th atom by shell count
    int* cnt = reinterpret_cast<int*>(red);
    for (int i = threadIdx.x; i < natom; i += kThreads) cnt[i] = J.shell_off[i + 1] - J.shell_off[i];
    __syncthreads();
    for (int i = threadIdx.x; i < natom; i += kThreads) {
      int rank = 0;
      for (int k = 0; k < natom; ++k) rank += cnt[k] < cnt[i] || (cnt[k] == cnt[i] && k < i);
      if (rank == local / nb) atom_s = i;
    }
    if (threadIdx.x == 0) late_s = 0;
    __syncthreads();
  }
  const int a = atom_s;
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const int t0 = b * T, t1 = min(t0 + T, nt);
  if (threadIdx.x < 2 * nsh) {
    amp[threadIdx.x] = J.keep[2 * s0 + threadIdx.x];
    cur[threadIdx.x] = prev[threadIdx.x] = J.cur[2 * s0 + threadIdx.x];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int it = 0;; ++it) {
    const unsigned long long tag = ((unsigned long long)seq << 32) | (unsigned)(it + 1);
    ulonglong2* pk = J.spk + (size_t)(2 * a + (it & 1)) * J.spk_nq * nt;
    for (int tile = t0; tile < t1; ++tile) {
      auto put = [&](int slot, double v) {
        put_packet(pk + (size_t)(slot == kQ - 1 ? 2 * nsh : slot) * nt + tile, v, tag);
      };
      if (!mbis_skip(J, a, tile, nsh, it == 0, cur, prev, tab, put, &skip_s))
        mbis_tile_n(nsh, J, a, tile, it == 0, amp, cur, prev, tab, red, put);
      if (tile + 1 < t1) __syncthreads();  // red
    }
    for (int q = warp; q < 2 * nsh + 1; q += kWarps) {
      const double v = packet_sum(pk + (size_t)q * nt, nt, tag, max_polls, &late_s);
      if (lane == 0) m[q] = v;
    }
    __syncthreads();
    if (late_s) {
      if (threadIdx.x == 0) atomicOr(&J.mail->i[MI_ERR], E_TIMEOUT);
      return;
    }
    // the update (mbis_update): the parameters on warp 0, the test on warp 1
    if (threadIdx.x < nsh) {
      double n, s;
      f64::mbis_shell(amp[2 * threadIdx.x], m[2 * threadIdx.x], m[2 * threadIdx.x + 1], n, s);
      prev[2 * threadIdx.x] = cur[2 * threadIdx.x];
      prev[2 * threadIdx.x + 1] = cur[2 * threadIdx.x + 1];
      cur[2 * threadIdx.x] = n;
      cur[2 * threadIdx.x + 1] = s;
      amp[2 * threadIdx.x] = f64::mbis_amp(n, s);
    } else if (threadIdx.x == 32) {
      const double change = it == 0 ? 1e100 : sqrt(m[2 * nsh]);
      state_s = change < J.inner_threshold ? 1 : it + 1 >= J.inner_maxiter ? 2 : 0;
      if (b == 0) J.atom_out[a * AO_COUNT + AO_INNER_CHANGE] = change;
    }
    __syncthreads();
    const int state = state_s;
    if (state == 0) continue;
    if (b == 0) {
      if (threadIdx.x < 2 * nsh) J.propars[2 * s0 + threadIdx.x] = cur[threadIdx.x];
      if (threadIdx.x == 0) {
        inner_done(J, a, it + 1);
        if (state == 2) atomicOr(&J.mail->i[MI_WARN], W_INNER);
      }
    }
    return;
  }
}

// Outer change sum w (pro(new) - pro(old))^2 (core/iterstock.py:32-45).
__global__ void __launch_bounds__(kThreads) k_change64(Batch bt) {
  __shared__ double tab[f64::kExpTab];
  __shared__ double red[kThreads];
  __shared__ double co[4 * kMbisMaxShell];  // per shell: A, S of new and old
  __shared__ int skip_s;
  int a, tile;
  const JobDev& J = decode_at_mb(bt, a, tile);
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const double* pn = J.propars + 2 * s0;
  const double* po = J.propars_old + 2 * s0;
  f64::load_exp64(tab, J.etab);
  __syncthreads();
  if (J.tgeo) {  // per-atom cutoff: bound of the pair's change term
    if (threadIdx.x < 32) {
      const double b = f64::mbis_bound_warp(pn, po, nsh, tile_rmin(J, a, tile), tab);
      skip_s = tile_weight(J, tile) * b * b < kSkipRel * J.threshold * J.threshold;
    }
    __syncthreads();
    if (skip_s) {
      if (threadIdx.x == 0) {
        J.apart[((size_t)a * J.qa + QA_CHANGE) * J.ntile + tile] = 0.0;
        count_skipped(J, tile, 2.0);
      }
      return;
    }
  }
  if (threadIdx.x < 2 * nsh) {
    const int k = threadIdx.x >> 1;
    const double* q = (threadIdx.x & 1) ? po : pn;
    co[4 * k + 2 * (threadIdx.x & 1)] = f64::mbis_amp(q[2 * k], q[2 * k + 1]);
    co[4 * k + 2 * (threadIdx.x & 1) + 1] = q[2 * k + 1];
  }
  __syncthreads();
  const double* rd = rd_row(J, a);
  double acc[1] = {0.0};
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
    const double r = f64::dist_of(J, rd, p, a);
    const double d = f64::mbis_pro(co, co + 1, 4, nsh, r, tab) - f64::mbis_pro(co + 2, co + 3, 4, nsh, r, tab);
    acc[0] = __fma_rn(J.w[p] * d, d, acc[0]);
  }
  f64::block_sums<1>(acc, 1, red, [&](int, double v) {
    J.apart[((size_t)a * J.qa + QA_CHANGE) * J.ntile + tile] = v;
  });
}

// at_weights output: clip(pro_a / promol, 0, 1) into rhoa (use_old: the
// parameters at the start of the last outer iteration).
__global__ void __launch_bounds__(kThreads) k_final_atweights64(Batch bt, int use_old) {
  __shared__ double tab[f64::kExpTab];
  __shared__ double co[2 * kMbisMaxShell];
  int a, tile;
  const JobDev& J = decode_at_mb(bt, a, tile);
  const int s0 = J.shell_off[a], nsh = J.shell_off[a + 1] - s0;
  const double* par = (use_old ? J.propars_old : J.propars) + 2 * s0;
  f64::load_exp64(tab, J.etab);
  if (threadIdx.x < nsh) {
    co[2 * threadIdx.x] = f64::mbis_amp(par[2 * threadIdx.x], par[2 * threadIdx.x + 1]);
    co[2 * threadIdx.x + 1] = par[2 * threadIdx.x + 1];
  }
  __syncthreads();
  const double* rd = rd_row(J, a);
  const int p1 = min((tile + 1) * J.tile_points, J.npoint);
  for (int p = tile * J.tile_points + threadIdx.x; p < p1; p += kThreads) {
    const double pro = f64::mbis_pro(co, co + 1, 2, nsh, f64::dist_of(J, rd, p, a), tab);
    J.rhoa[(size_t)a * J.npoint + p] = fmin(fmax(pro / J.promol[p], 0.0), 1.0);
  }
}

#define HP_LAUNCH_MB(kernel, kind, threads, ...)                                       \
  do {                                                                                 \
    if (hb.blocks[kind] > 0) {                                                         \
      kernel<<<hb.blocks[kind], threads, 0, st>>>(hb.b[kind], ##__VA_ARGS__);          \
      ++g_launch_count;                                                                \
    }                                                                                  \
  } while (0)

void launch_rdist64(const HostBatch& hb, cudaStream_t st) { HP_LAUNCH_MB(k_rdist64, K_POINT1, kThreads); }

void launch_promol64(const HostBatch& hb, cudaStream_t st, bool weights) {
  HP_LAUNCH_MB(k_promol64, K_POINT1, kThreads);
  if (weights) launch_atweights(hb, st);
}

void launch_mbis_inner64(const HostBatch& hb, cudaStream_t st) {
  launch_inner_kernel(k_mbis_inner64, hb, K_ATOM_TILE, st);
}

// Blocks of k_mbis_solve64 that are resident together on this device.
int mbis_solve_capacity() {
  static thread_local int dev_of = -1, cap = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev_of != dev) {
    int per_sm = 0, sms = 0, coop = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mbis_solve64, kThreads, 0);
    cap = coop ? per_sm * sms : 0;
    dev_of = dev;
  }
  return cap;
}

cudaError_t launch_mbis_solve64(const HostBatch& hb, cudaStream_t st, int polls) {
  Batch bt = hb.b[K_SOLVE];
  int T = hb.solve_tiles;
  // launches are numbered (packet tags), from 1: the packets start as zeros
  static std::atomic<unsigned> launches{0};
  unsigned seq = ++launches;
  if (seq == 0) seq = ++launches;
  void* args[] = {&bt, &T, &seq, &polls};
  const cudaError_t e = cudaLaunchCooperativeKernel((void*)k_mbis_solve64, dim3((unsigned)hb.blocks[K_SOLVE]),
                                                    dim3(kThreads), args, 0, st);
  if (e == cudaSuccess) ++g_launch_count;
  return e;
}

void launch_change64(const HostBatch& hb, cudaStream_t st) {
  HP_LAUNCH_MB(k_change64, K_ATOM_TILE, kThreads);
}

void launch_final_atweights64(const HostBatch& hb, cudaStream_t st, int use_old) {
  HP_LAUNCH_MB(k_final_atweights64, K_ATOM_TILE, kThreads, use_old);
}

}  // namespace hp
