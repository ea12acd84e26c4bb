// Inner iterations in one launch each: the blocks of an atom write their
// tile's partial sums, and the last of them to arrive (a counter per atom)
// sums the partials over the tiles in the fixed order of warp_tile_sum and
// updates the atom's parameters. No block waits for another one, and the
// values do not depend on which block comes last. Against an update kernel of
// one warp per atom this saves a launch per inner iteration, sums the
// quantities on several warps at once, and needs no kernel to count the atoms
// still active (MI_NACTIVE).
//
// The launches of consecutive inner iterations overlap (programmatic
// dependent launch): a kernel's blocks may start, and stage what no other
// kernel writes, while the previous iteration finishes; inner_begin waits for
// its results.
#pragma once

#include "hp_fp64.cuh"

namespace hp {

// Before the first read of anything the previous launch writes.
__device__ __forceinline__ void inner_begin() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename K>
inline void launch_inner_kernel(K kernel, const HostBatch& hb, int kind, cudaStream_t st) {
  if (hb.blocks[kind] <= 0) return;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)hb.blocks[kind]);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, hb.b[kind]);
  ++g_launch_count;
}

// True in the atom's last block (uniform over the block); call with all
// threads once the block's partials are written.
__device__ __forceinline__ bool last_block_of(const JobDev& J, int a) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&J.arrive[a], 1) == J.ntile - 1;
    if (last) {
      J.arrive[a] = 0;  // for the next launch
      __threadfence();
    }
  }
  __syncthreads();
  return last != 0;
}

// warp_tile_sum over partials that other blocks of this launch wrote (read
// from L2), the same order.
__device__ __forceinline__ double partial_value_cg(const JobDev& J, const double* slot) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(slot));
  return (double)v.x + (double)v.y;
}

__device__ __forceinline__ double warp_tile_sum_cg(const JobDev& J, const double* p, int ntile) {
  if (!J.mixed) return warp_tile_sum_of(ntile, [&](int t) { return __ldcg(p + t); });
  return warp_tile_sum_of(ntile, [&](int t) { return partial_value_cg(J, p + t); });
}

// Mixed precision only: the inner change of FP32-evaluated pro-atoms has a
// noise floor (about 1e-9 of the pro-atom's L2 norm), so the FP32 inner solve
// stops at 1000 x the inner threshold; the exact convergence to the
// threshold happens in the outer iterations that finish a mixed job.
__device__ __forceinline__ bool mixed_stalled(const JobDev& J, double change) {
  return J.mixed == PH_FP32 && change < 1e3 * J.inner_threshold;
}

// The atom's inner solve is over after `its` iterations.
__device__ __forceinline__ void inner_done(const JobDev& J, int a, int its) {
  J.active[a] = 0;
  atomicAdd(&J.mail->d[MD_INNER_TOTAL], (double)its);
  atomicMax(&J.mail->i[MI_INNER_MAX], its);
  atomicAdd(&J.mail->i[MI_NACTIVE], -1);
}

// Sums of the atom's quantities 0..nq-1 (slots QA_INNER + q; the last one at
// slot QA_INNER + qlast) over the tiles into m; one warp per quantity.
__device__ __forceinline__ void inner_sums(const JobDev& J, int a, int nq, int qlast, double* m) {
  const int warp = threadIdx.x >> 5;
  for (int q = warp; q < nq; q += kWarps) {
    const int slot = QA_INNER + (q == nq - 1 ? qlast : q);
    const double v = warp_tile_sum_cg(J, J.apart + ((size_t)a * J.qa + slot) * J.ntile, J.ntile);
    if ((threadIdx.x & 31) == 0) m[q] = v;
  }
  __syncthreads();
}

// MBIS update of one atom (mbis.py:140-160): N_k <- m0_k, S_k <- 3 m0_k /
// m1_k, convergence test. The moments of FP64 jobs are those of the bare
// exponentials: the amplitudes (keep) enter here, and those of the new
// parameters go there. Called by all threads of the atom's last block.
static __device__ __noinline__ void mbis_update(const JobDev& J, int a) {
  __shared__ double m[2 * kMbisMaxShell + 1];
  const int nsh = J.shell_off[a + 1] - J.shell_off[a];
  inner_sums(J, a, 2 * nsh + 1, 2 * kMbisMaxShell, m);
  if (threadIdx.x >= 32) return;  // one warp
  const int it = J.inner_it[a];
  __syncwarp();  // every lane has it before lane 0 writes the next one
  double* pc = J.cur + J.par_off[a];
  double* pp = J.prev + J.par_off[a];
  double* amp = J.keep + J.par_off[a];
  const int k = threadIdx.x;
  double n = 0.0, s = 0.0;
  if (k < nsh) {
    if (J.mixed) {
      n = m[2 * k];
      s = 3.0 * m[2 * k] / m[2 * k + 1];
    } else {
      f64::mbis_shell(amp[2 * k], m[2 * k], m[2 * k + 1], n, s);
    }
  }
  const double change = (it == 0) ? 1e100 : sqrt(m[2 * nsh]);
  const bool conv = change < J.inner_threshold || mixed_stalled(J, change);
  const bool stop = conv || it + 1 >= J.inner_maxiter;
  if (k < nsh) {
    if (stop) {
      double* pr = J.propars + J.par_off[a];
      pr[2 * k] = n;
      pr[2 * k + 1] = s;
    } else {
      pp[2 * k] = pc[2 * k];
      pp[2 * k + 1] = pc[2 * k + 1];
      pc[2 * k] = n;
      pc[2 * k + 1] = s;
      if (J.mixed) fill_fco(J, J.shell_off[a] + k, J.cur, J.prev);
      else amp[2 * k] = f64::mbis_amp(n, s);
    }
  }
  if (threadIdx.x == 0) {
    J.atom_out[a * AO_COUNT + AO_INNER_CHANGE] = change;
    if (!stop) {
      J.inner_it[a] = it + 1;
    } else {
      inner_done(J, a, it + 1);
      if (!conv) atomicOr(&J.mail->i[MI_WARN], W_INNER);
    }
  }
}

// NLIS update (nlis.py:99-195): N_k <- m0_k, S_k <- 3 / (n_k m1_k) (1e-5 where
// m1_k is within 1e-8 of zero, numpy.isclose), n_k fixed; convergence as MBIS.
static __device__ __noinline__ void nlis_update(const JobDev& J, int a) {
  __shared__ double m[2 * kMbisMaxShell + 1];
  const int nsh = J.shell_off[a + 1] - J.shell_off[a];
  inner_sums(J, a, 2 * nsh + 1, 2 * kMbisMaxShell, m);
  const int it = J.inner_it[a];
  const double change = (it == 0) ? 1e100 : sqrt(m[2 * nsh]);
  const bool conv = change < J.inner_threshold;
  const bool stop = conv || it + 1 >= J.inner_maxiter;
  double* pc = J.cur + J.par_off[a];
  double* pp = J.prev + J.par_off[a];
  if (threadIdx.x < nsh) {
    const int k = threadIdx.x;
    const double n = pc[3 * k + 2], m1 = m[2 * k + 1];
    const double nw[3] = {m[2 * k], fabs(m1) <= 1e-8 ? 1e-5 : 3.0 / (m1 * n), n};
    for (int q = 0; q < 3; ++q) {
      if (stop) {
        J.propars[J.par_off[a] + 3 * k + q] = nw[q];
      } else {
        pp[3 * k + q] = pc[3 * k + q];
        pc[3 * k + q] = nw[q];
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    J.atom_out[a * AO_COUNT + AO_INNER_CHANGE] = change;
    if (!stop) {
      J.inner_it[a] = it + 1;
    } else {
      inner_done(J, a, it + 1);
      if (!conv) atomicOr(&J.mail->i[MI_WARN], W_INNER);
    }
  }
}

// aLISA sc update (alisa.py:193-291): c_k <- m_k, convergence test.
static __device__ __noinline__ void lisa_sc_update(const JobDev& J, int a) {
  __shared__ double m[kMaxShells + 1];
  const int nsh = J.shell_off[a + 1] - J.shell_off[a];
  inner_sums(J, a, nsh + 1, kMaxShells, m);
  const int it = J.inner_it[a];
  const double change = (it == 0) ? 1e100 : sqrt(m[nsh]);
  const bool conv = change < J.inner_threshold || mixed_stalled(J, change);
  const bool stop = conv || it + 1 >= J.inner_maxiter;
  double* pc = J.cur + J.par_off[a];
  double* pp = J.prev + J.par_off[a];
  if (threadIdx.x < nsh) {
    const int k = threadIdx.x;
    if (stop) {
      J.propars[J.par_off[a] + k] = m[k];
    } else {
      pp[k] = pc[k];
      pc[k] = m[k];
      if (J.mixed) fill_fco(J, J.shell_off[a] + k, J.cur, J.prev);
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;  // the population test by warp 0 (warp_tile_sum)
  const double pop =
      conv && stop ? warp_tile_sum_cg(J, J.apart + ((size_t)a * J.qa + QA_POP) * J.ntile, J.ntile) : 0.0;
  if (threadIdx.x == 0) {
    J.atom_out[a * AO_COUNT + AO_INNER_CHANGE] = change;
    if (!stop) {
      J.inner_it[a] = it + 1;
    } else {
      inner_done(J, a, it + 1);
      double s = 0.0;
      for (int k = 0; k < nsh; ++k) s += m[k];
      if (!conv) atomicOr(&J.mail->i[MI_WARN], W_INNER);
      else if (fabs(s - pop) > J.population_cutoff) atomicOr(&J.mail->i[MI_WARN], W_POPULATION);
    }
  }
}

}  // namespace hp
