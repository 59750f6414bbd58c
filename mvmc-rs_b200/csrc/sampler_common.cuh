// Device helpers of the samplers: projection counters, the amplitude, configuration moves
// and the initial configuration.
#pragma once

#include "common.cuh"
#include "engine.cuh"
#include "sfmt.cuh"

namespace mvmcb {

// ---- projection counters --------------------------------------------------------------
__device__ inline void make_proj_cnt_serial(const DevModel& m, const int* num, int* cnt) {
  for (int k = 0; k < m.nproj; ++k) cnt[k] = 0;
  for (int ri = 0; ri < m.ns; ++ri) {
    const int g = m.gutz_idx[ri];
    if (m.n_gutz > 0 && g >= 0 && g < m.nproj) cnt[g] += num[ri] * num[ri + m.ns];
  }
  if (m.n_jast > 0)
    for (int ri = 0; ri < m.ns; ++ri) {
      const int xi = num[ri] + num[ri + m.ns] - 1;
      if (xi == 0) continue;
      for (int rj = ri + 1; rj < m.ns; ++rj) {
        const int j = __ldg(m.jast_idx + ri * m.ns + rj);
        if (j < 0) continue;
        const int xj = num[rj] + num[rj + m.ns] - 1;
        if (m.n_gutz + j < m.nproj) cnt[m.n_gutz + j] += xi * xj;
      }
    }
}

// Projection counters from the configuration by the whole CTA (make_proj_cnt,
// projection.rs:179): integer sums, so the order of the atomics does not matter.
__device__ inline void make_proj_cnt_cta(const DevModel& m, const int* jtab, const int* num, int* cnt) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
  const int ns = m.ns;
  for (int k = tid; k < m.nproj; k += nt) cnt[k] = 0;
  __syncthreads();
  if (m.n_gutz > 0)
    for (int r = tid; r < ns; r += nt) {
      const int g = m.gutz_idx[r];
      const int v = num[r] * num[r + ns];
      if (v && g >= 0 && g < m.nproj) atomicAdd(cnt + g, v);
    }
  if (m.n_jast > 0)
    for (int ri = warp; ri < ns; ri += nwarp) {
      const int xi = num[ri] + num[ri + ns] - 1;
      if (xi == 0) continue;
      for (int rj = ri + 1 + lane; rj < ns; rj += 32) {
        const int j = jtab[ri * ns + rj];
        if (j < 0) continue;
        const int xj = num[rj] + num[rj + ns] - 1;
        if (xj != 0 && m.n_gutz + j < m.nproj) atomicAdd(cnt + m.n_gutz + j, xi * xj);
      }
    }
  __syncthreads();
}

__device__ __forceinline__ double log_ip_of(const DevModel& m, const double* pf, const double* qpw) {
  double ip = 0.0;
  for (int q = 0; q < m.nqp; ++q) ip += qpw[q] * pf[q];
  return log(fabs(ip));
}

// ---- serial helpers for thread 0 ------------------------------------------------------------
__device__ __forceinline__ void move_electron(const DevModel& m, int* idx, int* cfg, int* num, int mi,
                                              int ri, int rj, int sp) {
  const int msa = mi + sp * m.ne, ro = ri + sp * m.ns, rn = rj + sp * m.ns;
  idx[msa] = rj;
  cfg[ro] = -1;
  cfg[rn] = mi;
  num[ro] = 0;
  num[rn] = 1;
}
__device__ __forceinline__ void revert_electron(const DevModel& m, int* idx, int* cfg, int* num, int mi,
                                                int ri, int rj, int sp) {
  const int msa = mi + sp * m.ne, ro = ri + sp * m.ns, rn = rj + sp * m.ns;
  idx[msa] = ri;
  cfg[ro] = mi;
  cfg[rn] = -1;
  num[ro] = 1;
  num[rn] = 0;
}

__device__ inline void make_initial_sample_dev(const DevModel& m, SfmtRef& rng, int* idx, int* cfg, int* num,
                                        int* cnt) {
  for (int k = 0; k < m.n; ++k) idx[k] = -1;
  for (int k = 0; k < m.ns2; ++k) cfg[k] = -1;
  for (int si = 0; si < 2; ++si)
    for (int mi = 0; mi < m.ne; ++mi) {
      int guard = 0;
      while (true) {
        const int ri = static_cast<int>(rng.mod(m.ns));
        if (cfg[ri + si * m.ns] == -1) {
          cfg[ri + si * m.ns] = mi;
          idx[mi + si * m.ne] = ri;
          break;
        }
        if (++guard > (1 << 24)) break;  // unreachable for ne <= nsite
      }
    }
  for (int r = 0; r < m.ns2; ++r) num[r] = cfg[r] < 0 ? 0 : 1;
  make_proj_cnt_serial(m, num, cnt);
}

}  // namespace mvmcb
