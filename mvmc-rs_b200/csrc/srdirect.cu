// Direct SR on the device (NSRCG = 0): the Gram of the SR sample matrix, the S/g
// assembly on the active set, and the Cholesky solve.
//
// Reference: stochastic_opt_real_with_sr_info_timed (crates/mvmc-core/src/sr.rs:77-160 of
// AtelierArith/mvmc-rs) over the SrStages seam — gram_real (sr_backend.rs:464; the C order
// is one dgemm of the stored rows, c_order_gram_real :312), assemble_s_g (:484-511) and
// cholesky_solve (sr.rs:535: LAPACK dpotrf('U') + dpotrs).
//
// K6 k_gram: OO = Σ_s O_s O_sᵀ / Wc over the stored rows on the FP64 tensor instruction
// (mma.sync m8n8k4; tcgen05 has no FP64 kind): 64×64 output tiles of the lower triangle, one
// per block of four warps, the sample axis through a three-stage cp.async ring, mirrored.
// K7 k_cholesky: one cooperative launch, right-looking with 64-wide panels: all blocks solve
// the panel rows below the diagonal block, then update the trailing lower triangle in 64×64
// mma tiles; block 0 updates and factors the next diagonal block meanwhile, so a panel costs
// two grid barriers. The right-hand side rides along as one more row, which makes it
// y = L⁻¹b. S = L Lᵀ with L = Uᵀ of dpotrf('U'). K8 k_cholesky_back: Lᵀx = y, one grid barrier
// per 64 unknowns. 64 rather than 32 columns a panel: half the barriers and half the traffic of
// the trailing matrix. The direct step at 4096 samples × 4226 parameters: 33.9 → 8.4 ms (FP64
// FMA tiles, 32-wide panels with three barriers, substitutions on one block before).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/mvmc_b200.h"
#include "../host/abi_common.h"
#include "common.cuh"
#include "skewtile.cuh"

namespace cgr = cooperative_groups;

namespace mvmcb {

constexpr int kGramTile = 64;
constexpr int kGramK = 16;       // samples per stage
constexpr int kGramStages = 3;
constexpr int kGramThreads = 128;
constexpr int kGramLd = kGramTile + 4;  // ≡ 4 mod 16: a fragment's four rows in different banks
constexpr int kCholB = 64;       // panel width and trailing-update tile
constexpr int kCholLd = kCholB + 4;
constexpr int kCholThreads = 256;

// Triangular tile index → (ti, tj), ti ≥ tj.
__device__ __forceinline__ void tri_index(int t, int& ti, int& tj) {
  ti = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) / 2.0);
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  while (ti * (ti + 1) / 2 > t) --ti;
  tj = t - ti * (ti + 1) / 2;
}

// Eight bytes to shared memory without a register (rows of an odd number of doubles allow no
// wider copy); zero where !on.
__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool on) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(on ? 8 : 0) : "memory");
}

// OO[i][j] (i ≥ j tiles) of the rows store[s][0..n) for s < ns, scaled by inv_w. A warp owns
// 32×32 outputs as 4×4 accumulators: eight fragment loads for sixteen mma's, a quarter of the
// shared-memory rate beside the full FP64 rate. Four blocks of 52 KB per SM: the 2278 tiles
// of 4227 columns fill 3.85 waves of 592.
__global__ void __launch_bounds__(kGramThreads, 4) k_gram(const double* __restrict__ store, int n, long long ns,
                                                          double inv_w, double* __restrict__ oo) {
  extern __shared__ __align__(16) unsigned char smem[];
  double* buf = reinterpret_cast<double*>(smem);  // [stage][A, B][kGramK][kGramLd]
  constexpr int kHalf = kGramK * kGramLd, kStage = 2 * kHalf;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, k4 = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  int ti, tj;
  tri_index(blockIdx.x, ti, tj);
  const int i0 = ti * kGramTile, j0 = tj * kGramTile;
  const long long chunks = (ns + kGramK - 1) / kGramK;
  auto load = [&](long long c) {
    double* dst = buf + static_cast<int>(c % kGramStages) * kStage;
    const int col = tid & 63;
    const bool ia = i0 + col < n, ja = j0 + col < n;
#pragma unroll
    for (int e = 0; e < kGramK / 2; ++e) {
      const int r = (tid >> 6) + 2 * e;
      const long long s = c * kGramK + r;
      const double* row = store + (s < ns ? s : 0) * n;
      cp_async8(dst + r * kGramLd + col, row + (ia ? i0 + col : 0), ia && s < ns);
      cp_async8(dst + kHalf + r * kGramLd + col, row + (ja ? j0 + col : 0), ja && s < ns);
    }
  };
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  for (int c = 0; c < kGramStages - 1; ++c) {
    if (c < chunks) load(c);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (long long c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGramStages - 2) : "memory");
    __syncthreads();  // chunk c has arrived; chunk c − 1 has been read
    if (c + kGramStages - 1 < chunks) load(c + kGramStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double* A = buf + static_cast<int>(c % kGramStages) * kStage + k4 * kGramLd + wm + g;
    const double* B = buf + static_cast<int>(c % kGramStages) * kStage + kHalf + k4 * kGramLd + wn + g;
#pragma unroll
    for (int k = 0; k < kGramK; k += 4) {
      double av[4], bv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) av[a] = A[k * kGramLd + 8 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) bv[b] = B[k * kGramLd + 8 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma884(acc[a][b][0], acc[a][b][1], av[a], bv[b]);
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + wm + 8 * a + g, j = j0 + wn + 8 * b + 2 * k4 + h;
        if (i < n && j < n && i >= j) {
          const double v = acc[a][b][h] * inv_w;
          oo[static_cast<size_t>(i) * n + j] = v;
          oo[static_cast<size_t>(j) * n + i] = v;
        }
      }
}

// S[si][sj] = OO[pi][pj] − OO[0][pi]·OO[0][pj] (pi = map[si] + 1), diagonal × (1 + sta_del).
__global__ void k_assemble_s(const double* __restrict__ oo, int n, const int* __restrict__ map, int na,
                             double ratio_diag, double* __restrict__ s) {
  const long long total = static_cast<long long>(na) * na;
  for (long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; k < total;
       k += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int si = static_cast<int>(k / na), sj = static_cast<int>(k - static_cast<long long>(si) * na);
    const int pi = map[si] + 1, pj = map[sj] + 1;
    double v = oo[static_cast<size_t>(pi) * n + pj] - oo[pi] * oo[pj];
    if (si == sj) v *= ratio_diag;
    s[k] = v;
  }
}

// S of the active block from the tensor-core Gram of the centred, column-scaled samples
// (G = ÕᵀÕ, FP32, row stride ldg): S_ij = Wc⁻¹·cs_i·G_ij·cs_j, plus sta_del·var_i on the
// diagonal (the same operator the Gram form of SR-CG applies), in FP64.
__global__ void k_assemble_s_gram(const float* __restrict__ g, int ldg, const double* __restrict__ cs,
                                  const double* __restrict__ var, int na, double inv_wc, double sta_del,
                                  double* __restrict__ s) {
  const long long total = static_cast<long long>(na) * na;
  for (long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; k < total;
       k += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(k / na), j = static_cast<int>(k - static_cast<long long>(i) * na);
    double v = inv_wc * (cs[i] * static_cast<double>(g[static_cast<size_t>(i) * ldg + j]) * cs[j]);
    if (i == j) v += sta_del * var[i];
    s[k] = v;
  }
}

// Factor of the kb×kb diagonal block in D (lower, in place) by the whole block. fail: 1-based
// column of the first non-positive or non-finite pivot, 0 none (such a pivot counts as 1).
__device__ int factor_diagonal(double (*D)[kCholLd], int kb) {
  const int tid = threadIdx.x, nt = blockDim.x;
  int fail = 0;
  for (int j = 0; j < kb; ++j) {
    double d = D[j][j];
    if (!(d > 0.0) || !isfinite(d)) {  // the same value in every thread
      if (!fail) fail = j + 1;
      d = 1.0;
    }
    d = sqrt(d);
    const double rd = 1.0 / d;
    __syncthreads();  // D[j][j] read
    for (int i = j + tid; i < kb; i += nt) D[i][j] = i == j ? d : D[i][j] * rd;
    __syncthreads();
    // sixteen threads per row of the trailing block
    for (int i = j + 1 + tid / 16; i < kb; i += nt / 16) {
      const double lij = D[i][j];
      for (int c = j + 1 + tid % 16; c <= i; c += 16) D[i][c] -= lij * D[c][j];
    }
    __syncthreads();
  }
  return fail;
}

// In-place lower Cholesky of the row-major n×n matrix a (the lower triangle is read and
// written) with b as row n: b becomes L⁻¹b. info: 0, or the 1-based row of the first
// non-positive / non-finite pivot.
__global__ void __launch_bounds__(kCholThreads, 2) k_cholesky(double* __restrict__ a, int n, double* __restrict__ b,
                                                              int* info) {
  cgr::grid_group grid = cgr::this_grid();
  extern __shared__ __align__(16) unsigned char smem[];
  double(*Li)[kCholLd] = reinterpret_cast<double(*)[kCholLd]>(smem);
  double(*Lj)[kCholLd] = Li + kCholB;
  __shared__ double rdiag[kCholB];
  const int tid = threadIdx.x, nt = kCholThreads, lane = tid & 31, warp = tid >> 5, g = lane >> 2, k4 = lane & 3;
  auto row_of = [&](int r) { return r < n ? a + static_cast<size_t>(r) * n : b; };
  // block 0: factor the diagonal block at k (in Li, or read from a) and store it
  auto diagonal = [&](int k, bool loaded) {
    const int kb = min(kCholB, n - k);
    if (!loaded)
      for (int e = tid; e < kb * kb; e += nt) {
        const int r = e / kb, c = e - r * kb;
        Li[r][c] = c <= r ? a[static_cast<size_t>(k + r) * n + k + c] : 0.0;
      }
    __syncthreads();
    const int fail = factor_diagonal(Li, kb);
    for (int e = tid; e < kb * kb; e += nt) {
      const int r = e / kb, c = e - r * kb;
      if (c <= r) a[static_cast<size_t>(k + r) * n + k + c] = Li[r][c];
    }
    if (tid == 0 && fail && *info == 0) *info = k + fail;
    __syncthreads();
  };
  if (blockIdx.x == 0) diagonal(0, false);
  grid.sync();
  for (int k0 = 0; k0 < n; k0 += kCholB) {
    if (*reinterpret_cast<volatile int*>(info) != 0) return;  // every block reads the same flag after the barrier
    const int kb = min(kCholB, n - k0), top = k0 + kb;
    const int rest = n + 1 - top;  // rows below, the right-hand side among them
    // (1) panel rows: L[i][k0..) = A[i][k0..)·D⁻ᵀ, 32 rows per block, eight lanes per row, eight
    // columns at a time: the finished columns' products, then the 8×8 triangle by shuffles
    if (blockIdx.x * 32 < rest) {
      for (int e = tid; e < kCholB * kCholB; e += nt) {
        const int r = e / kCholB, c = e % kCholB;
        Li[r][c] = r < kb && c <= r ? a[static_cast<size_t>(k0 + r) * n + k0 + c] : (r == c ? 1.0 : 0.0);
      }
      __syncthreads();
      if (tid < kCholB) rdiag[tid] = 1.0 / Li[tid][tid];
      for (int r0 = blockIdx.x * 32; r0 < rest; r0 += gridDim.x * 32) {
        __syncthreads();
        for (int e = tid; e < 32 * kCholB; e += nt) {
          const int r = e / kCholB, c = e % kCholB;
          Lj[r][c] = r0 + r < rest && c < kb ? row_of(top + r0 + r)[k0 + c] : 0.0;
        }
        __syncthreads();
        double* x = Lj[warp * 4 + (lane >> 3)];
        const int c8 = lane & 7;
        for (int jb = 0; jb < kCholB; jb += 8) {
          const int j = jb + c8;
          double t0 = x[j], t1 = 0.0;
          for (int k = 0; k < jb; k += 2) {
            t0 -= x[k] * Li[j][k];
            t1 -= x[k + 1] * Li[j][k + 1];
          }
          double t = t0 + t1;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const double xc = __shfl_sync(0xffffffffu, t * rdiag[jb + c8], c, 8);
            if (c8 == c) t = xc;
            if (c8 > c) t -= xc * Li[j][jb + c];
          }
          __syncwarp();
          x[j] = t;
          __syncwarp();
        }
        __syncthreads();
        for (int e = tid; e < 32 * kCholB; e += nt) {
          const int r = e / kCholB, c = e % kCholB;
          if (r0 + r < rest && c < kb) row_of(top + r0 + r)[k0 + c] = Lj[r][c];
        }
      }
    }
    if (top >= n) break;  // only the right-hand side was left
    grid.sync();
    // (2) trailing update of the lower triangle and of the right-hand side in 64×64 tiles
    const int mt = (rest + kCholB - 1) / kCholB;
    const int ntiles = mt * (mt + 1) / 2;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 32;
    const int step = max(1, static_cast<int>(gridDim.x) - 1);
    for (int t = gridDim.x == 1 ? 0 : (blockIdx.x == 0 ? 0 : static_cast<int>(blockIdx.x)); t < ntiles;
         t += blockIdx.x == 0 && gridDim.x > 1 ? ntiles : step) {
      int ti, tj;
      tri_index(t, ti, tj);
      const int i0 = top + ti * kCholB, j0 = top + tj * kCholB;
      if (j0 >= n) continue;
      __syncthreads();
      for (int e = tid; e < kCholB * kCholB; e += nt) {
        const int r = e / kCholB, c = e % kCholB;
        const bool on = c < kb;
        Li[r][c] = on && i0 + r <= n ? __ldcg(row_of(i0 + r) + k0 + c) : 0.0;
        Lj[r][c] = on && j0 + r < n ? __ldcg(a + static_cast<size_t>(j0 + r) * n + k0 + c) : 0.0;
      }
      double acc[2][4][2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = i0 + wm + 8 * u + g, j = j0 + wn + 8 * v + 2 * k4 + h;
            acc[u][v][h] = i <= n && j < n && j <= i ? __ldcg(row_of(i) + j) : 0.0;
          }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < kCholB; k += 4) {
        double av[2], bv[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) av[u] = -Li[wm + 8 * u + g][k + k4];
#pragma unroll
        for (int v = 0; v < 4; ++v) bv[v] = Lj[wn + 8 * v + g][k + k4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) dmma884(acc[u][v][0], acc[u][v][1], av[u], bv[v]);
      }
      const bool next_diagonal = t == 0;
      if (next_diagonal) __syncthreads();  // Li is rewritten below
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = wm + 8 * u + g, c = wn + 8 * v + 2 * k4 + h, i = i0 + r, j = j0 + c;
            if (next_diagonal && i < n && j < n) Li[r][c] = j <= i ? acc[u][v][h] : 0.0;
            else if (i <= n && j < n && j <= i) row_of(i)[j] = acc[u][v][h];
          }
      if (next_diagonal) diagonal(top, true);
    }
    grid.sync();
  }
}

// x = L⁻ᵀ y in place (b), L the lower factor: from the last 64 unknowns up, every block solves
// the 64×64 triangle itself and takes 32 of the columns still to be updated per pass.
__global__ void __launch_bounds__(kCholThreads) k_cholesky_back(const double* __restrict__ l, int n,
                                                                double* __restrict__ b, const int* info) {
  cgr::grid_group grid = cgr::this_grid();
  __shared__ double D[kCholB][kCholB + 1];
  __shared__ double x[kCholB];
  __shared__ double part[kCholThreads / 32][32];
  if (*info != 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kCholThreads / 32;
  for (int k0 = (n - 1) / kCholB * kCholB; k0 >= 0; k0 -= kCholB) {
    const int kb = min(kCholB, n - k0);
    for (int e = tid; e < kCholB * kCholB; e += kCholThreads) {
      const int r = e / kCholB, c = e % kCholB;
      D[r][c] = r < kb && c <= r ? l[static_cast<size_t>(k0 + r) * n + k0 + c] : (r == c ? 1.0 : 0.0);
    }
    __syncthreads();
    if (warp == 0) {
      double y0 = lane < kb ? __ldcg(b + k0 + lane) : 0.0, y1 = lane + 32 < kb ? __ldcg(b + k0 + lane + 32) : 0.0;
      const double r0 = 1.0 / D[lane][lane], r1 = 1.0 / D[lane + 32][lane + 32];
#pragma unroll 8
      for (int j = kCholB - 1; j >= 32; --j) {
        const double xj = __shfl_sync(0xffffffffu, y1 * r1, j - 32);
        if (lane + 32 == j) y1 = xj;
        if (lane + 32 < j) y1 -= D[j][lane + 32] * xj;
        y0 -= D[j][lane] * xj;
      }
#pragma unroll 8
      for (int j = 31; j >= 0; --j) {
        const double xj = __shfl_sync(0xffffffffu, y0 * r0, j);
        if (lane == j) y0 = xj;
        if (lane < j) y0 -= D[j][lane] * xj;
      }
      x[lane] = y0;
      x[lane + 32] = y1;
    }
    __syncthreads();
    for (int c0 = blockIdx.x * 32; c0 < k0; c0 += gridDim.x * 32) {
      const int c = c0 + lane;
      double t = 0.0;
      if (c < k0) {
#pragma unroll
        for (int r = 0; r < kCholB / kWarps; ++r) {
          const int rr = warp * (kCholB / kWarps) + r;
          if (rr < kb) t += l[static_cast<size_t>(k0 + rr) * n + c] * x[rr];
        }
      }
      part[warp][lane] = t;
      __syncthreads();
      if (warp == 0 && c < k0) {
        double s = 0.0;
        for (int u = 0; u < kWarps; ++u) s += part[u][lane];
        b[c] = __ldcg(b + c) - s;
      }
      __syncthreads();
    }
    grid.sync();  // the blocks have read their y before block 0 puts x there
    if (blockIdx.x == 0 && tid < kb) b[k0 + tid] = x[tid];
    __syncthreads();
  }
}

int launch_gram(const double* store, int n, long long ns, double inv_w, double* oo, cudaStream_t stream) {
  const int ntile = (n + kGramTile - 1) / kGramTile;
  const size_t smem = sizeof(double) * kGramStages * 2 * kGramK * kGramLd;
  MVMCB_CUDA(cudaFuncSetAttribute(k_gram, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  k_gram<<<ntile * (ntile + 1) / 2, kGramThreads, smem, stream>>>(store, n, ns, inv_w, oo);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

int launch_assemble_s(const double* oo, int n, const int* map, int na, double ratio_diag, double* s,
                      cudaStream_t stream) {
  const long long total = static_cast<long long>(na) * na;
  const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>((total + 255) / 256, 148LL * 16)));
  k_assemble_s<<<grid, 256, 0, stream>>>(oo, n, map, na, ratio_diag, s);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

int launch_assemble_s_gram(const float* g, int ldg, const double* cs, const double* var, int na, double inv_wc,
                           double sta_del, double* s, cudaStream_t stream) {
  const long long total = static_cast<long long>(na) * na;
  const int grid = static_cast<int>(std::max<long long>(1, std::min<long long>((total + 255) / 256, 148LL * 16)));
  k_assemble_s_gram<<<grid, 256, 0, stream>>>(g, ldg, cs, var, na, inv_wc, sta_del, s);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

// Factor a (n×n, device) and solve for b (device) in place; *info_dev set on failure.
int launch_cholesky_solve(double* a, int n, double* b, int* info_dev, cudaStream_t stream) {
  const size_t smem = sizeof(double) * 2 * kCholB * kCholLd;
  MVMCB_CUDA(cudaFuncSetAttribute(k_cholesky, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  int per = 0;
  MVMCB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cholesky, kCholThreads, smem));
  const int sms = current_device_attr(cudaDevAttrMultiProcessorCount);
  const int m = (n + kCholB) / kCholB;  // tile rows, the right-hand side's row among them
  // block 0 takes the next diagonal block, the others the rest of a step's tiles
  const int blocks = std::max(1, std::min(sms * std::max(1, std::min(per, 2)), m * (m + 1) / 2 + 1));
  MVMCB_CUDA(cudaMemsetAsync(info_dev, 0, sizeof(int), stream));
  void* args[] = {&a, &n, &b, &info_dev};
  MVMCB_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cholesky), blocks, kCholThreads, args, smem, stream));
  void* back[] = {&a, &n, &b, &info_dev};
  MVMCB_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_cholesky_back), std::max(1, std::min(sms, (n + 31) / 32)),
                                         kCholThreads, back, 0, stream));
  return kOk;
}

}  // namespace mvmcb

namespace {
struct DevBuf {
  void* p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
};
}  // namespace

// SrStages::gram_real (sr_backend.rs:464): out = Σ_s store[s]·store[s]ᵀ (host buffers;
// store rows of n values, samples rows).
extern "C" int mvmc_b200_gram(const double* store, int n, long long samples, double* out) {
  using namespace mvmcb;
  if (!store || !out || n <= 0 || samples < 0) return kErrArgument;
  DevBuf s, o;
  MVMCB_CUDA(cudaMalloc(&s.p, sizeof(double) * std::max<long long>(1, samples * n)));
  MVMCB_CUDA(cudaMalloc(&o.p, sizeof(double) * static_cast<size_t>(n) * n));
  if (samples > 0) MVMCB_CUDA(cudaMemcpy(s.p, store, sizeof(double) * samples * n, cudaMemcpyHostToDevice));
  const int rc = launch_gram(static_cast<double*>(s.p), n, samples, 1.0, static_cast<double*>(o.p), nullptr);
  if (rc != kOk) return rc;
  MVMCB_CUDA(cudaMemcpy(out, o.p, sizeof(double) * static_cast<size_t>(n) * n, cudaMemcpyDeviceToHost));
  return kOk;
}

// SrStages::cholesky_solve (sr_backend.rs:243-247): solve S x = rhs for the symmetric
// positive-definite row-major S (host buffers); rhs becomes x. Returns 1 when the
// factorisation meets a non-positive pivot or the solution is not finite (the reference's
// Err(())), 0 on success, < 0 on argument / CUDA errors.
extern "C" int mvmc_b200_cholesky_solve(const double* s, double* rhs, int n) {
  using namespace mvmcb;
  if (!s || !rhs || n <= 0) return kErrArgument;
  DevBuf a, b, info;
  MVMCB_CUDA(cudaMalloc(&a.p, sizeof(double) * static_cast<size_t>(n) * n));
  MVMCB_CUDA(cudaMalloc(&b.p, sizeof(double) * n));
  MVMCB_CUDA(cudaMalloc(&info.p, sizeof(int)));
  MVMCB_CUDA(cudaMemcpy(a.p, s, sizeof(double) * static_cast<size_t>(n) * n, cudaMemcpyHostToDevice));
  MVMCB_CUDA(cudaMemcpy(b.p, rhs, sizeof(double) * n, cudaMemcpyHostToDevice));
  const int rc = launch_cholesky_solve(static_cast<double*>(a.p), n, static_cast<double*>(b.p),
                                       static_cast<int*>(info.p), nullptr);
  if (rc != kOk) return rc;
  int h_info = 0;
  MVMCB_CUDA(cudaMemcpy(&h_info, info.p, sizeof(int), cudaMemcpyDeviceToHost));
  MVMCB_CUDA(cudaMemcpy(rhs, b.p, sizeof(double) * n, cudaMemcpyDeviceToHost));
  if (h_info != 0) return 1;
  for (int i = 0; i < n; ++i)
    if (!std::isfinite(rhs[i])) return 1;
  return kOk;
}
