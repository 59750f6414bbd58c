// Blocked skew Gauss–Jordan sweep on 8×8 tiles of the upper triangle, for the FP64 tensor
// instruction (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind).
//
// The sweep of pfinv.cuh takes n/2 rank-2 passes over the matrix. Here K pivots are taken
// together: their row pairs are formed one after the other from the stored matrix plus the
// panel's own pending updates, and the matrix takes one rank-2K update per panel as a
// product of the panel with itself. Same pivot rule (p the smallest unswept index, q the first
// maximum of |A(p, j)| over unswept j), same status codes, same Pf product.
//
// With u, v the rows p and q before the step and a = A(p, q), the swept matrix is
//   A'(i, j) = Z(A)(i, j) + (ṽ_i ũ_j − ũ_i ṽ_j)/a,
// Z(A) the matrix with rows and columns p, q zeroed, ũ = u except ũ_p = −1, ũ_q = 0, and
// ṽ = v except ṽ_p = 0, ṽ_q = −1: no row or column is a special case of the update. A later
// pivot (p', q') of the same panel zeroes the panel's entries p', q' instead, so Z commutes
// with the pending updates and the panel can be applied at its end.
//
// Storage: tile (I, J), I ≤ J, holds A(8I + r, 8J + c) at 8r + (c ^ s(r)), s(r) = bit 1 of r in
// bit 2 and bit 2 of r in bit 1: the two values of an accumulator fragment stay side by side
// (a tile moves with one conflict-free 128-bit access per lane), a column of a tile falls into
// eight different bank pairs, and a tile read as the mma's left operand, plain or transposed,
// is free of conflicts too. Diagonal tiles keep only r < c valid. Why 8×8: the
// m8n8k4 accumulator, and the smallest padding of a triangle; the tiles of n = 224 (203 KB)
// and a K = 4 panel fill an SM's shared memory. m8n8k4 was measured at the FP64 pipe's full
// 64 FMA/clk/SM from eight warps on, like the larger f64 shapes.
#pragma once

#include "common.cuh"

namespace mvmcb {

constexpr int kTilePivots = 4;  // pivots per panel (K): rank-8 updates

__host__ __device__ constexpr int tri_blocks(int n) { return (n + 7) / 8; }
__host__ __device__ constexpr size_t tri_tile_doubles(int n) {
  return static_cast<size_t>(tri_blocks(n)) * (tri_blocks(n) + 1) / 2 * 64;
}
// Panel row stride (doubles): ≡ 4 mod 16, so that the four panel rows a fragment reads lie
// in different banks.
__host__ __device__ constexpr int tri_pan_stride(int n) { return (n + 15) / 16 * 16 + 4; }
__host__ __device__ constexpr size_t tri_pan_doubles(int n) {
  return static_cast<size_t>(2 * kTilePivots) * tri_pan_stride(n);
}
// Cross-warp pivot search (|x| and column of each panel warp's candidate), the status, the
// parity and Pf.
constexpr size_t kTriRedBytes = 8 * 8 + 8 * 4 + 2 * 4 + 8;

__device__ __forceinline__ int tri_tile(int nb, int I, int J) { return I * nb - I * (I + 1) / 2 + J; }

__device__ __forceinline__ int tri_swz(int r) { return ((r << 1) & 4) | ((r >> 1) & 2); }

// Offset of A(i, j), i < j (or i, j in one diagonal tile), in doubles.
__device__ __forceinline__ int tri_at(int nb, int i, int j) {
  return (tri_tile(nb, i >> 3, j >> 3) << 6) + ((i & 7) << 3) + ((j & 7) ^ tri_swz(i));
}

// Offset (in pairs of doubles) of the lane's accumulator fragment, row lane/4, columns
// 2·(lane % 4) and the next, in a tile.
__device__ __forceinline__ int tri_frag(int lane) {
  return ((lane >> 2) << 2) + ((lane & 3) ^ (tri_swz(lane >> 2) >> 1));
}

__device__ __forceinline__ double tri_get(const double* T, int nb, int i, int j) {
  if (i == j) return 0.0;
  return i < j ? T[tri_at(nb, i, j)] : -T[tri_at(nb, j, i)];
}

// T ← the skew matrix with A(i, j) = at(i, j) for i < j, by the warps of the block (each lane
// its two fragment entries, four tiles in flight per warp).
template <class F>
__device__ __forceinline__ void tri_fill(double* T, int n, int warp, int nwarp, F at) {
  const int lane = threadIdx.x & 31, nb = tri_blocks(n), ntile = nb * (nb + 1) / 2;
  const int r = lane >> 2, c0 = (lane & 3) * 2;
  double2* C = reinterpret_cast<double2*>(T) + tri_frag(lane);
  constexpr int W = 4;
  int I = 0, J = warp;
  while (I < nb && J >= nb) J += ++I - nb;
  for (int t = warp; t < ntile; t += W * nwarp) {
    double2 a[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const int i = 8 * I + r, j = 8 * J + c0;
      a[w].x = I < nb && i < j && j < n ? at(i, j) : 0.0;
      a[w].y = I < nb && i < j + 1 && j + 1 < n ? at(i, j + 1) : 0.0;
      J += nwarp;
      while (I < nb && J >= nb) J += ++I - nb;
    }
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (t + w * nwarp < ntile) C[(t + w * nwarp) * 32] = a[w];
  }
}

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// W tiles of a block row, C[32k] += a·b_k over kChunks steps of four: every load before the
// first mma, no test in between (the caller splits a row into runs of four and the rest).
template <int W, int kChunks>
__device__ __forceinline__ void tile_run(double2* C, const double* b, int bstep, int bchunk, const double (&a)[kChunks]) {
  double2 c[W];
  double bb[W][kChunks];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    c[w] = C[32 * w];
#pragma unroll
    for (int h = 0; h < kChunks; ++h) bb[w][h] = b[w * bstep + h * bchunk];
  }
#pragma unroll
  for (int h = 0; h < kChunks; ++h)
#pragma unroll
    for (int w = 0; w < W; ++w) dmma884(c[w].x, c[w].y, a[h], bb[w][h]);
#pragma unroll
  for (int w = 0; w < W; ++w) C[32 * w] = c[w];
}
template <int kChunks>
__device__ __forceinline__ void tile_row(double2* C, const double* b, int bstep, int bchunk, const double (&a)[kChunks],
                                         int tiles) {
  for (; tiles >= 4; tiles -= 4, C += 128, b += 4 * bstep) tile_run<4, kChunks>(C, b, bstep, bchunk, a);
  if (tiles == 3) tile_run<3, kChunks>(C, b, bstep, bchunk, a);
  else if (tiles == 2) tile_run<2, kChunks>(C, b, bstep, bchunk, a);
  else if (tiles == 1) tile_run<1, kChunks>(C, b, bstep, bchunk, a);
}

// T(I, J) += Σ_k L(8I.., k)·R(k, 8J..) over the panel's 4·chunks rows, R row k = pan[k],
// L column 2l = pan[2l + 1], L column 2l + 1 = −pan[2l]. The warps take equal contiguous runs
// of tiles. Bound by shared memory: 8 wavefronts a tile for the tile itself and 4 for the
// fragments, against 8 cycles of the FP64 pipe.
template <int kChunks>
__device__ __forceinline__ void tri_update(double* T, const double* pan, int ps, int nb, int warp, int nwarp) {
  const int lane = threadIdx.x & 31, g = lane >> 2, k4 = lane & 3;
  const int ntile = nb * (nb + 1) / 2;
  int t = ntile * warp / nwarp;
  const int t1 = ntile * (warp + 1) / nwarp;
  int I = 0;
  while (I + 1 < nb && tri_tile(nb, I + 1, I + 1) <= t) ++I;
  int J = t - tri_tile(nb, I, I) + I;
  const double* bp = pan + k4 * ps + g;
  const double* ap = pan + (k4 ^ 1) * ps + g;
  double2* C = reinterpret_cast<double2*>(T) + tri_frag(lane);
  while (t < t1) {
    double a[kChunks];
#pragma unroll
    for (int h = 0; h < kChunks; ++h) {
      const double v = ap[4 * h * ps + 8 * I];
      a[h] = (k4 & 1) ? -v : v;
    }
    const int run = min(nb - J, t1 - t);
    tile_row<kChunks>(C + t * 32, bp + 8 * J, 8, 4 * ps, a, run);
    t += run;
    J = ++I;
  }
}

template <int G>
__device__ __forceinline__ void tri_bar() {
  if constexpr (G == 32) __syncwarp();
  else __syncthreads();
}
// Barrier of the first PG threads (the panel's) of a block of G.
template <int G, int PG>
__device__ __forceinline__ void tri_panel_bar() {
  if constexpr (PG == 32) __syncwarp();
  else if constexpr (PG == G) __syncthreads();
  else asm volatile("bar.sync 1, %0;" ::"n"(PG) : "memory");
}

// |x| as an integer of the same order; 0 (no pivot) for zero and NaN.
__device__ __forceinline__ unsigned long long tri_abs(double x) {
  return x == x ? static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7fffffffffffffffull : 0ull;
}

// The lane that holds the largest |x| of the warp's candidates (`at`, in column `col`), the
// lowest column among equal ones; -1 where all are zero. The high words decide unless two
// agree in them (then the low words, then the columns): one reduction and one vote on the chain.
__device__ __forceinline__ int tri_warp_max(unsigned long long at, int col) {
  constexpr unsigned kAll = 0xffffffffu;
  const unsigned hi = static_cast<unsigned>(at >> 32), lo = static_cast<unsigned>(at);
  const unsigned top = __reduce_max_sync(kAll, hi);
  unsigned who = __ballot_sync(kAll, hi == top);
  if (who & (who - 1)) {
    const unsigned low = __reduce_max_sync(kAll, hi == top ? lo : 0u);
    if ((top | low) == 0u) return -1;
    const bool mine = hi == top && lo == low;
    const unsigned first = __reduce_min_sync(kAll, mine ? static_cast<unsigned>(col) : kAll);
    who = __ballot_sync(kAll, mine && static_cast<unsigned>(col) == first);
  }
  return __ffs(static_cast<int>(who)) - 1;
}

// Sweep of the n×n skew matrix in T by G threads (a warp, or the whole block; every thread
// calls), n ≤ 256. The first PG threads form the panels: thread t < PG owns columns
// t + PG·c, c < CPT, PG·CPT ≥ n. pan: tri_pan_doubles(n) doubles; red: kTriRedBytes. On exit
// T holds X⁻¹ and every thread Pf and the status (0; k > 0: row k, 1-based, has no non-zero
// pivot; -1 non-finite). T is taken as complete after the call's first barrier and is
// complete after the call.
//
// A panel is a chain of latencies (row, maximum, partner row, reciprocal; about 1.1k cycles a
// pivot at n = 224), so the row of the next pivot is read and brought up to date (but for the
// current pivot) beside the partner row, and the sign of the permutation is summed per lane
// and reduced once at the end. n = 224, one plane per SM: 0.22 ms, half of it panels and half
// updates (1.75 ms as a packed triangle with one rank-2 pass per pivot).
template <int G, int PG, int CPT>
__device__ void tri_sweep(double* T, double* pan, unsigned char* red, int n, double& pf_out, int& status_out) {
  constexpr int K = kTilePivots;
  const int tg = G == 32 ? (threadIdx.x & 31) : threadIdx.x;
  const int lane = tg & 31, warp = tg >> 5;
  const int nb = tri_blocks(n), ps = tri_pan_stride(n);
  unsigned long long* rabs = reinterpret_cast<unsigned long long*>(red);
  int* rcol = reinterpret_cast<int*>(red + 64);
  int* rint = reinterpret_cast<int*>(red + 96);
  for (int j = tg; j < 2 * K * ps; j += G) pan[j] = 0.0;  // the padding stays zero
  if (tg == 0) rint[0] = 0;
  const bool panel = tg < PG;
  // swept set: lane l < 8 of a warp holds the bits of columns 32l .. 32l + 31 (set: swept or
  // beyond n)
  unsigned swept = 0xffffffffu;
  if (32 * lane < n) swept = n - 32 * lane >= 32 ? 0u : ~((1u << (n - 32 * lane)) - 1u);
  unsigned own = 0;  // bit c: column tg + PG·c swept or beyond n
  int row_at[CPT], col_at[CPT];  // offsets of the column as a row (j < i) and as a column
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    const int j = tg + PG * c;
    if (j >= n) own |= 1u << c;
    row_at[c] = (tri_tile(nb, j >> 3, 0) << 6) + ((j & 7) << 3);
    col_at[c] = (j >> 3) << 6;
  }
  // row i of the stored matrix at the own columns (zeroed behind the read), columns skip1 and
  // skip2 left alone
  auto take_row = [&](int i, int skip1, int skip2, double (&x)[CPT]) {
    const int bi = (tri_tile(nb, i >> 3, 0) << 6) + ((i & 7) << 3), ci = (i >> 3) << 6;
    const int si = tri_swz(i);
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const int j = tg + PG * c;
      x[c] = 0.0;
      if (j < n && j != i && j != skip1 && j != skip2) {
        double* e = T + (j > i ? bi + col_at[c] + ((j & 7) ^ si) : row_at[c] + ci + ((i & 7) ^ tri_swz(j)));
        x[c] = j > i ? *e : -*e;
        *e = 0.0;
      }
    }
  };
  int p = 0, status = 0, passed = 0;
  double pf = 1.0;
  for (int k0 = 0; k0 < n / 2; k0 += K) {
    const int kk = min(K, n / 2 - k0);
    tri_bar<G>();  // the matrix is complete
    if (panel) {
      double u[K][CPT], v[K][CPT];  // the panel's entries of the own columns
      double x[CPT];                // row p
      take_row(p, -1, -1, x);
      int pend = -1;  // q of the previous step, whose panel entries are zeroed one barrier late
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k >= kk) {  // a short last panel: empty rows
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            const int j = tg + PG * c;
            if (j < n) pan[2 * k * ps + j] = pan[(2 * k + 1) * ps + j] = 0.0;
          }
          continue;
        }
        if (k > 0) {
          tri_panel_bar<G, PG>();  // the previous step's panel rows
          const double up = pan[2 * (k - 1) * ps + p], vp = pan[(2 * k - 1) * ps + p];
#pragma unroll
          for (int c = 0; c < CPT; ++c) x[c] = fma(vp, u[k - 1][c], fma(-up, v[k - 1][c], x[c]));
        }
        unsigned long long big = 0ull;
        int q = n;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const int j = tg + PG * c;
          const unsigned long long v = tri_abs(x[c]);
          if (!((own >> c) & 1u) && j != p && v > big) {
            big = v;
            q = j;
          }
          if (j < n) pan[2 * k * ps + j] = x[c];
        }
        int src = tri_warp_max(big, q);
        if constexpr (PG == 32) {
          __syncwarp();
        } else {
          if (lane == max(src, 0)) {
            rabs[warp] = big;
            rcol[warp] = q;
          }
          tri_panel_bar<G, PG>();
          big = lane < PG / 32 ? rabs[lane] : 0ull;
          q = lane < PG / 32 ? rcol[lane] : n;
          src = tri_warp_max(big, q);
        }
        if (src < 0) {  // no pivot: every thread of the panel sees it
          status = p + 1;
          break;
        }
        q = __shfl_sync(0xffffffffu, q, src);
        const double a = pan[2 * k * ps + q];
        if (lane == (p >> 5)) swept |= 1u << (p & 31);
        if (lane == (q >> 5)) swept |= 1u << (q & 31);
        const int pn = __reduce_min_sync(0xffffffffu, ~swept ? 32 * lane + __ffs(~swept) - 1 : n);
        {  // unswept indices between p and q (everything below p is swept): this lane's share
          const int d = q - 32 * lane;
          passed += __popc(~swept & (d >= 32 ? 0xffffffffu : (d <= 0 ? 0u : (1u << d) - 1u)));
        }
        const bool more = k + 1 < kk;
        double y[CPT], xn[CPT];
        take_row(q, -1, -1, y);
        if (more) take_row(pn, p, q, xn);
        const double ia = 1.0 / a;
        pf *= a;
#pragma unroll
        for (int l = 0; l < k; ++l) {
          const double uq = pan[2 * l * ps + q], vq = pan[(2 * l + 1) * ps + q];
#pragma unroll
          for (int c = 0; c < CPT; ++c) y[c] = fma(vq, u[l][c], fma(-uq, v[l][c], y[c]));
          if (more) {
            const double un = pan[2 * l * ps + pn], vn = pan[(2 * l + 1) * ps + pn];
#pragma unroll
            for (int c = 0; c < CPT; ++c) xn[c] = fma(vn, u[l][c], fma(-un, v[l][c], xn[c]));
          }
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const int j = tg + PG * c;
          const bool is_p = j == p, is_q = j == q;
          u[k][c] = is_p ? -1.0 : (is_q ? 0.0 : x[c]);
          v[k][c] = is_p ? 0.0 : (is_q ? -ia : y[c] * ia);
          if (is_p || is_q) {
            own |= 1u << c;
            xn[c] = 0.0;
#pragma unroll
            for (int l = 0; l < k; ++l) u[l][c] = v[l][c] = 0.0;
          }
          // The panel's entries at p were last read before the pivot search. Those at q (and
          // the pivot itself) are being read: they are zeroed after the next barrier.
          if (is_p) {
#pragma unroll
            for (int l = 0; l < k; ++l) pan[2 * l * ps + j] = pan[(2 * l + 1) * ps + j] = 0.0;
            pan[2 * k * ps + j] = -1.0;
          }
          if (j < n) pan[(2 * k + 1) * ps + j] = v[k][c];
          if (k > 0 && j == pend) {
#pragma unroll
            for (int l = 0; l < k - 1; ++l) pan[2 * l * ps + j] = pan[(2 * l + 1) * ps + j] = 0.0;
            pan[2 * (k - 1) * ps + j] = 0.0;
          }
          x[c] = xn[c];
        }
        pend = q;
        p = pn;
      }
      if (status == 0) {
        tri_panel_bar<G, PG>();
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          if (tg + PG * c == pend) {
            for (int l = 0; l < kk - 1; ++l) pan[2 * l * ps + pend] = pan[(2 * l + 1) * ps + pend] = 0.0;
            pan[2 * (kk - 1) * ps + pend] = 0.0;
          }
      } else if (tg == 0) {
        rint[0] = status;
      }
    }
    tri_bar<G>();
    if (rint[0] != 0) break;
    tri_update<K / 2>(T, pan, ps, nb, tg >> 5, G / 32);
  }
  status = rint[0];
  tri_bar<G>();  // the matrix is complete
  // sgn(σ) and Pf from the panel's first warp
  double* rpf = reinterpret_cast<double*>(red + 104);
  if (tg < 32) {
    passed = __reduce_add_sync(0xffffffffu, passed);
    if (tg == 0) {
      rint[1] = passed;
      *rpf = pf;
    }
  }
  tri_bar<G>();
  double r = (rint[1] & 1) ? -*rpf : *rpf;
  if (status == 0 && !isfinite(r)) status = -1;
  if (status != 0) r = 0.0;
  pf_out = r;
  status_out = status;
  tri_bar<G>();
}

}  // namespace mvmcb
