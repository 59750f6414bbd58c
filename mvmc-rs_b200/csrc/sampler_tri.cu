// K2t: the FP64 sampler with every plane of a walker in shared memory as tiles of the upper
// triangle, several proposals evaluated per pass (one CTA per walker).
//
// The draws, moves, decision rule and refresh rule are those of k_sample (sampler_impl.cuh).
// Sums run in another order, so that at a near-singular plane, where an FP64 log-weight is off
// by up to order 1 in any order, a chain may part from k_sample's (2D 8×8, eight planes: about
// one decision in 10⁷; neither is nearer to a long-double chain). Two things differ.
//
// Storage. A skew plane needs its upper triangle only, so planes that as squares live in L2
// (2D 8×8 with eight planes of 64: 256 KB; 2D 16×16, n = 224: 401 KB) fit one SM as tiles
// (147 KB, 203 KB), in the operand order of the FP64 mma (skewtile.cuh).
//
// Batches. Three of four proposals are rejected, and a rejected proposal leaves the
// configuration and the generator's next word unchanged but for the words it drew. So the
// control thread draws the candidates of the following proposals on the assumption that all
// are rejected, as many as fill eight vectors (one for a hop, two for an exchange), and
// one pass of mma's (M = plane rows, N = the eight vectors, K = plane columns) forms X·V of
// all of them. The decisions are then taken in order; the first acceptance ends the batch
// and sets the generator back to the word after its own draw. The pass also yields the
// vectors of the accepted move's update, which is then one rank-4 mma per tile:
//   hop:      X += v1′ ⊗ v2 − v2 ⊗ v1′, v1′ = X·slt + e_msa, v2 = −X[msa]/(X·slt)[msa]
//   exchange: X += Ct ⊗ t + Cs ⊗ s + Cq ⊗ (q + e_msb) + Cp ⊗ (p + e_msa) (update_two_real)
// A candidate that would need a new generator block is left to the next batch, since the
// words before it would be lost to a set-back.
//
// Bound by the latency of a batch's phases (2D 8×8, eight planes, one walker per SM: about 15k
// cycles of vectors and products, 5k of decisions, 11k of update per acceptance, for 2.4
// proposals). Sampling and measurement against k_sample with its planes in L2: 2D 8×8, 1024
// walkers, 68.7 → 44.7 ms; 2D 16×16, 1024 walkers, 60.3 → 23.3 ms; a step of the chain of 16
// sites with 256 walkers, 2.39 → 1.95 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "sampler_common.cuh"
#include "sfmt.cuh"
#include "skewtile.cuh"

namespace mvmcb {

namespace {

constexpr int kSlots = 8;  // proposals per batch at most, and vectors per pass

struct Slot {
  int type, skip, mi, ri, rj, sp, mj, t, msa, msb, col, cursor;
  int draws, pad;  // words drawn since the batch began
  double u, dproj;
};

// What the control warp counts (its first lane writes).
struct WalkerStats {
  long long counter[4], n_sched, n_guard;
  double drift_max;
  unsigned long long ph[kPhCount];
};

struct TriSampLayout {
  size_t sf, slots, ctl, stats, idx, cfg, num, pf, pfn, qpw, sc, bpart, vec, yvec, tiles, total;
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~size_t(15); }

__host__ __device__ inline size_t tri_vec_doubles(const DevModel& m) {
  return static_cast<size_t>(m.nqp) * tri_blocks(m.n) * 64;  // [plane][row][8]
}

// ysmem: the products beside the vectors in shared memory, else in the walker's workspace.
// sweeps: planes swept at a time by a refresh (their panels overlay the vectors).
__host__ __device__ inline TriSampLayout tri_samp_layout(const DevModel& m, bool ysmem, int sweeps) {
  TriSampLayout L;
  size_t o = 0;
  L.sf = o; o = al16(o + sizeof(uint32_t) * kSfmtN32);
  L.slots = o; o = al16(o + sizeof(Slot) * kSlots);
  L.ctl = o; o = al16(o + 64);
  L.stats = o; o = al16(o + sizeof(WalkerStats));
  L.idx = o; o = al16(o + sizeof(int) * m.n);
  L.cfg = o; o = al16(o + sizeof(int) * m.ns2);
  L.num = o; o = al16(o + sizeof(int) * m.ns2);
  L.pf = o; o = al16(o + sizeof(double) * m.nqp);
  L.pfn = o; o = al16(o + sizeof(double) * m.nqp * kSlots);
  L.qpw = o; o = al16(o + sizeof(double) * m.nqp);
  L.sc = o; o = al16(o + sizeof(double) * 8 * m.nqp * kSlots);
  L.bpart = o; o = al16(o + sizeof(double) * 4 * m.nqp * tri_blocks(m.n));
  L.vec = o;
  const size_t vec = sizeof(double) * tri_vec_doubles(m);
  const size_t pan = sweeps * al16(sizeof(double) * tri_pan_doubles(m.n) + kTriRedBytes);
  size_t room = ysmem ? 2 * vec : vec;
  room = room > pan ? room : pan;
  const size_t cnt = sizeof(int) * (m.nproj + 1);
  L.yvec = o + vec;
  o = al16(o + (room > cnt ? room : cnt));
  L.tiles = o; o += sizeof(double) * m.nqp * tri_tile_doubles(m.n);
  L.total = o;
  return L;
}

// The walker's generator, its cursor and word count in the control warp's registers.
struct Rng {
  uint32_t* s;
  int idx;
  unsigned long long draws;
  __device__ uint32_t u32() {
    if (idx >= kSfmtN32) {
      sfmt_gen_all(s);
      idx = 0;
    }
    ++draws;
    return s[idx++];
  }
  __device__ double real2() { return static_cast<double>(u32()) * (1.0 / 4294967296.0); }
  __device__ int mod(int n) { return static_cast<int>(u32() % static_cast<uint32_t>(n)); }
};

// x mod d by two multiplications (Lemire, Kaser, Kurz: Faster remainder by direct computation).
struct FastMod {
  unsigned long long m;
  uint32_t d;
  __device__ explicit FastMod(int n) : m(~0ull / static_cast<uint32_t>(n) + 1ull), d(static_cast<uint32_t>(n)) {}
  __device__ int operator()(uint32_t x) const { return static_cast<int>(__umul64hi(m * x, d)); }
};

// One proposal drawn word by word (by one thread), refilling the generator where needed: the
// first proposal of a batch near the end of a generator block, and every case the window of
// draw_window does not cover. The draws are those of get_update_type and
// make_candidate_hopping / _exchange, then the decision's.
__device__ int draw_serial(const DevModel& m, Rng& rng, const int* idx, const int* cfg, const int* num, Slot* slots,
                           unsigned* status) {
  const int ns = m.ns, ne = m.ne;
  const unsigned long long base = rng.draws;
  Slot& s = slots[0];
  int skip = 1, mi = 0, ri = 0, rj = 0, sp = 0, mj = 0, t = 0, type = 3;
  if (m.nex_path == 0) type = 0;
  else if (m.nex_path == 1) type = rng.real2() < 0.5 ? 1 : 0;
  else if (m.nex_path == 2) type = 1;
  if (type == 0) {
    mi = rng.mod(ne);
    sp = rng.real2() < 0.5 ? 0 : 1;
    ri = idx[mi + sp * ne];
    for (int icnt = 0; skip != 0; ++icnt) {
      rj = rng.mod(ns);
      if (icnt > ns * ns) break;  // no empty site found
      if (cfg[rj + sp * ns] == -1) skip = 0;
    }
  } else if (type == 1) {
    bool single = false;
    for (int r = 0; r < ns && !single; ++r) single = num[r] + num[r + ns] == 1;
    if (single) {
      constexpr int kLoopBound = 1 << 22;  // as in k_sample: only a malformed input gets there
      int guard = 0;
      while (true) {
        mi = rng.mod(ne);
        sp = rng.real2() < 0.5 ? 0 : 1;
        ri = idx[mi + sp * ne];
        if (cfg[ri + (1 - sp) * ns] == -1 || ++guard > kLoopBound) break;
      }
      t = 1 - sp;
      while (guard <= kLoopBound) {
        mj = rng.mod(ne);
        rj = idx[mj + t * ne];
        if (cfg[rj + sp * ns] == -1 || ++guard > kLoopBound) break;
      }
      if (guard > kLoopBound) atomicOr(status, kDevCandidateLoop);
      else skip = 0;
    }
  }
  s.type = type;
  s.skip = skip;
  s.mi = mi;
  s.ri = ri;
  s.rj = rj;
  s.sp = sp;
  s.mj = mj;
  s.t = t;
  s.msa = mi + sp * ne;
  s.msb = mj + t * ne;
  s.col = 0;
  s.u = skip ? 0.0 : rng.real2();
  s.cursor = rng.idx;
  s.draws = static_cast<int>(rng.draws - base);
  s.dproj = 0.0;
  return 1;
}

// Candidates of the next proposals by one warp, all but the first on the assumption that
// those before are rejected; returns their number (≥ 1, ≤ left). The next 64 words of the
// generator block are tested at once, two per lane, for every role a word can have (a
// spin, an electron of either spin that may be exchanged, a site empty for either spin);
// the draws of draw_serial are then a walk over the ballots of those tests, with no memory
// access in its chain. Proposals whose words the window does not hold stay undrawn.
__device__ int draw_window(const DevModel& m, const FastMod& by_ne, const FastMod& by_ns, Rng& rng, const int* idx,
                           const int* cfg, const int* num, Slot* slots, int left, unsigned* status) {
  const int ns = m.ns, ne = m.ne, lane = threadIdx.x & 31, path = m.nex_path;
  const int nw = min(64, kSfmtN32 - rng.idx);
  const uint32_t* w = rng.s + rng.idx;
  unsigned long long low = 0, s0 = 0, s1 = 0, h0 = 0, h1 = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool on = 32 * h + lane < nw;
    const uint32_t x = on ? w[32 * h + lane] : 0u;
    const int e = by_ne(x), r = by_ns(x);
    low |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, x < 0x80000000u)) << (32 * h);
    s0 |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, on && cfg[idx[e] + ns] == -1)) << (32 * h);
    s1 |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, on && cfg[idx[e + ne]] == -1)) << (32 * h);
    h0 |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, on && cfg[r] == -1)) << (32 * h);
    h1 |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, on && cfg[r + ns] == -1)) << (32 * h);
  }
  bool single = false;
  for (int r = lane; r < ns; r += 32) single = single || num[r] + num[r + ns] == 1;
  single = __any_sync(0xffffffffu, single);
  // bit k: words (k, k + 1) are an electron and its spin that may be exchanged
  const unsigned long long sh = low >> 1;
  const unsigned long long pair = ((sh & s0) | (~sh & s1)) & (nw > 0 ? (~0ull >> (64 - nw)) >> 1 : 0ull);
  auto from = [](unsigned long long mask, int k) { return k < 64 ? mask & (~0ull << k) : 0ull; };
  int n = 0, col = 0, p = 0;
  int my_type = 0, my_skip = 0, my_k = 0, my_j = 0, my_sp = 0, my_col = 0, my_end = 0;
  while (n < kSlots && n < left) {
    int q = p, type = 3, skip = 1, k = 0, j = 0, sp = 0;
    if (path == 1) {
      if (q >= nw) break;
      type = (low >> q) & 1ull ? 1 : 0;
      ++q;
    } else if (path == 0 || path == 2) {
      type = path >> 1;
    }
    if (type == 0) {
      k = q;
      if (k + 2 >= nw) break;
      sp = (low >> (k + 1)) & 1ull ? 0 : 1;
      const unsigned long long d = from(sp ? h1 : h0, k + 2);
      if (d == 0ull) break;
      j = __ffsll(static_cast<long long>(d)) - 1;
      if (j + 1 >= nw || j - (k + 2) > ns * ns) break;
      skip = 0;
      q = j + 2;
    } else if (type == 1 && single) {
      const unsigned long long a = from(pair & (0x5555555555555555ull << (q & 1)), q);
      if (a == 0ull) break;
      k = __ffsll(static_cast<long long>(a)) - 1;
      sp = (low >> (k + 1)) & 1ull ? 0 : 1;
      const unsigned long long d = from(sp ? s0 : s1, k + 2);
      if (d == 0ull) break;
      j = __ffsll(static_cast<long long>(d)) - 1;
      if (j + 1 >= nw) break;
      skip = 0;
      q = j + 2;
    }
    const int at = type == 1 ? (col + 1) & ~1 : col;
    const int next = skip ? col : at + (type == 1 ? 2 : 1);
    if (next > kSlots) break;
    if (lane == n) {
      my_type = type;
      my_skip = skip;
      my_k = k;
      my_j = j;
      my_sp = sp;
      my_col = at;
      my_end = q;
    }
    col = next;
    p = q;
    ++n;
  }
  if (n == 0) {
    if (lane == 0) draw_serial(m, rng, idx, cfg, num, slots, status);
    rng.idx = __shfl_sync(0xffffffffu, rng.idx, 0);
    rng.draws = __shfl_sync(0xffffffffu, rng.draws, 0);
    __syncwarp();
    return 1;
  }
  if (lane < n) {
    Slot& s = slots[lane];
    s.type = my_type;
    s.skip = my_skip;
    s.sp = my_sp;
    s.t = 1 - my_sp;
    s.col = my_col;
    s.cursor = rng.idx + my_end;
    s.draws = my_end;
    s.dproj = 0.0;
    if (!my_skip) {
      const int mi = by_ne(w[my_k]);
      s.mi = mi;
      s.ri = idx[mi + my_sp * ne];
      s.msa = mi + my_sp * ne;
      const int mj = by_ne(w[my_j]);
      s.mj = mj;
      s.msb = mj + (1 - my_sp) * ne;
      s.rj = my_type == 0 ? by_ns(w[my_j]) : idx[s.msb];
      s.u = static_cast<double>(w[my_end - 1]) * (1.0 / 4294967296.0);
    }
  }
  rng.idx += p;
  rng.draws += p;
  __syncwarp();
  return n;
}

// Δ ln P of a hop slot by one warp, from the configuration before the move
// (log_proj_ratio_hop_warp of sampler_impl.cuh, whose occupations are those after it).
__device__ double hop_dproj(const DevModel& m, const int* num, const Slot& s) {
  const int lane = threadIdx.x & 31, ns = m.ns, src = s.ri, dst = s.rj;
  double z = 0.0;
  if (m.n_jast > 0) {
    const double* vd = m.jast_pair + static_cast<size_t>(dst) * ns;
    const double* vs = m.jast_pair + static_cast<size_t>(src) * ns;
#pragma unroll 8
    for (int k = lane; k < ns; k += 32) {
      const int x = (k == src || k == dst) ? 0 : num[k] + num[k + ns] - 1;
      const double d = __ldg(vd + k) - __ldg(vs + k);
      if (x != 0) z += d * static_cast<double>(x);
    }
    z = warp_sum(z);
  }
  const int n_src = num[src] + num[src + ns] - 1, n_dst = num[dst] + num[dst + ns] + 1;
  z -= __ldg(m.gutz_site + src) * static_cast<double>(n_src);
  z += __ldg(m.gutz_site + dst) * static_cast<double>(num[dst + (1 - s.sp) * ns]);
  z += __ldg(m.jast_pair + static_cast<size_t>(src) * ns + dst) * static_cast<double>(n_src - n_dst + 1);
  return z;
}

// W tiles' share of a block row of X·V: acc_h += A_h(k)·B_h(k) for the two halves h of the
// eight columns (two accumulators: a chain of mma's waits for each other). Every load before
// the first mma.
template <int W, class At>
__device__ __forceinline__ void product_run(double (&acc)[2][2], const double* b, int at0, int at1, At tile) {
  double a0[W], a1[W], b0[W], b1[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const double* t = tile(w);
    a0[w] = t[at0];
    a1[w] = t[at1];
    b0[w] = b[64 * w];
    b1[w] = b[64 * w + 32];
  }
#pragma unroll
  for (int w = 0; w < W; ++w) {
    dmma884(acc[0][0], acc[0][1], a0[w], b0[w]);
    dmma884(acc[1][0], acc[1][1], a1[w], b1[w]);
  }
}

// Y = X·V of one block row of a plane, by one warp: Y[8I.., 8] = Σ_J X(I, J)·V[8J.., 8], with
// X(I, J) = −T(J, I)ᵀ left of the diagonal. Also the row block's share of Σ_i b_i·(X·a)_i for
// the vector pairs (a, b) = columns (2k, 2k + 1).
__device__ __forceinline__ void plane_row_product(const double* T, int nb, int I, const double* V, double* Y,
                                                  double* bpart) {
  const int lane = threadIdx.x & 31, g = lane >> 2, k4 = lane & 3;
  const double* b = V + k4 * 8 + g;
  double up[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, lo[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  const int cl0 = k4 * 8 + (g ^ tri_swz(k4)), cl1 = (k4 + 4) * 8 + (g ^ tri_swz(k4 + 4));
  const int cu0 = g * 8 + (k4 ^ tri_swz(g)), cu1 = g * 8 + ((k4 + 4) ^ tri_swz(g));
  {
    auto below = [&](int J) { return T + ((J * nb - J * (J + 1) / 2 + I) << 6); };
    int J = 0;
    for (; J + 4 <= I; J += 4) product_run<4>(lo, b + 64 * J, cl0, cl1, [&](int w) { return below(J + w); });
    if (I & 2) {
      product_run<2>(lo, b + 64 * J, cl0, cl1, [&](int w) { return below(J + w); });
      J += 2;
    }
    if (I & 1) product_run<1>(lo, b + 64 * J, cl0, cl1, [&](int w) { return below(J + w); });
  }
  const double* t = T + (tri_tile(nb, I, I) << 6);
  {
    const double u0 = t[cu0], u1 = t[cu1], l0 = t[cl0], l1 = t[cl1];
    const double b0 = b[64 * I], b1 = b[64 * I + 32];
    dmma884(up[0][0], up[0][1], g < k4 ? u0 : (g > k4 ? -l0 : 0.0), b0);
    dmma884(up[1][0], up[1][1], g < k4 + 4 ? u1 : (g > k4 + 4 ? -l1 : 0.0), b1);
  }
  {
    int J = I + 1;
    const int rest = nb - J;
    for (; J + 4 <= nb; J += 4)
      product_run<4>(up, b + 64 * J, cu0, cu1, [&](int w) { return t + ((J - I + w) << 6); });
    if (rest & 2) {
      product_run<2>(up, b + 64 * J, cu0, cu1, [&](int w) { return t + ((J - I + w) << 6); });
      J += 2;
    }
    if (rest & 1) product_run<1>(up, b + 64 * J, cu0, cu1, [&](int w) { return t + ((J - I + w) << 6); });
  }
  const double y0 = (up[0][0] + up[1][0]) - (lo[0][0] + lo[1][0]);
  const double y1 = (up[0][1] + up[1][1]) - (lo[0][1] + lo[1][1]);
  const int row = 8 * I + g;
  *reinterpret_cast<double2*>(Y + row * 8 + 2 * k4) = make_double2(y0, y1);
  double p = y0 * V[row * 8 + 2 * k4 + 1];
  p += __shfl_xor_sync(0xffffffffu, p, 4);
  p += __shfl_xor_sync(0xffffffffu, p, 8);
  p += __shfl_xor_sync(0xffffffffu, p, 16);
  if (g == 0) bpart[k4] = p;
}

// T(I, J) += L(8I..)·R(8J..)ᵀ over four columns for every plane's tiles, by warps w of nw.
__device__ __forceinline__ void rank4_update(double* tiles, size_t plane, const double* vec, int nqp, int nb, int w,
                                             int nw) {
  const int lane = threadIdx.x & 31, g = lane >> 2, k4 = lane & 3;
  for (int unit = w; unit < nqp * nb; unit += nw) {
    // rows in the order longest, shortest, second longest, … so that the warps end together
    const int q = unit / nb, e = unit - q * nb, I = (e & 1) ? nb - 1 - (e >> 1) : e >> 1;
    const double* L = vec + static_cast<size_t>(q) * nb * 64;
    double2* C = reinterpret_cast<double2*>(tiles + q * plane) + tri_tile(nb, I, I) * 32 + tri_frag(lane);
    const double a[1] = {L[(8 * I + g) * 4 + k4]};
    tile_row<1>(C, L + nb * 32 + (8 * I + g) * 4 + k4, 32, 0, a, nb - I);
  }
}

// NT threads per walker; PG = 32: a refresh sweeps a plane per warp, else the block sweeps the
// planes in turn, PG threads forming the panels.
template <int NT, int PG, int CPT>
__global__ void __launch_bounds__(NT, 512 / NT)
    k_sample_tri(DevModel m, DevWalkers w, int ysmem) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NW = NT / 32;
  constexpr bool kWarpSweep = PG == 32;
  const int wk = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = m.n, ns = m.ns, ne = m.ne, nqp = m.nqp, nb = tri_blocks(n);
  const TriSampLayout L = tri_samp_layout(m, ysmem != 0, kWarpSweep ? min(NW, nqp) : 1);
  uint32_t* sf = reinterpret_cast<uint32_t*>(smem + L.sf);
  Slot* slots = reinterpret_cast<Slot*>(smem + L.slots);
  int* ctl = reinterpret_cast<int*>(smem + L.ctl);  // batch size, accepted slot, consumed, refresh, info, burn
  double* dctl = reinterpret_cast<double*>(smem + L.ctl + 32);  // ln|IP|, refresh mask
  int* idx = reinterpret_cast<int*>(smem + L.idx);
  int* cfg = reinterpret_cast<int*>(smem + L.cfg);
  int* num = reinterpret_cast<int*>(smem + L.num);
  double* pf = reinterpret_cast<double*>(smem + L.pf);
  double* pfn = reinterpret_cast<double*>(smem + L.pfn);
  double* qpw = reinterpret_cast<double*>(smem + L.qpw);
  double* sc = reinterpret_cast<double*>(smem + L.sc);
  double* bpart = reinterpret_cast<double*>(smem + L.bpart);
  double* vec = reinterpret_cast<double*>(smem + L.vec);
  int* cnt = reinterpret_cast<int*>(smem + L.vec);  // projection counters, at save points
  double* tiles = reinterpret_cast<double*>(smem + L.tiles);
  const size_t plane = tri_tile_doubles(n);
  const size_t nn = static_cast<size_t>(n) * n;
  double* yvec = ysmem ? reinterpret_cast<double*>(smem + L.yvec) : w.ws64 + static_cast<size_t>(wk) * 2 * nn;
  const size_t vplane = static_cast<size_t>(nb) * 64;

  for (int k = tid; k < kSfmtN32; k += NT) sf[k] = w.sfmt[static_cast<size_t>(wk) * kSfmtN32 + k];
  for (int k = tid; k < n; k += NT) idx[k] = w.ele_idx[static_cast<size_t>(wk) * n + k];
  for (int k = tid; k < m.ns2; k += NT) {
    cfg[k] = w.ele_cfg[static_cast<size_t>(wk) * m.ns2 + k];
    num[k] = w.ele_num[static_cast<size_t>(wk) * m.ns2 + k];
  }
  for (int k = tid; k < nqp; k += NT) qpw[k] = m.qpw[k];
  Rng rng{sf, w.sfmt_idx[wk], w.draws[wk]};  // kept by warp 0
  const FastMod by_ne(ne), by_ns(ns);
  if (tid == 0) ctl[5] = w.burn[wk];
  __syncthreads();
  bool burn = ctl[5] != 0;

  // CalculateMAll of the planes in `mask`; returns 0 or the first failing plane's status
  auto calc_m_all = [&](unsigned long long mask) {
    __syncthreads();
    auto fill = [&](int q, int w0, int nw) {
      const double* sl = m.slater + static_cast<size_t>(q) * m.ns2 * m.ns2;
      tri_fill(tiles + q * plane, n, w0, nw, [&](int i, int j) {
        return __ldg(sl + static_cast<size_t>(idx[i] + (i >= ne ? ns : 0)) * m.ns2 + idx[j] + (j >= ne ? ns : 0));
      });
    };
    int* first = ctl + 4;
    if (tid == 0) *first = 0x7fffffff;
    __syncthreads();
    const size_t pan_stride = al16(sizeof(double) * tri_pan_doubles(n) + kTriRedBytes);
    for (int q = kWarpSweep ? warp : 0; q < nqp; q += kWarpSweep ? NW : 1) {
      if (q < 64 && !((mask >> q) & 1ull)) continue;
      double pfv;
      int st;
      double* pan = reinterpret_cast<double*>(smem + L.vec + (kWarpSweep ? warp * pan_stride : 0));
      unsigned char* red = reinterpret_cast<unsigned char*>(pan + tri_pan_doubles(n));
      if constexpr (kWarpSweep) {
        fill(q, 0, 1);
        __syncwarp();
        tri_sweep<32, 32, CPT>(tiles + q * plane, pan, red, n, pfv, st);
      } else {
        fill(q, warp, NW);
        tri_sweep<NT, PG, CPT>(tiles + q * plane, pan, red, n, pfv, st);
      }
      if ((kWarpSweep ? lane : tid) == 0) {
        if (st == 0) pf[q] = pfv;
        else atomicMin(first, (q << 16) | (st < 0 ? 0xffff : st));  // lowest plane wins
      }
    }
    __syncthreads();
    const int f = *first;
    __syncthreads();
    return f == 0x7fffffff ? 0 : ((f & 0xffff) == 0xffff ? -1 : f & 0xffff);
  };
  auto log_ip = [&]() {
    if (tid == 0) dctl[0] = log_ip_of(m, pf, qpw);
    __syncthreads();
  };
  // makeInitialSample with the C retry rule
  auto initial = [&]() {
    for (int attempt = 1; attempt <= 101; ++attempt) {
      if (tid == 0) {
        SfmtRef ref{sf, &rng.idx, &rng.draws};
        make_initial_sample_dev(m, ref, idx, cfg, num, cnt);
      }
      if (warp == 0) {
        rng.idx = __shfl_sync(0xffffffffu, rng.idx, 0);
        rng.draws = __shfl_sync(0xffffffffu, rng.draws, 0);
      }
      const int info = calc_m_all(~0ull);
      if (attempt > 100) {
        if (tid == 0) atomicOr(w.status, kDevInitLoops);
        return;
      }
      if (info <= 0) return;
    }
  };
  if (!burn) initial();
  else calc_m_all(~0ull);
  log_ip();
  if (!isfinite(dctl[0])) {
    __syncthreads();
    initial();
    log_ip();
    burn = false;
  }
  const int S = m.saved;
  const int n_out = burn ? S + 1 : m.warmup + S;
  const long long n_in = static_cast<long long>(m.interval) * max(1, ns);
  int n_acc_win = 0;
  WalkerStats& stats = *reinterpret_cast<WalkerStats*>(smem + L.stats);
  if (tid == 0) stats = WalkerStats{};
  const bool timing = w.timers != nullptr && tid == 0;
  unsigned long long t_last = timing ? clock64() : 0ull;
  const unsigned long long t_begin = t_last;
  auto lap = [&](int phase) {
    if (timing) {
      const unsigned long long t = clock64();
      stats.ph[phase] += t - t_last;
      t_last = t;
    }
  };

  for (int out = 0; out < n_out; ++out) {
    long long step = 0;
    auto draw = [&](long long left) {  // warp 0
      const int got = draw_window(m, by_ne, by_ns, rng, idx, cfg, num, slots, static_cast<int>(min(left, 64ll)), w.status);
      if (lane == 0) ctl[0] = got;
    };
    if (warp == 0 && n_in > 0) draw(n_in);
    __syncthreads();
    while (step < n_in) {
      const int ns_batch = ctl[0];
      lap(kPhCandidate);
      // The batch's vectors: column(s) of slot u hold the Slater row(s) of the moved electron(s)
      // against the moved configuration; unused columns are zero. The upper half of the warps
      // gathers them; the lower half forms the hops' Δ ln P and fetches the exchanges' old pair
      // elements (update), two more chains of L2 latency.
      constexpr int NG = NW >= 8 ? NT / 2 : NT;  // gathering threads
      if (NW < 8 || tid < NT - NG) {
        for (int u = warp; u < ns_batch; u += NW - (NW >= 8 ? NG / 32 : 0))
          if (!slots[u].skip && slots[u].type == 0) {
            const double z = hop_dproj(m, num, slots[u]);
            if (lane == 0) slots[u].dproj = z;
          }
        for (int e = tid; e < ns_batch * nqp; e += NW >= 8 ? NT - NG : NT) {
          const int u = e / nqp, q = e - u * nqp;
          const Slot& s = slots[u];
          if (!s.skip && s.type == 1)
            sc[e * 8 + 3] = __ldg(m.slater + (static_cast<size_t>(q) * m.ns2 + s.ri + s.sp * ns) * m.ns2 + s.rj + s.t * ns);
        }
      }
      if (NW < 8 || tid >= NT - NG) {
        // a thread serves one column of every NG/8-th row, on all planes (eight loads in flight)
        const int gt = tid - (NT - NG), col = gt & 7;
        int us = -1, second = 0;
        for (int u = 0; u < ns_batch; ++u) {
          const int c = col - slots[u].col;
          if (!slots[u].skip && (c == 0 || (c == 1 && slots[u].type == 1))) {
            us = u;
            second = c;
          }
        }
        int msa = -1, msb = -1, ra = 0, rb = 0;
        if (us >= 0) {
          const Slot& s = slots[us];
          msa = s.msa;
          ra = s.rj + s.sp * ns;
          if (s.type == 1) {
            msb = s.msb;
            rb = s.ri + s.t * ns;
          }
        }
        const double* srow = m.slater + static_cast<size_t>(second ? rb : ra) * m.ns2;
        const size_t tab = static_cast<size_t>(m.ns2) * m.ns2;
        for (int i = gt >> 3; i < 8 * nb; i += NG / 8) {
          const bool on = us >= 0 && i < n;
          const int r = i == msa ? ra : (i == msb ? rb : (i < n ? idx[i] + (i >= ne ? ns : 0) : 0));
          const double* src = srow + r;
          double* dst = vec + i * 8 + col;
          int q = 0;
          for (; q + 8 <= nqp; q += 8) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = on ? __ldg(src + (q + k) * tab) : 0.0;
#pragma unroll
            for (int k = 0; k < 8; ++k) dst[(q + k) * vplane] = v[k];
          }
#pragma unroll 4
          for (; q < nqp; ++q) dst[q * vplane] = on ? __ldg(src + q * tab) : 0.0;
        }
      }
      __syncthreads();
      for (int unit = warp; unit < nqp * nb; unit += NW) {
        const int q = unit / nb, I = unit - q * nb;
        plane_row_product(tiles + q * plane, nb, I, vec + q * vplane, yvec + q * vplane, bpart + 4 * unit);
      }
      __syncthreads();
      lap(kPhRatio);
      if (warp == 0) {
        // Pfaffian ratios of every (slot, plane)
        for (int e = lane; e < ns_batch * nqp; e += 32) {
          const int u = e / nqp, q = e - u * nqp;
          const Slot& s = slots[u];
          if (s.skip) continue;
          const double* Y = yvec + q * vplane;
          const double* V = vec + q * vplane;
          const double* T = tiles + q * plane;
          double* o = sc + (u * nqp + q) * 8;
          const double pa = Y[s.msa * 8 + s.col];
          if (s.type == 0) {
            o[0] = pa;
            pfn[u * nqp + q] = -pa * pf[q];
          } else {
            const double pb = Y[s.msb * 8 + s.col], qa = Y[s.msa * 8 + s.col + 1], qb = Y[s.msb * 8 + s.col + 1];
            const double vba = V[s.msa * 8 + s.col + 1], vab = V[s.msb * 8 + s.col];
            const double iab = tri_get(T, nb, s.msa, s.msb);
            double bma = 0.0;
#pragma unroll 4
            for (int I = 0; I < nb; ++I) bma += bpart[4 * (q * nb + I) + (s.col >> 1)];
            const double ratio = iab * vba + iab * bma + pa * qb - pb * qa;
            // vs of the update is va but for entry msb, which holds the old pair's element
            const double delta = o[3] - vab;
            o[0] = pa; o[1] = pb; o[2] = qa; o[3] = delta; o[4] = bma; o[5] = iab; o[6] = vba; o[7] = qb;
            pfn[u * nqp + q] = ratio * pf[q];
          }
        }
        __syncwarp();
        // Metropolis: lane u decides slot u; the first acceptance in order counts
        double lip_new = 0.0;
        bool acc = false;
        if (lane < ns_batch && !slots[lane].skip) {
          double ip = 0.0;
          for (int q = 0; q < nqp; ++q) ip += qpw[q] * pfn[lane * nqp + q];
          lip_new = log(fabs(ip));
          double wgt = exp(2.0 * ((slots[lane].dproj + 0.0 + lip_new) - dctl[0]));
          if (!isfinite(wgt)) wgt = -1.0;
          acc = wgt > slots[lane].u;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, acc);
        const int hit = hits ? __ffs(hits) - 1 : -1;
        lip_new = __shfl_sync(0xffffffffu, lip_new, hit < 0 ? 0 : hit);
        const int used = hit < 0 ? ns_batch : hit + 1;
        const int my_type = lane < used ? slots[lane].type : 3;
        const unsigned hops = __ballot_sync(0xffffffffu, my_type == 0);
        const unsigned exchanges = __ballot_sync(0xffffffffu, my_type == 1);
        if (lane == 0) {
          stats.counter[0] += __popc(hops);
          stats.counter[2] += __popc(exchanges);
        }
        int refresh = 0;
        unsigned long long guard = 0ull;
        if (hit >= 0) {
          const Slot s = slots[hit];
          // the generator goes back to the word after this decision
          rng.draws -= static_cast<unsigned long long>(slots[ns_batch - 1].draws - s.draws);
          rng.idx = s.cursor;
          __syncwarp();
          if (lane == 0) {
            move_electron(m, idx, cfg, num, s.mi, s.ri, s.rj, s.sp);
            if (s.type == 1) move_electron(m, idx, cfg, num, s.mj, s.rj, s.ri, s.t);
            dctl[0] = lip_new;
            stats.counter[s.type == 0 ? 1 : 3]++;
          }
          ++n_acc_win;
          if (w.refresh_guard > 0.0)
            for (int q = 0; q < nqp; ++q) {
              const double r = fabs(pfn[hit * nqp + q] / pf[q]);
              if (!(r >= w.refresh_guard && r * w.refresh_guard <= 1.0)) guard |= q < 64 ? (1ull << q) : ~0ull;
            }
          if (n_acc_win > ns) {
            refresh = 1;  // C rule: recompute when the accept window exceeds Nsite
            n_acc_win = 0;
          }
          if (guard && !refresh) refresh = 3;
          if (lane == 0 && refresh == 3) stats.n_guard++;
          else if (lane == 0 && refresh) stats.n_sched++;
        }
        if (lane == 0) {
          reinterpret_cast<unsigned long long*>(dctl)[1] = refresh == 3 ? guard : ~0ull;
          ctl[1] = hit;
          ctl[2] = used;
          ctl[3] = refresh;
        }
        if (hit < 0 && step + used < n_in) draw(n_in - step - used);
      }
      __syncthreads();
      lap(kPhMetropolis);
      const int hit = ctl[1], refresh = ctl[3];
      step += ctl[2];
      if (hit < 0) continue;
      // the accepted move's four-column update, over the vectors
      {
        const Slot s = slots[hit];
        const int rows = 8 * nb;
        for (int k = tid; k < nqp * rows; k += NT) {
          const int q = k / rows, i = k - q * rows;
          const double* Y = yvec + q * vplane;
          const double* T = tiles + q * plane;
          const double* o = sc + (hit * nqp + q) * 8;
          double2 l0 = make_double2(0.0, 0.0), l1 = l0, r0 = l0, r1 = l0;
          if (i < n) {
            const double xa = tri_get(T, nb, s.msa, i), ya = Y[i * 8 + s.col];
            if (s.type == 0) {
              const double v2 = xa * (-1.0 / o[0]);
              const double v1 = ya + (i == s.msa ? 1.0 : 0.0);
              l0 = make_double2(v1, -v2);
              r0 = make_double2(v2, v1);
              if (i == 0) pf[q] *= -o[0];
            } else {
              const double pa = o[0], pb = o[1], qa = o[2], qb = o[7], delta = o[3], iab = o[5], vba = o[6];
              const double pam = pa + iab * delta, bma = o[4] - delta * qb;
              if (i == 0) pf[q] *= iab * vba + iab * bma + pam * qb - pb * qa;
              const double a = -pam, b = pb, c = qa, d = -qb, e = -bma - vba, f = iab;
              const double det = a * d - b * c - e * f, idet = 1.0 / det;
              const double edet = e * det, fidet = f * idet;
              const double xb = tri_get(T, nb, s.msb, i);
              const double si = idet * xa, ti = idet * xb, pi = ya - xb * delta, qi = Y[i * 8 + s.col + 1];
              double ct = a * qi + c * pi + edet * si, cs = b * qi + d * pi - edet * ti;
              double cq = fidet * pi - a * ti - b * si, cp = -(c * ti + d * si + fidet * qi);
              if (i == s.msa) {
                ct += c;
                cs += d;
                cq += fidet;
              }
              if (i == s.msb) {
                ct += a;
                cs += b;
                cp -= fidet;
              }
              l0 = make_double2(ct, cs);
              l1 = make_double2(cq, cp);
              r0 = make_double2(ti, si);
              r1 = make_double2(qi + (i == s.msb ? 1.0 : 0.0), pi + (i == s.msa ? 1.0 : 0.0));
            }
          }
          double2* l = reinterpret_cast<double2*>(vec + q * vplane) + i * 2;
          double2* r = l + rows * 2;
          l[0] = l0;
          l[1] = l1;
          r[0] = r0;
          r[1] = r1;
        }
      }
      __syncthreads();
      // the next batch's candidates beside the update (the slots are read no more)
      if (warp == 0 && step < n_in) draw(n_in - step);
      if constexpr (NW >= 8) {
        if (warp > 0) rank4_update(tiles, plane, vec, nqp, nb, warp - 1, NW - 1);
      } else {
        __syncwarp();
        rank4_update(tiles, plane, vec, nqp, nb, warp, NW);
      }
      __syncthreads();
      lap(kPhUpdate);
      if (refresh) {
        const int info = calc_m_all(reinterpret_cast<const unsigned long long*>(dctl)[1]);
        if (tid == 0 && info == 0) {
          // drift of the incrementally updated amplitude against the recomputation
          const double fresh = log_ip_of(m, pf, qpw);
          const double d = fabs(fresh - dctl[0]);
          if (isfinite(d) && d > stats.drift_max) stats.drift_max = d;
          dctl[0] = fresh;
        }
        __syncthreads();
        lap(kPhRefresh);
      }
    }
    if (out + S >= n_out) {
      make_proj_cnt_cta(m, m.jast_idx, num, cnt);
      const size_t sample = static_cast<size_t>(wk) * S + (out + S - n_out);
      for (int k = tid; k < n; k += NT) w.s_idx[sample * n + k] = idx[k];
      for (int k = tid; k < m.ns2; k += NT) {
        w.s_cfg[sample * m.ns2 + k] = cfg[k];
        w.s_num[sample * m.ns2 + k] = num[k];
      }
      for (int k = tid; k < m.nproj; k += NT) w.s_cnt[sample * m.nproj + k] = cnt[k];
      if (w.s_inv) {
        // resident measurement: this sample's Pf and X⁻¹ as the walker holds them
        double* dst = w.s_inv + sample * nqp * nn;
        for (int r = warp; r < nqp * n; r += NW) {
          const int q = r / n, i = r - q * n;
          for (int j = lane; j < n; j += 32) dst[static_cast<size_t>(r) * n + j] = tri_get(tiles + q * plane, nb, i, j);
        }
        for (int k = tid; k < nqp; k += NT) w.s_pf[sample * nqp + k] = pf[k];
      }
      __syncthreads();
    }
  }
  __syncthreads();
  make_proj_cnt_cta(m, m.jast_idx, num, cnt);
  for (int k = tid; k < kSfmtN32; k += NT) w.sfmt[static_cast<size_t>(wk) * kSfmtN32 + k] = sf[k];
  for (int k = tid; k < n; k += NT) w.ele_idx[static_cast<size_t>(wk) * n + k] = idx[k];
  for (int k = tid; k < m.ns2; k += NT) {
    w.ele_cfg[static_cast<size_t>(wk) * m.ns2 + k] = cfg[k];
    w.ele_num[static_cast<size_t>(wk) * m.ns2 + k] = num[k];
  }
  for (int k = tid; k < m.nproj; k += NT) w.proj_cnt[static_cast<size_t>(wk) * m.nproj + k] = cnt[k];
  for (int k = tid; k < nqp; k += NT) w.pf[static_cast<size_t>(wk) * nqp + k] = pf[k];
  if (tid == 0) {
    w.sfmt_idx[wk] = rng.idx;
    w.draws[wk] = rng.draws;
    w.burn[wk] = 1;
    for (int k = 0; k < 6; ++k) w.counter[static_cast<size_t>(wk) * 6 + k] = k < 4 ? stats.counter[k] : 0;
    if (w.drift) w.drift[wk] = stats.drift_max;
    if (w.nrefresh) {
      w.nrefresh[2 * static_cast<size_t>(wk)] = stats.n_sched;
      w.nrefresh[2 * static_cast<size_t>(wk) + 1] = stats.n_guard;
    }
    if (timing) {
      stats.ph[kPhTotal] = clock64() - t_begin;
      for (int k = 0; k < kPhCount; ++k) w.timers[static_cast<size_t>(wk) * kPhCount + k] = stats.ph[k];
    }
  }
}

struct TriSampPlan {
  int threads = 0;  // 0: not applicable
  bool warp_sweep = false, ysmem = false;
  size_t smem = 0;
};

// Threads per walker: 512 where one walker fills an SM or the walkers do not fill the SMs
// (2D 16×16: 203 KB of tiles);
// 256 or 128, two or four walkers per SM, where that many fit and there are as many: a batch
// is a chain of phases (candidates, vectors, products, decisions, update), and walkers beside
// each other fill each other's waits. Sides up to 32 with one plane always take 128.
TriSampPlan tri_samp_plan(const DevModel& m, int W, int precision, int limit) {
  TriSampPlan p;
  if (precision != 64 || m.n > 224 || m.n < 2 || m.nqp > 4096) return p;
  const int sms = current_device_attr(cudaDevAttrMultiProcessorCount);
  const int want = (W + sms - 1) / sms;  // walkers per SM
  const bool tiny = m.n <= 32 && m.nqp == 1;
  for (const int per_sm : {4, 2, 1}) {
    const int threads = 512 / per_sm;
    if (tiny ? per_sm != 4 : (per_sm > want || (per_sm == 4 && m.n > 64) || (per_sm == 2 && m.n > 128))) continue;
    const bool warp_sweep = m.n <= 64 && (m.nqp >= 4 || threads == 128);
    const int sweeps = warp_sweep ? std::min(threads / 32, m.nqp) : 1;
    for (const bool ysmem : {true, false}) {
      if (!ysmem && (per_sm > 1 || 8 * m.nqp * 8 * tri_blocks(m.n) > 2 * m.n * m.n)) continue;  // the walker's workspace
      const size_t total = tri_samp_layout(m, ysmem, sweeps).total;
      if (total > (static_cast<size_t>(limit) + 1024) / (tiny ? 1 : per_sm) - 1024) continue;
      p.threads = threads;
      p.warp_sweep = warp_sweep;
      p.ysmem = ysmem;
      p.smem = total;
      return p;
    }
  }
  return p;
}

template <int NT, int PG, int CPT>
int launch_tri(const DevModel& m, const DevWalkers& w, const TriSampPlan& p, cudaStream_t stream) {
  auto kernel = k_sample_tri<NT, PG, CPT>;
  MVMCB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(p.smem)));
  kernel<<<w.W, NT, p.smem, stream>>>(m, w, p.ysmem ? 1 : 0);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

}  // namespace

int residency_policy();

// FP64 walkers whose tiles and batch vectors fit one SM (MVMC_B200_RESIDENCY=global keeps the
// planes in L2).
bool sample_tri_applies(const DevModel& m, int precision, int limit) {
  return residency_policy() != 1 && tri_samp_plan(m, 1, precision, limit).threads != 0;
}

int launch_sample_tri(const DevModel& m, const DevWalkers& w, int precision, int limit, cudaStream_t stream) {
  const TriSampPlan p = tri_samp_plan(m, w.W, precision, limit);
  if (p.threads == 128 && m.n <= 32) return launch_tri<128, 32, 1>(m, w, p, stream);
  if (p.threads == 128) return launch_tri<128, 32, 2>(m, w, p, stream);
  if (p.threads == 256 && p.warp_sweep) return launch_tri<256, 32, 2>(m, w, p, stream);
  if (p.threads == 256) return launch_tri<256, 128, 1>(m, w, p, stream);
  if (p.threads == 512 && p.warp_sweep) return launch_tri<512, 32, 2>(m, w, p, stream);
  if (p.threads == 512) return launch_tri<512, 256, 1>(m, w, p, stream);
  return kErrArgument;
}

}  // namespace mvmcb
