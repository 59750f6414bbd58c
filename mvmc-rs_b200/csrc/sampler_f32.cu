// K2 in FP32 (the mixed path): residency and launch of the FP32 instances of k_sample
// (sampler_impl.cuh), and the FP64 planes a call starts from.
#include "sampler_impl.cuh"
#include "skewtile.cuh"

namespace mvmcb {

bool fp32_prefers_l2(const DevModel& m);

namespace {

constexpr int kPlaneThreads = 512;

// CalculateMAll of every walker's configuration before a call, one block per (walker, plane), for
// walkers beside whose FP32 planes no FP64 sweep buffer fits (2D 16×16: one plane of 224):
// the tile sweep in shared memory (skewtile.cuh), rounded to the FP32 square that k_sample
// loads. Left to k_sample the sweep ran in L2 with three barriers a pivot; at two sweeps per
// call it was a third of the call. Walkers without a configuration are skipped; a failed
// sweep leaves a non-finite Pf and k_sample repeats it.
__global__ void __launch_bounds__(kPlaneThreads, 1) k_planes_tri(DevModel m, DevWalkers w) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int wk = blockIdx.x / m.nqp, q = blockIdx.x - wk * m.nqp, n = m.n, ns = m.ns, ne = m.ne;
  if (w.burn[wk] == 0) return;
  double* T = reinterpret_cast<double*>(smem);
  double* pan = T + tri_tile_doubles(n);
  unsigned char* red = reinterpret_cast<unsigned char*>(pan + tri_pan_doubles(n));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* idx = w.ele_idx + static_cast<size_t>(wk) * n;
  const double* sl = m.slater + static_cast<size_t>(q) * m.ns2 * m.ns2;
  tri_fill(T, n, warp, kPlaneThreads / 32, [&](int i, int j) {
    return __ldg(sl + static_cast<size_t>(idx[i] + (i >= ne ? ns : 0)) * m.ns2 + idx[j] + (j >= ne ? ns : 0));
  });
  double pfv;
  int st;
  tri_sweep<kPlaneThreads, 256, 1>(T, pan, red, n, pfv, st);
  float* dst = reinterpret_cast<float*>(w.ws64 + static_cast<size_t>(wk) * 2 * n * n) + static_cast<size_t>(q) * n * n;
  const int nb = tri_blocks(n);
  for (int i = warp; i < n; i += kPlaneThreads / 32)
    for (int j = lane; j < n; j += 32) dst[i * n + j] = static_cast<float>(tri_get(T, nb, i, j));
  if (threadIdx.x == 0)
    w.pf[static_cast<size_t>(wk) * m.nqp + q] = st == 0 ? pfv : __longlong_as_double(0x7ff8000000000000ll);
}

int launch_planes_tri(const DevModel& m, const DevWalkers& w, cudaStream_t stream) {
  const size_t smem = sizeof(double) * (tri_tile_doubles(m.n) + tri_pan_doubles(m.n)) + kTriRedBytes;
  MVMCB_CUDA(cudaFuncSetAttribute(k_planes_tri, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  k_planes_tri<<<w.W * m.nqp, kPlaneThreads, smem, stream>>>(m, w);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

template <int JPL>
int launch_jpl(const DevModel& m, DevWalkers w, int limit, cudaStream_t stream) {
  if (residency_policy() == 1 || fp32_prefers_l2(m)) return launch_sample_global<float, JPL>(m, w, stream);
  if (samp_layout<float>(m, true, true).total <= static_cast<size_t>(limit)) {
    if constexpr (JPL == 1) {
      // small planes: 128 threads per walker, as for FP64
      const char* e = std::getenv("MVMC_B200_SMEM_THREADS");
      if (!e || std::atoi(e) == 128) return launch_sample_t<float, JPL, 128, true, true>(m, w, stream);
    }
    return launch_sample_t<float, JPL, 512, true, true>(m, w, stream);
  }
  if (samp_layout<float>(m, true, false).total > static_cast<size_t>(limit))
    return launch_sample_global<float, JPL>(m, w, stream);
  // FP32 planes in shared memory without room for the FP64 sweep: the call's first planes from
  // k_planes_tri where the tiles fit (n ≤ 224) and the planes the walker's slice of ws64
  if (m.n > 64 && m.n <= 224 && m.nqp <= 4) {
    const int rc = launch_planes_tri(m, w, stream);
    if (rc != kOk) return rc;
    w.preset = true;
  }
  return launch_sample_t<float, JPL, 512, true, false>(m, w, stream);
}

}  // namespace

int launch_sample_f32(const DevModel& m, DevWalkers w, int limit, cudaStream_t stream) {
  const int n = m.n;
  if (n <= 32) return launch_jpl<1>(m, w, limit, stream);
  if (n <= 64) return launch_jpl<2>(m, w, limit, stream);
  if (n <= 128) return launch_jpl<4>(m, w, limit, stream);
  if (n <= 224) return launch_jpl<7>(m, w, limit, stream);
  if (n <= 256) return launch_jpl<8>(m, w, limit, stream);
  return kErrArgument;
}

}  // namespace mvmcb
