// K2 on the host: residency and launch of the FP64 instances of k_sample (sampler_impl.cuh; the
// FP32 ones are in sampler_f32.cu), and one walker's Pfaffian stage.
#include "sampler_impl.cuh"

namespace mvmcb {

int launch_sample_f32(const DevModel& m, DevWalkers w, int limit, cudaStream_t stream);

// Shared-memory residency: planes (and for FP32 the FP64 refresh workspace) in shared
// memory when they fit the per-block opt-in limit.
int residency_policy();
// FP32 planes: several small QP planes (side ≤ 64) go to L2 with two walkers per SM, which
// overlap each other's serial phases (2D 8×8, eight planes of 64: 2.08 against 2.63 s per
// SR step with one walker per SM holding its planes in shared memory); one wide plane stays
// in shared memory (2D 16×16: 68.7 against 84.2 ms in L2).
bool fp32_prefers_l2(const DevModel& m) { return residency_policy() == 0 && m.nqp >= 4 && m.n <= 64; }
bool sample_planes_in_smem(const DevModel& m, int precision, int limit) {
  if (residency_policy() == 1) return false;
  if (precision == 32 && fp32_prefers_l2(m)) return false;
  if (precision == 32) return samp_layout<float>(m, true, true).total <= static_cast<size_t>(limit) ||
                              samp_layout<float>(m, true, false).total <= static_cast<size_t>(limit);
  return m.n <= 64 && samp_layout<double>(m, true, true).total <= static_cast<size_t>(limit);
}

// Plane residency: "shared" keeps a walker's planes in shared memory (one walker per SM
// when they are large), "global" keeps them in the walker's L2-resident slice so several
// walkers share an SM; "auto" (default) prefers shared memory. MVMC_B200_RESIDENCY selects.
int residency_policy() {
  static int policy = -1;
  if (policy < 0) {
    const char* v = std::getenv("MVMC_B200_RESIDENCY");
    policy = 0;
    if (v && std::strcmp(v, "global") == 0) policy = 1;
    if (v && std::strcmp(v, "shared") == 0) policy = 2;
  }
  return policy;
}

// Walkers resident per SM when planes are in L2 (MVMC_B200_WPS=k; 0 = as many as fit).
int walkers_per_sm() {
  static int k = -1;
  if (k < 0) {
    const char* v = std::getenv("MVMC_B200_WPS");
    k = v ? std::max(0, std::atoi(v)) : 0;
  }
  return k;
}

// CTA size for walkers whose planes are in L2 (MVMC_B200_THREADS=128|256|512; 0 = auto).
int global_threads() {
  static int nt = -1;
  if (nt < 0) {
    const char* v = std::getenv("MVMC_B200_THREADS");
    nt = (v && std::strcmp(v, "128") == 0) ? 128 : ((v && std::strcmp(v, "256") == 0) ? 256 : 0);
    if (v && std::strcmp(v, "512") == 0) nt = 512;
  }
  return nt;
}

template <int JPL>
int launch_sample_f64(const DevModel& m, const DevWalkers& w, int limit, cudaStream_t stream) {
  if (residency_policy() == 1) return launch_sample_global<double, JPL>(m, w, stream);
  // FP64 squares in shared memory: sides up to 64 with more planes than fit as tiles and batch
  // vectors (wider planes always fit as tiles when they fit as squares)
  if constexpr (JPL <= 2) {
    if (samp_layout<double>(m, true, true).total <= static_cast<size_t>(limit)) {
      if constexpr (JPL == 1) {
        // small planes (n ≤ 32): 128 threads per walker (1D L16: 1.95M vs 1.33M sweeps/s
        // with 512, whose barriers cost more than the work they split); MVMC_B200_SMEM_THREADS
        // = 64|128|256|512 overrides
        const char* e = std::getenv("MVMC_B200_SMEM_THREADS");
        const int nt = e ? std::atoi(e) : 128;
        if (nt == 64) return launch_sample_t<double, JPL, 64, true, true>(m, w, stream);
        if (nt == 128) return launch_sample_t<double, JPL, 128, true, true>(m, w, stream);
        if (nt == 256) return launch_sample_t<double, JPL, 256, true, true>(m, w, stream);
      }
      return launch_sample_t<double, JPL, 512, true, true>(m, w, stream);
    }
  }
  return launch_sample_global<double, JPL>(m, w, stream);
}

int launch_sample(const DevModel& m, const DevWalkers& w, int precision, cudaStream_t stream) {
  int dev = 0, limit = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (precision == 32) return launch_sample_f32(m, w, limit, stream);
  const int n = m.n;
  if (n <= 32) return launch_sample_f64<1>(m, w, limit, stream);
  if (n <= 64) return launch_sample_f64<2>(m, w, limit, stream);
  if (n <= 128) return launch_sample_f64<4>(m, w, limit, stream);
  if (n <= 224) return launch_sample_f64<7>(m, w, limit, stream);
  if (n <= 256) return launch_sample_f64<8>(m, w, limit, stream);
  return kErrArgument;
}

// ---- one walker's Pfaffian stage (RealPfStage, sampling/stage.rs:56-129) -----------------
// The five stage operations as single-CTA launches on FP64 planes held in global memory, for
// host-driven (teacher-forced) replay: the host owns the chain and passes the candidate
// configuration with every call; the device owns Pf and the inverses.
template <int JPL>
__global__ void __launch_bounds__(kStageThreads)
    k_stage(DevModel m, StageBufs b, int op, int msa, int msb, int rsa_old, int rsb_old, unsigned* status) {
  extern __shared__ __align__(16) unsigned char smem[];
  const SampLayout L = samp_layout<double>(m, false, false);
  WalkerSmem<double> s{};
  s.idx = reinterpret_cast<int*>(smem + L.idx);
  s.pf = reinterpret_cast<double*>(smem + L.pf);
  s.pfn = reinterpret_cast<double*>(smem + L.pfn);
  s.qpw = reinterpret_cast<double*>(smem + L.qpw);
  s.jidx = m.jast_idx;
  s.vec = reinterpret_cast<double*>(smem + L.vec);
  s.pscal = reinterpret_cast<double*>(smem + L.vec + sizeof(double) * 4 * static_cast<size_t>(m.nqp) * m.n);
  s.gj = gj_carve<double>(smem + L.gj, m.n);
  const size_t nn = static_cast<size_t>(m.n) * m.n;
  s.ws = b.ws;
  s.ws2 = b.ws + nn;
  s.planes = b.planes;
  const int tid = threadIdx.x;
  for (int k = tid; k < m.n; k += blockDim.x) s.idx[k] = b.idx[k];
  for (int k = tid; k < m.nqp; k += blockDim.x) {
    s.pf[k] = b.pf[k];
    s.pfn[k] = b.pfn[k];
    s.qpw[k] = m.qpw[k];
  }
  __syncthreads();
  if (op == kStageRecompute) {
    const int info = calc_m_all_dev<double, JPL, false, false>(m, s, status);
    if (tid == 0) b.info[0] = info;
  } else if (op == kStageProposeHop) {
    ratio_hop_dev<double>(m, s, msa);
  } else if (op == kStageAcceptHop) {
    update_hop_dev<double, JPL>(m, s, msa, false);
  } else if (op == kStageProposeExchange) {
    ratio_exchange_dev<double, JPL>(m, s, msa, msb);
  } else if (op == kStageAcceptExchange) {
    update_exchange_dev<double, JPL>(m, s, msa, msb, rsa_old, rsb_old, false);
  }
  __syncthreads();
  for (int k = tid; k < m.nqp; k += blockDim.x) {
    b.pf[k] = s.pf[k];
    b.pfn[k] = s.pfn[k];
  }
}

template <int JPL>
int launch_stage_jpl(const DevModel& m, const StageBufs& b, int op, int msa, int msb, int rsa_old, int rsb_old,
                     unsigned* status, cudaStream_t stream) {
  const size_t smem = samp_layout<double>(m, false, false).total;
  auto kernel = k_stage<JPL>;
  MVMCB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kernel<<<1, kStageThreads, smem, stream>>>(m, b, op, msa, msb, rsa_old, rsb_old, status);
  MVMCB_CUDA(cudaGetLastError());
  return kOk;
}

int launch_stage(const DevModel& m, const StageBufs& b, int op, int msa, int msb, int rsa_old, int rsb_old,
                 unsigned* status, cudaStream_t stream) {
  const int n = m.n;
  if (n <= 32) return launch_stage_jpl<1>(m, b, op, msa, msb, rsa_old, rsb_old, status, stream);
  if (n <= 64) return launch_stage_jpl<2>(m, b, op, msa, msb, rsa_old, rsb_old, status, stream);
  if (n <= 128) return launch_stage_jpl<4>(m, b, op, msa, msb, rsa_old, rsb_old, status, stream);
  if (n <= 224) return launch_stage_jpl<7>(m, b, op, msa, msb, rsa_old, rsb_old, status, stream);
  if (n <= 256) return launch_stage_jpl<8>(m, b, op, msa, msb, rsa_old, rsb_old, status, stream);
  return kErrArgument;
}

}  // namespace mvmcb
