// rhs_f64.cu -- double instantiations of the fused RHS kernel (orders 1..8,
// advection / Maxwell TM / Maxwell TE).
#include "rhs_launch.cuh"
#include "dg_rhs_eo.cuh"

namespace dgk {

// The even / odd kernel, or the node-by-node one for operators without the
// reflection symmetry (dgc_set_operators).
template <int N, int P>
static cudaError_t rhs_f64(const RhsParams& p, int sm, cudaStream_t s, LaunchInfo* info) {
  using C = EoConfig<double, N, P>;
  if (!info && !p.mats_eo) return rhs_launch<double, N, P>(p, sm, s);
  static std::once_flag once;
  static cudaError_t st = cudaSuccess;
  static int bps = 0;
  std::call_once(once, [] {
    st = cudaFuncSetAttribute(dg_rhs_eo_kernel<double, N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
    // one shared-memory carveout for all kernels that launch overlapped: a change
    // of it between two launches drains the SMs in between
    if (st == cudaSuccess)
      st = cudaFuncSetAttribute(dg_rhs_eo_kernel<double, N, P>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (st == cudaSuccess)
      st = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, dg_rhs_eo_kernel<double, N, P>, C::kThreads, C::kSmem);
  });
  if (st != cudaSuccess) return st;
  if (info) {
    info->threads = C::kThreads;
    info->tile = C::TE;
    info->smem = C::kSmem;
    info->blocks_per_sm = bps;
    return cudaSuccess;
  }
  const int ntiles = eo_tiles<double, N, P>(p.K, sm);
  // Overlapped launch only where the grid leaves SMs one CTA each: its prologue
  // then runs beside the previous stage (K = 2048, N = 4, advection: 6.0 us per
  // stage against 6.8 without).  A larger grid launched early is placed on the
  // SMs that have room at that moment, unevenly (K = 2048, N = 6, Maxwell TE:
  // 24.9 us against 17.3 launched plainly).
  if (ntiles <= sm) return launch_stage(dg_rhs_eo_kernel<double, N, P>, ntiles, C::kThreads, C::kSmem, s, p);
  dg_rhs_eo_kernel<double, N, P><<<ntiles, C::kThreads, C::kSmem, s>>>(p);
  return cudaGetLastError();
}

template <int N>
static cudaError_t by_phys(int P, const RhsParams& p, int sm, cudaStream_t s, LaunchInfo* info) {
  switch (P) {
    case PHYS_ADV: return rhs_f64<N, PHYS_ADV>(p, sm, s, info);
    case PHYS_TM: return rhs_f64<N, PHYS_TM>(p, sm, s, info);
    case PHYS_TE: return rhs_f64<N, PHYS_TE>(p, sm, s, info);
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t rhs_dispatch<double>(int N, int P, int v, const RhsParams& p, int sm, cudaStream_t s, LaunchInfo* info) {
  (void)v;
  switch (N) {
    case 1: return by_phys<1>(P, p, sm, s, info);
    case 2: return by_phys<2>(P, p, sm, s, info);
    case 3: return by_phys<3>(P, p, sm, s, info);
    case 4: return by_phys<4>(P, p, sm, s, info);
    case 5: return by_phys<5>(P, p, sm, s, info);
    case 6: return by_phys<6>(P, p, sm, s, info);
    case 7: return by_phys<7>(P, p, sm, s, info);
    case 8: return by_phys<8>(P, p, sm, s, info);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace dgk
