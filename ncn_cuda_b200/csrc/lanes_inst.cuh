// Explicit instantiation of the register-resident row kernels (ncn_lanes.cuh) for one group size
// (NCN_NG) and one direction (NCN_BWD defined or not).
#include "ncn_lanes_pipe.cuh"

namespace ncn {

template <int ACT, typename T, bool RAG, int AHEAD = LANE_AHEAD_NONE>
static cudaError_t launch_form(const LaneParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
#ifdef NCN_BWD
  auto k = lane_bwd_kernel<NCN_NG, ACT, T, kLaneMaxThreads, kLaneBwdBlocks * kLaneThreads / kLaneMaxThreads, AHEAD, RAG>;
#else
  auto k = lane_fwd_kernel<NCN_NG, ACT, T, kLaneMaxThreads, kLaneFwdBlocks * kLaneThreads / kLaneMaxThreads, RAG>;
#endif
  static SmemGrant granted;
  cudaError_t e = grant_smem(granted, k, smem);
  if (e != cudaSuccess) return e;
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, threads, smem);
  return launch_behind(k, dim3(grid), threads, smem, st, p);
}

template <int ACT, typename T>
static cudaError_t launch_one(const LaneParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
#ifdef NCN_BWD
#if NCN_NG == 4
  if (p.pipelined) {  // two half-rows per thread, half a stage apart (ncn_lanes_pipe.cuh)
    static SmemGrant granted_p[5];
    auto go = [&](auto kp, SmemGrant& granted) {
      cudaError_t ep = grant_smem(granted, kp, smem);
      if (ep != cudaSuccess) return ep;
      if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kp, threads, smem);
      return launch_behind(kp, dim3(grid), threads, smem, st, p);
    };
#define NCN_PIPE(A) go(lanep_bwd_kernel<NCN_NG, ACT, T, kLaneMaxThreads, kLaneBwdBlocks * kLaneThreads / kLaneMaxThreads, A>, granted_p[A])
    switch (p.ahead) {
      case LANE_AHEAD_OUTPUT: return NCN_PIPE(LANE_AHEAD_OUTPUT);
      case LANE_AHEAD_TAPE: return NCN_PIPE(LANE_AHEAD_TAPE);
      case LANE_AHEAD_TAPES: return NCN_PIPE(LANE_AHEAD_TAPES);
      case LANE_STATES_GLOBAL: return NCN_PIPE(LANE_STATES_GLOBAL);
      default: return NCN_PIPE(LANE_AHEAD_NONE);
    }
#undef NCN_PIPE
  }
#endif
#else
#if NCN_NG == 4
  if (p.pipelined) {  // (A/B runs only: measured slower than lane_fwd_kernel)
    auto kp = lanep_fwd_kernel<NCN_NG, ACT, T, kLaneMaxThreads, kLaneBwdBlocks * kLaneThreads / kLaneMaxThreads>;
    static SmemGrant granted_pf;
    cudaError_t ep = grant_smem(granted_pf, kp, smem);
    if (ep != cudaSuccess) return ep;
    if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kp, threads, smem);
    return launch_behind(kp, dim3(grid), threads, smem, st, p);
  }
#endif
#endif
#ifdef NCN_BWD
#define NCN_AHEAD(A, OK)                                                                                \
  if (p.ahead == A) {                                                                                   \
    if (!p.ragged) return launch_form<ACT, T, false, A>(p, grid, threads, smem, st, occ);                \
    if constexpr (OK) return launch_form<ACT, T, true, A>(p, grid, threads, smem, st, occ);              \
    return cudaErrorNotSupported;                                                                       \
  }
  NCN_AHEAD(LANE_AHEAD_OUTPUT, true)
  NCN_AHEAD(LANE_AHEAD_TAPE, lane_ahead_tape(NCN_NG, true))
  NCN_AHEAD(LANE_AHEAD_TAPES, lane_ahead_tape(NCN_NG, true))
#undef NCN_AHEAD
#endif
  return p.ragged ? launch_form<ACT, T, true>(p, grid, threads, smem, st, occ) : launch_form<ACT, T, false>(p, grid, threads, smem, st, occ);
}

template <typename T>
static cudaError_t launch_act(int act, const LaneParams& p, int grid, int threads, size_t smem, cudaStream_t st,
                              int* occ) {
  if constexpr (sizeof(T) == 2) {  // bf16 storage only
    if (act == ACT_TANH_FAST) return launch_one<ACT_TANH_FAST, T>(p, grid, threads, smem, st, occ);
  }
  switch (act) {
    case ACT_TANH: return launch_one<ACT_TANH, T>(p, grid, threads, smem, st, occ);
    case ACT_RELU: return launch_one<ACT_RELU, T>(p, grid, threads, smem, st, occ);
    case ACT_SIGMOID: return launch_one<ACT_SIGMOID, T>(p, grid, threads, smem, st, occ);
    default: return launch_one<ACT_LINEAR, T>(p, grid, threads, smem, st, occ);
  }
}

#define NCN_CAT2(a, b) a##b
#define NCN_CAT(a, b) NCN_CAT2(a, b)
#ifdef NCN_BWD
#define NCN_FN NCN_CAT(launch_lane_bwd_n, NCN_NG)
#else
#define NCN_FN NCN_CAT(launch_lane_fwd_n, NCN_NG)
#endif

cudaError_t NCN_FN(int act, int dtype, const LaneParams& p, int grid, int threads, size_t smem, cudaStream_t st,
                   int* occ) {
  if (dtype == DT_BF16) return launch_act<__nv_bfloat16>(act, p, grid, threads, smem, st, occ);
  return launch_act<float>(act, p, grid, threads, smem, st, occ);
}

}  // namespace ncn
