// Explicit instantiation of the kernels with one group per thread (ncn_solo.cuh) for one group size (NCN_NG) and one
// direction (NCN_BWD defined or not).
#include "ncn_solo.cuh"

namespace ncn {

template <typename K>
static cudaError_t launch_kernel(K k, SmemGrant& granted, const SoloParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
  cudaError_t e = grant_smem(granted, k, smem);
  if (e != cudaSuccess) return e;
  if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, threads, smem);
  return launch_behind(k, dim3(grid), threads, smem, st, p);
}

template <int ACT, typename T>
static cudaError_t launch_one(const SoloParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
#ifdef NCN_BWD
  static SmemGrant granted[3];
#define NCN_GO(A) return launch_kernel(solo_bwd_kernel<NCN_NG, ACT, T, kSoloThreads, kSoloBwdBlocks, A>, granted[A], p, grid, threads, smem, st, occ)
  if (p.ahead == SOLO_AHEAD_OUTPUT) NCN_GO(SOLO_AHEAD_OUTPUT);
  if (p.ahead == SOLO_AHEAD_TAPE) NCN_GO(SOLO_AHEAD_TAPE);
  NCN_GO(SOLO_AHEAD_NONE);
#undef NCN_GO
#else
  static SmemGrant granted;
  return launch_kernel(solo_fwd_kernel<NCN_NG, ACT, T, kSoloThreads, kSoloFwdBlocks>, granted, p, grid, threads, smem, st, occ);
#endif
}

template <typename T>
static cudaError_t launch_act(int act, const SoloParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
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
#define NCN_FN NCN_CAT(launch_solo_bwd_n, NCN_NG)
#else
#define NCN_FN NCN_CAT(launch_solo_fwd_n, NCN_NG)
#endif

cudaError_t NCN_FN(int act, int dtype, const SoloParams& p, int grid, int threads, size_t smem, cudaStream_t st, int* occ) {
#if defined(NCN_BWD) && NCN_NG == 8
  if (dtype == DT_BF16) return cudaErrorNotSupported;  // the shared-memory kernels are faster there (solo_pays_n8)
#else
  if (dtype == DT_BF16) return launch_act<__nv_bfloat16>(act, p, grid, threads, smem, st, occ);
#endif
  return launch_act<float>(act, p, grid, threads, smem, st, occ);
}

}  // namespace ncn
