// Explicit instantiation of the register-tiled multi-feature stage kernels (ncn_feat.cuh) for one
// n_cache (NCN_NC) and one direction (NCN_BWD defined or not); one translation unit each.
// Head widths d = 2, 4 (one lane per position), 8, 16, 32, 64, 128 (8 features per lane), 24, 48 (6 per lane), up to
// kFeatMaxRows rows of positions per group (n_cache * d <= 2048).  Every other shape, and bf16 storage with the exact
// tanh, stays with the shared-memory kernels of ncn_generic.cuh.
#include "ncn_feat.cuh"

namespace ncn {

template <int LD, int KF, int W, int ACT, typename T>
static cudaError_t launch_one(const FeatParams& p, int grid, int threads, cudaStream_t st, int* occ) {
  auto go = [&](auto k) {
    if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, threads, 0);
    k<<<grid, threads, 0, st>>>(p);
    return cudaGetLastError();
  };
  constexpr bool SEVERAL = feat_groups_per_warp(NCN_NC, LD) > 1;
#ifdef NCN_BWD
  if constexpr (SEVERAL && sizeof(T) == 4) {
    if (p.ctxlen != nullptr) return go(feat_bwd_kernel<NCN_NC, LD, KF, W, ACT, T, false, true>);
  }
  if constexpr (NCN_NC >= 16) {
    if (p.saved == 1 || p.saved == 2) return go(feat_bwd_kernel<NCN_NC, LD, KF, W, ACT, T, true, false>);
  }
  if (p.saved != 0 && NCN_NC < 16) return cudaErrorNotSupported;
  if ((SEVERAL || sizeof(T) != 4) && p.ctxlen != nullptr) return cudaErrorNotSupported;
  return go(feat_bwd_kernel<NCN_NC, LD, KF, W, ACT, T, false, false>);
#else
  if constexpr (SEVERAL && sizeof(T) == 4) {
    if (p.ctxlen != nullptr) return go(feat_fwd_kernel<NCN_NC, LD, KF, W, ACT, T, true>);
  }
  if (p.mid != nullptr && NCN_NC < 16) return cudaErrorNotSupported;
  if ((SEVERAL || sizeof(T) != 4) && p.ctxlen != nullptr) return cudaErrorNotSupported;
  return go(feat_fwd_kernel<NCN_NC, LD, KF, W, ACT, T, false>);
#endif
}

template <int LD, int KF, int W>
static cudaError_t launch_act(int act, int dtype, const FeatParams& p, int grid, int threads, cudaStream_t st, int* occ) {
  if (dtype == DT_F32) {
    switch (act) {
      case ACT_TANH: return launch_one<LD, KF, W, ACT_TANH, float>(p, grid, threads, st, occ);
      case ACT_RELU: return launch_one<LD, KF, W, ACT_RELU, float>(p, grid, threads, st, occ);
      case ACT_SIGMOID: return launch_one<LD, KF, W, ACT_SIGMOID, float>(p, grid, threads, st, occ);
      case ACT_LINEAR: return launch_one<LD, KF, W, ACT_LINEAR, float>(p, grid, threads, st, occ);
      case ACT_LEAKY: return launch_one<LD, KF, W, ACT_LEAKY, float>(p, grid, threads, st, occ);
      default: return cudaErrorNotSupported;
    }
  }
  if constexpr (feat_bf16_exact_tanh(NCN_NC, LD * KF)) {
    if (act == ACT_TANH) return launch_one<LD, KF, W, ACT_TANH, __nv_bfloat16>(p, grid, threads, st, occ);
  } else {  // (the exact tanh, NCN_EXACT_TANH=1, stays with the shared-memory kernels)
    if (act == ACT_TANH_FAST) return launch_one<LD, KF, W, ACT_TANH_FAST, __nv_bfloat16>(p, grid, threads, st, occ);
  }
  switch (act) {
    case ACT_RELU: return launch_one<LD, KF, W, ACT_RELU, __nv_bfloat16>(p, grid, threads, st, occ);
    case ACT_SIGMOID: return launch_one<LD, KF, W, ACT_SIGMOID, __nv_bfloat16>(p, grid, threads, st, occ);
    case ACT_LINEAR: return launch_one<LD, KF, W, ACT_LINEAR, __nv_bfloat16>(p, grid, threads, st, occ);
    case ACT_LEAKY: return launch_one<LD, KF, W, ACT_LEAKY, __nv_bfloat16>(p, grid, threads, st, occ);
    default: return cudaErrorNotSupported;
  }
}

template <int LD, int KF>
static cudaError_t launch_geo(int team, int act, int dtype, const FeatParams& p, int grid, int threads, cudaStream_t st, int* occ) {
#ifdef NCN_BWD
  constexpr bool BWD = true;
#else
  constexpr bool BWD = false;
#endif
  constexpr int ROWS = feat_rows(NCN_NC, LD);
  if constexpr (ROWS > kFeatMaxRows) {
    return cudaErrorNotSupported;
  } else {
    // (the branches of team sizes without a kernel instantiate the smallest one)
    constexpr int LEAST = feat_team_min(ROWS);
    if (!feat_team_ok(ROWS, BWD, team)) return cudaErrorNotSupported;
    if (team == 4) return launch_act<LD, KF, feat_team_ok(ROWS, BWD, 4) ? 4 : LEAST>(act, dtype, p, grid, threads, st, occ);
    if (team == 2) return launch_act<LD, KF, feat_team_ok(ROWS, BWD, 2) ? 2 : LEAST>(act, dtype, p, grid, threads, st, occ);
    return launch_act<LD, KF, LEAST>(act, dtype, p, grid, threads, st, occ);
  }
}

#define NCN_CAT2(a, b) a##b
#define NCN_CAT(a, b) NCN_CAT2(a, b)
#ifdef NCN_BWD
#define NCN_FN NCN_CAT(launch_feat_bwd_n, NCN_NC)
#else
#define NCN_FN NCN_CAT(launch_feat_fwd_n, NCN_NC)
#endif

cudaError_t NCN_FN(int d, int team, int act, int dtype, const FeatParams& p, int grid, int threads, cudaStream_t st, int* occ) {
  switch (d) {
    case 2: return launch_geo<1, 2>(team, act, dtype, p, grid, threads, st, occ);
    case 4: return launch_geo<1, 4>(team, act, dtype, p, grid, threads, st, occ);
    case 8: return launch_geo<1, 8>(team, act, dtype, p, grid, threads, st, occ);
    case 16: return launch_geo<2, 8>(team, act, dtype, p, grid, threads, st, occ);
    case 24: return launch_geo<4, 6>(team, act, dtype, p, grid, threads, st, occ);
    case 32: return launch_geo<4, 8>(team, act, dtype, p, grid, threads, st, occ);
    case 48: return launch_geo<8, 6>(team, act, dtype, p, grid, threads, st, occ);
    case 64: return launch_geo<8, 8>(team, act, dtype, p, grid, threads, st, occ);
    case 128: return launch_geo<16, 8>(team, act, dtype, p, grid, threads, st, occ);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace ncn
