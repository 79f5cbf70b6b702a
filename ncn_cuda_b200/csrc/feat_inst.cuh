// Explicit instantiation of the register-tiled multi-feature stage kernels (ncn_feat.cuh) for one
// n_cache (NCN_NC) and one direction (NCN_BWD defined or not); one translation unit each.
// Head widths d = 2, 4 (one lane per position), 8, 16, 32, 64, 128 (8 features per lane), 24, 48 (6 per lane), up to
// kFeatMaxRows rows of positions per group (n_cache * d <= 2048).  Every other shape stays with the shared-memory kernels
// of ncn_generic.cuh, and so do bf16 storage with context lengths and, where tanh.approx is the rule (feat_bf16_exact_tanh
// false), bf16 storage with the exact tanh.
#include "ncn_feat.cuh"

namespace ncn {

template <int LD, int KF, int W, int ACT, typename T>
static cudaError_t launch_one(const FeatParamsX& p, int grid, int threads, cudaStream_t st, int* occ) {
  auto go = [&](auto k, const auto& args) {
    if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, threads, 0);
    return launch_behind(k, dim3(grid), threads, 0, st, args);
  };
  constexpr int P = FeatGeom<NCN_NC, LD, KF, W>::P;
  constexpr bool SEVERAL = feat_groups_per_warp(NCN_NC, LD) > 1, BF16 = sizeof(T) != 4;
  const bool ctx = p.ctxlen != nullptr;
  if (ctx && BF16) return cudaErrorNotSupported;
#ifdef NCN_BWD
#define NCN_KERNEL feat_bwd_kernel
  const bool stored = p.saved == 3;
  constexpr bool OWN_PLAIN = feat_bwd_own(FM_PLAIN, NCN_NC, P, W, LD, BF16), OWN_STORED = feat_bwd_own(FM_STORED, NCN_NC, P, W, LD, BF16);
  if constexpr (NCN_NC >= 16) {
    if (p.saved == 1) return go(feat_bwd_kernel<NCN_NC, LD, KF, W, ACT, T, FM_REPLAY>, p);
  }
  if (p.saved != 0 && NCN_NC < 16) return cudaErrorNotSupported;
#else
#define NCN_KERNEL feat_fwd_kernel
  const bool stored = p.mid != nullptr;
  constexpr bool OWN_PLAIN = feat_fwd_own(FM_PLAIN, NCN_NC, P, W, LD, BF16), OWN_STORED = feat_fwd_own(FM_STORED, NCN_NC, P, W, LD, BF16);
  if (stored && NCN_NC < 16) return cudaErrorNotSupported;
#endif
  if constexpr (SEVERAL && !BF16) {
    if (ctx) return go(NCN_KERNEL<NCN_NC, LD, KF, W, ACT, T, FM_MASK>, p);
  }
  if constexpr (!SEVERAL && !BF16) {
    if (ctx && p.even) return go(NCN_KERNEL<NCN_NC, LD, KF, W, ACT, T, FM_CTX>, p);
  }
  if constexpr (OWN_PLAIN) {
    const FeatParams& plain = p;
    if (!ctx && !stored) return go(NCN_KERNEL<NCN_NC, LD, KF, W, ACT, T, FM_PLAIN>, plain);
  }
  if constexpr (OWN_STORED && NCN_NC >= 16) {
    if (!ctx && stored) return go(NCN_KERNEL<NCN_NC, LD, KF, W, ACT, T, FM_STORED>, p);
  }
  // what is left for the kernel with the branches, where anything is
  constexpr bool LEFT = !OWN_PLAIN || (!SEVERAL && !BF16) || (NCN_NC >= 16 && !OWN_STORED);
  if constexpr (LEFT) return go(NCN_KERNEL<NCN_NC, LD, KF, W, ACT, T, FM_ANY>, p);
  return cudaErrorNotSupported;
}

template <int LD, int KF, int W>
static cudaError_t launch_act(int act, int dtype, const FeatParamsX& p, int grid, int threads, cudaStream_t st, int* occ) {
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
static cudaError_t launch_geo(int team, int act, int dtype, const FeatParamsX& p, int grid, int threads, cudaStream_t st, int* occ) {
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

cudaError_t NCN_FN(int d, int team, int act, int dtype, const FeatParamsX& p, int grid, int threads, cudaStream_t st, int* occ) {
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
