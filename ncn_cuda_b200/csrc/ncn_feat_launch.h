// Host-side entry points of the register-tiled multi-feature stage kernels (one per direction
// and n_cache).  With occ != nullptr nothing is launched: *occ receives the resident CTAs per SM.
// cudaErrorNotSupported: no kernel for this (n_cache, d, dtype, activation).
#pragma once
#include "ncn_common.cuh"

namespace ncn {

struct FeatParamsX;

constexpr int kFeatWarps = 4;  // warps per CTA

// Whether the groups of a padded batch are dealt out evenly (FeatUnits, ncn_feat.cuh).  Up to eight warps per SM have a group
// each, and the scan of the lengths only costs (32 x 256 x 128, 1024 groups: forward 24.7 -> 26.3 us); more than 1024 rows have
// enough groups per team to even out by themselves.  Between: 64 x 256 x 128 42 + 80 -> 34 + 48 us a stage, 128 rows 65 + 140 ->
// 56 + 103, 300 x 128 x 128, groups of 16 39 + 78 -> 32 + 62, 1000 x 96 x 64 87 + 162 -> 75 + 138.
constexpr int kFeatCtxRows = 1024;
inline bool feat_ctx_even(long long rows, long long groups, int sms) { return rows <= kFeatCtxRows && groups > 8LL * sms; }

// team: warps per group (feat_team)
#define NCN_DECL(n)                                                                                                   \
  cudaError_t launch_feat_fwd_n##n(int d, int team, int act, int dtype, const FeatParamsX& p, int grid, int threads,   \
                                   cudaStream_t st, int* occ);                                                        \
  cudaError_t launch_feat_bwd_n##n(int d, int team, int act, int dtype, const FeatParamsX& p, int grid, int threads,   \
                                   cudaStream_t st, int* occ);
NCN_DECL(2)
NCN_DECL(4)
NCN_DECL(8)
NCN_DECL(16)
NCN_DECL(32)
#undef NCN_DECL

// lanes that share a position of d features (8 features per lane, 6 for 24 and 48); 0: no kernel
constexpr int feat_lanes(int d) {
  switch (d) {
    case 2: case 4: case 8: return 1;
    case 16: return 2;
    case 24: case 32: return 4;
    case 48: case 64: return 8;
    case 128: return 16;
    default: return 0;
  }
}
// rows of 32 / lanes positions in a group of n; 0: no kernel
constexpr int feat_rows(int n, int lanes) { return lanes == 0 ? 0 : n * lanes <= 32 ? 1 : n * lanes / 32; }
// groups a warp works on side by side
constexpr int feat_groups_per_warp(int n, int lanes) { return n * lanes >= 32 ? 1 : 32 / (n * lanes); }

// bf16 storage: heads of 24 and 48 features and tiles of more than 1024 elements keep the exact tanh that the
// shared-memory kernels take; the other shapes take tanh.approx (relative error 2^-11), unless NCN_EXACT_TANH=1 sends them
// to the shared-memory kernels.  (64 x 256 x 128, groups of 32, replayed from the bf16 input: dW 8e-7 off the fp64 result of the
// same input for heads of 64, 3.5e-6 for heads of 32.)
constexpr bool feat_bf16_exact_tanh(int n, int d) { return d == 24 || d == 48 || n * d > 1024; }

// Warps per group.  The widest share (four rows per lane, as few warps as that takes) does the least work per element:
// the step's shared part is paid once per warp.  Larger teams shorten a step: taken while all groups' teams together
// leave the SMs at no more than this many warps.  Measured (us, start = one warp per group always; 256 tokens of 128
// features in 4 heads, groups of 32):  4 sequences forward 17.7 -> 13.4 (W = 4), backward 34.0 -> 21.8 (W = 4); 16
// sequences forward 19.5 -> 18.0 (W = 4), backward W = 4 40.1, W = 2 32.5, W = 1 36.2; 32 sequences (14 warps per SM with
// W = 2) backward W = 2 57, W = 1 50.
constexpr int kFeatMaxRows = 8;
constexpr int kFeatTeamFwd = 16, kFeatTeamBwd = 8;
constexpr int feat_team_min(int rows) { return rows <= 4 ? 1 : rows / 4; }
constexpr int feat_team_max(int rows) { return rows < kFeatWarps ? rows : kFeatWarps; }
// team sizes there are kernels for
constexpr bool feat_team_ok(int rows, bool bwd, int w) {
  if (w < feat_team_min(rows) || w > feat_team_max(rows)) return false;
  return bwd || w == feat_team_min(rows) || w == feat_team_max(rows);
}
inline int feat_team(int rows, bool bwd, long long groups, int sms) {
  for (int w = feat_team_max(rows); w > feat_team_min(rows); w /= 2)
    if (feat_team_ok(rows, bwd, w) && groups * w <= (long long)sms * (bwd ? kFeatTeamBwd : kFeatTeamFwd)) return w;
  return feat_team_min(rows);
}

}  // namespace ncn
