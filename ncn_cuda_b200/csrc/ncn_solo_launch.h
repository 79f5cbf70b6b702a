// Host-side entry points and parameter block of the kernels with one group per thread (ncn_solo.cuh).
#pragma once
#include "ncn_common.cuh"

namespace ncn {

struct SoloParams {
  const void* in[4];   // fwd: x, xa, -, - ; bwd: y, ya, dy, dya
  void* out[4];        // fwd: y, ya, -, - ; bwd: dx, dxa, x_rec (or null), xa_rec (or null)
  float* ckpt;         // [K][B*N] (x, a) pairs, [o m + g] per row, or null
  const float* W;      // [L][2]
  WeightList list;     // fwd: the weights one by one
  float* partials;     // bwd: [gridDim.x][L][2]
  int* status;         // device status word
  long long B;
  long long tiles;
  int N, m, R, L, l0, ckpt_every, n_ckpt, flags;
  float alpha, oma;
  uint32_t off_res, off_red, off_w, off_bar;  // byte offsets into dynamic shared memory; the tile buffer is at 0
  uint32_t off_land;   // bwd: buffer of the streams that are copied a tile ahead
  int ahead;           // bwd: SoloAhead
};

// Backward: what is fetched a tile ahead (solo_bwd_kernel): nothing; all four streams; with F_TAPE dy, dya and the state.
enum SoloAhead : int { SOLO_AHEAD_NONE = 0, SOLO_AHEAD_OUTPUT = 1, SOLO_AHEAD_TAPE = 2 };

constexpr int kSoloThreads = 512;  // block size the kernels are compiled for: backward one such CTA per SM, forward two
constexpr int kSoloFwdBlocks = 2, kSoloBwdBlocks = 1;

// With occ != nullptr nothing is launched: *occ receives the resident CTAs per SM.
#define NCN_DECL(n)                                                                                                       \
  cudaError_t launch_solo_fwd_n##n(int act, int dtype, const SoloParams& p, int grid, int threads, size_t smem,           \
                                   cudaStream_t st, int* occ);                                                            \
  cudaError_t launch_solo_bwd_n##n(int act, int dtype, const SoloParams& p, int grid, int threads, size_t smem,           \
                                   cudaStream_t st, int* occ);
NCN_DECL(8)
NCN_DECL(16)
#undef NCN_DECL

}  // namespace ncn
