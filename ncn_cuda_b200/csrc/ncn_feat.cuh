// Per-stage NCN kernels for several features per position (E > 1, heads of d = E / n_head
// features), with the whole group tile in registers.
//
// Behaviour replaced: ncn_cuda/ncn_fwd_cuda_kernel.cu:28-112 (forward_kernel) and
// ncn_cuda/ncn_bwd_cuda_kernel.cu:27-229 (backward_kernel), at the shapes the reference's own
// benchmark uses (grad_test_bench.py:22-28: E = 128, 4 heads, n_cache = 32); math as
// torch_ref/ncn_pytorch.py:74-94 (step) and torch_ref/ncn_pytorch_invertible.py:97-111, 164-172
// (inverse, gradient).
//
// A TEAM of W warps owns one group (or, with W = 1, several small ones) for all its n_cache steps:
//   lane = (slot, sub): LD = d / KF lanes share a position, each holding KF contiguous features;
//   the 32 / LD slots of a warp hold positions, P per lane; warp t of the team holds rows
//   t P .. t P + P-1, and position i = row * SEG + slot.
// Two things per step cross the lanes: the row x_j reaches everyone, and the backward's column sums
// (one value per feature) reach the lanes of position j.  Within a warp x_j goes by shuffles; between
// the warps of a team both go through a few hundred bytes of shared memory, double-buffered, behind ONE
// team barrier per step: the column sums of a step are picked up after the barrier of the next one,
// which is when H_j is needed first.
//
// What bounds them: with few groups (4 sequences = 128 groups of the reference's shape) the chain of
// instructions of a step, which a team of four warps shortens (4 x 256 x 128, groups of 32: forward
// 17.8 -> 13.4 us, backward 34 -> 22 us against one warp per group); with many groups the backward's four
// streams of 1024 elements leave room for two warps per scheduler (issue slots half busy), and smaller
// tiles per warp pay the step's shared part more often than their occupancy returns (see FeatTune).
#pragma once
#include <type_traits>

#include "ncn_common.cuh"
#include "ncn_feat_launch.h"

namespace ncn {

struct FeatParams {
  const void* in[4];  // fwd: x, xa ; bwd: y, ya, dy, dya
  void* out[4];       // fwd: y, ya ; bwd: dx, dxa, x_rec|null, xa_rec|null
  const float* W;     // [2E]
  float* partials;    // bwd: [gridDim.x][2E]
  long long B;
  long long units;    // B * mg work units per head
  int N, E, C, m, mg, stride;  // mg = ceil(m / groups per team)
  float alpha, oma;
};
// What the kernels beyond the plain call take as well.
struct FeatParamsX : FeatParams {
  const int* ctxlen;  // [B] context length per batch row, or null
  int even;           // with ctxlen: the groups that take steps are dealt out evenly (FM_CTX)
  const void* xin[2]; // bwd with the stage input saved: x, xa
  float* mid;         // fp32 states after every 16th step: state k, stream s at mid + (2k + s) * bne, in the
                      // element order of the activations (fwd: written if not null; bwd with saved == 3: read)
  long long bne;      // elements per activation tensor
  int saved;          // bwd: 1 = the first half of the steps is replayed from the saved input, with bf16 storage all
                      // steps are (y, ya are not read); 3 = the states the forward stored in `mid` replace the
                      // rebuilt ones
  int mid_end;        // the state after the LAST step is stored / read as well (bf16 storage: y, ya are not read)
};
enum FeatMode : int {
  FM_ANY,     // context lengths and stored states where the parameters have them (a run-time test)
  FM_PLAIN,   // neither
  FM_STORED,  // stored states
  FM_REPLAY,  // backward: states replayed from the saved stage input
  FM_MASK,    // context lengths, groups with different numbers of steps side by side in a warp
  FM_CTX      // context lengths, one group per team at a time, the groups that take steps dealt out evenly (FeatUnits)
};
template <int MODE>
using FeatArgs = std::conditional_t<MODE == FM_PLAIN, FeatParams, FeatParamsX>;

template <int NC, int LD, int KF, int W>
struct FeatGeom {
  static_assert(KF % 2 == 0 && 32 % LD == 0, "features are processed in pairs");
  static constexpr int D = LD * KF;
  static constexpr int SLOTS = 32 / LD;
  static constexpr int ROWS = NC >= SLOTS ? NC / SLOTS : 1;  // rows of SLOTS positions in a group
  static constexpr int P = ROWS / W;                         // positions per lane
  static constexpr int SEG = NC >= SLOTS ? SLOTS : NC;       // slots of one group
  static constexpr int GPW = SLOTS / SEG;                    // groups per warp (1 unless W = 1)
  static constexpr int KP = KF / 2;
  static constexpr int XS = GPW * D;                         // floats of one x_j buffer
  static constexpr int TEAMS = kFeatWarps / W;
  static_assert(ROWS * SEG == NC, "n_cache must be a power of two");
  static_assert(P * W == ROWS && kFeatWarps % W == 0, "the team divides the rows");
};

// CTAs per SM the register budget is set for.  Measured (us): backward of 1024 x 256 x 128, groups of 32: four rows per
// lane, two CTAs 1064; two rows per lane, three CTAs 1125, two CTAs 1269, four CTAs (spills) 1592.  1024 x 512 x 256, groups
// of 16 (two rows): forward with three CTAs 1188, four 1136.  2048 x 256 x 128, groups of 8 (one row): backward with three
// CTAs 766, four 702, five 950; forward with four CTAs 348, six 326.
template <int P>
struct FeatTune {
  static constexpr int fwd_blocks = P >= 4 ? 3 : P == 1 ? 6 : 4;
  static constexpr int bwd_blocks = P >= 4 ? 2 : P == 1 ? 4 : 3;
};
// One row per lane and few steps: the steps are unrolled, which makes the powers of the decay and the lane numbers
// constants; per step they cost as much as an element otherwise (2048 x 256 x 128, groups of 8, heads of 8: forward 396
// -> 377 us, backward 756 -> 706).  With several lanes per position the backward's body is too long for eight copies (heads
// of 32: 755 us against 700).
constexpr bool feat_unrolled(int n, int p, int w) { return p == 1 && w == 1 && n <= 8; }
constexpr bool feat_bwd_unrolled(int n, int p, int w, int lanes) { return feat_unrolled(n, p, w) && (n <= 4 || lanes == 1); }

// Which calls have a kernel of their own.  At these register counts a branch that is never taken costs 2 to 10 per cent
// (it is the schedule of the whole step loop that changes, not the branch), and now and then the kernel with the branches
// comes out better: taken is what measured faster (us, with the branches -> without).
//   forward, plain: bf16 1024 x 256 x 128, groups of 32 376 -> 366; 1024 x 512 x 256, groups of 16 855 -> 805; heads of 32,
//     groups of 8 248 -> 234, fp32 326 -> 323; one row per lane, fp32: heads of 8, groups of 16 173 -> 155.  But fp32,
//     several rows per lane: 530 -> 536 and 1138 -> 1162; heads of 8, groups of 8 (unrolled) 376 -> 385.
//   forward with stored states: one row per lane 325 -> 312 (heads of 8, groups of 32); four rows 540 -> 566.
//   backward, plain: bf16 2024 -> 1889 (groups of 16), 1023 -> 840 (groups of 32), fp32 2270 -> 2200; heads of 16, groups
//     of 16 (256 x 256 x 128) bf16 169 -> 158.  But fp32 unrolled: 703 -> 710.
//   backward with stored states: four rows 1070 -> 1033; two rows 575 -> 581, one row 668 -> 678.
// Small batches (teams of several warps) wait for the chain of a step; one kernel serves all their calls.
constexpr bool feat_fwd_own(int mode, int n, int p, int w, int lanes, bool bf16) {
  if (w > 1) return false;
  if (mode == FM_STORED) return p == 1;
  return bf16 || (p == 1 && (!feat_unrolled(n, p, w) || lanes >= 4));
}
constexpr bool feat_bwd_own(int mode, int n, int p, int w, int lanes, bool bf16) {
  return w == 1 && (mode == FM_STORED ? p >= 4 : bf16 || !feat_bwd_unrolled(n, p, w, lanes));
}

// Whether the decay of the two streams is carried as a power of m outside the steps.  It saves one instruction per
// element pair and stream, and costs a dozen per step and lane for the constants of the step: too many for one row per lane
// (forward, heads of 16, groups of 16, 256 x 256 x 128: 85 -> 80.5 us without; heads of 8, 1024 x 256 x 64: 161 -> 154.5),
// and too many registers for the four-row backward with the exact tanh (with the power it spills: stored states 1065 ->
// 1033 us without, replay 1374 -> 1317; heads of 64, groups of 16, 1024 x 256 x 128: 603 -> 551.  Plain with heads of 32 has
// room for it: 1029 against 1043; tanh.approx too: 840 against 881; and linear: 767 against 831).
// Groups of 2 and 4 save next to nothing by it, and the multiplications back to true scale cost them 10 per cent in accuracy.
constexpr bool feat_fwd_scaled(int mode, int n, int p, int w) {
  if (n <= 4) return false;
  return mode == FM_ANY || mode == FM_MASK || mode == FM_CTX || p > 1 || w > 1 || feat_unrolled(n, p, w);
}
constexpr bool feat_bwd_scaled(int mode, int n, int p, int w, int lanes, int act) {
  if (n <= 4) return false;
  const bool exact = act == ACT_TANH || act == ACT_SIGMOID;
  return !(exact && p >= 4 && w == 1 && mode != FM_ANY && mode != FM_CTX) || (mode == FM_PLAIN && lanes <= 4);
}
// Reciprocals of tanh / sigmoid that share one special-function reciprocal in the backward (act_r_all, ncn_common.cuh; 0 =
// one each; the forward takes four): context lengths, four rows (64 x 256 x 128): two 85 us, single 86.5; the kernels of
// their own 1040 -> 1030 with single ones (groups of 32), 1024 x 512 x 256, groups of 16 (two rows): 2346 -> 2279.
constexpr int feat_bwd_batch(int mode, int p, int w) { return p >= 4 && (w > 1 || mode == FM_ANY || mode == FM_CTX) ? 2 : 0; }
constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }

// m^k and m^-k: x = m^k X in the forward, x = m^-k X in the reverse sweep (k steps done), so that the
// decay of the two streams costs no instruction per element (as in ncn_common.cuh, but without the
// constant offsets, whose cancellation would cost accuracy over 32 steps).
// The powers are those of 0.9 itself, not of its fp32 value: that one is 2.6e-8 off, the same way in every step (8e-7 of
// the result after 32 steps, more than all roundings together).
struct FeatPowers {
  float pos[33], neg[33];
};
constexpr double kFeatM = 0.9, kFeatC = 0.1;
constexpr FeatPowers feat_powers() {
  FeatPowers t{};
  double a = 1.0, b = 1.0;
  for (int k = 0; k <= 32; ++k) {
    t.pos[k] = (float)a;
    t.neg[k] = (float)b;
    a *= kFeatM;
    b /= kFeatM;
  }
  return t;
}
static __constant__ FeatPowers kPow = feat_powers();

// Which group of which row a team's unit is.
template <bool EVEN>
struct FeatUnits {  // in order of rows and groups
  __device__ __forceinline__ void unit(long long u, int mg, long long& b, int& g) const {
    b = u / mg;
    g = (int)(u - b * mg);
  }
};
// FM_CTX.  A row's groups take steps up to its length and none beyond, so by row and group half of a padded batch's units cost
// nothing, and how many of the others a team gets is luck: of the 2048 groups of 64 x 256 x 128 (32 positions each) some of
// 1184 warps took two and many none (forward 42 us, backward 80 a stage; so: 34 and 48).  Here the units count the groups
// that take steps first, in row order, then the others: no team gets two of the former before all have one.  The counts come from a
// scan of the lengths in every CTA (feat_ctx_even says where it pays).
template <>
struct FeatUnits<true> {
  const int* pre;  // [B + 1]: groups that take steps in the rows before
  int rows, m, total;
  __device__ __forceinline__ void init(const int* ctxlen, int B, int m_, int n, int* pre_, int* warp_sum) {
    pre = pre_;
    rows = B;
    m = m_;
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
    const int per = (B + nthr - 1) / nthr, b0 = min(B, tid * per), b1 = min(B, b0 + per);
    auto groups = [&](int b) { return (int)min((long long)m_, max(0LL, ((long long)ctxlen[b] + n - 1) / n)); };
    int sum = 0;
    for (int b = b0; b < b1; ++b) sum += pre_[b] = groups(b);
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) warp_sum[tid >> 5] = inc;
    __syncthreads();
    int at = inc - sum;
    for (int w = 0; w < (tid >> 5); ++w) at += warp_sum[w];
    for (int b = b0; b < b1; ++b) {
      const int own = pre_[b];
      pre_[b] = at;
      at += own;
    }
    if (tid == nthr - 1) pre_[B] = at;
    __syncthreads();
    total = pre_[B];
  }
  __device__ __forceinline__ void unit(long long u, int, long long& b, int& g) const {
    const bool beyond = (int)u >= total;  // counts groups that take no steps: i m - pre[i] of them in the rows before i
    const int v = beyond ? (int)u - total : (int)u;
    int lo = 0, hi = rows;  // the last row that no more than v come before
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((beyond ? mid * m - pre[mid] : pre[mid]) <= v) lo = mid; else hi = mid;
    }
    b = lo;
    g = beyond ? pre[lo + 1] - pre[lo] + v - (lo * m - pre[lo]) : v - pre[lo];
  }
};

__device__ __forceinline__ float2 shfl2(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// sum over the LD lanes that share a position
template <int LD>
__device__ __forceinline__ float red_sub(float v) {
#pragma unroll
  for (int o = 1; o < LD; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// KF contiguous features.  Rows of 6 (d = 24, 48) start on 8-byte (bf16: 4-byte) boundaries only.
template <int KF, typename T>
__device__ __forceinline__ void ld_feat(const T* p, float2 (&v)[KF / 2]) {
  if constexpr (KF % 4 != 0) {
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) {
      float t[2];
      ld_vec<2>(p + 2 * q, t);
      v[q] = make_float2(t[0], t[1]);
    }
  } else {
    float t[KF];
    ld_vec<KF>(p, t);
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) v[q] = make_float2(t[2 * q], t[2 * q + 1]);
  }
}
template <int KF, typename T>
__device__ __forceinline__ void st_feat(T* p, const float2 (&v)[KF / 2]) {
  if constexpr (KF % 4 != 0) {
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) {
      const float t[2] = {v[q].x, v[q].y};
      st_vec<2>(p + 2 * q, t);
    }
  } else {
    float t[KF];
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) { t[2 * q] = v[q].x; t[2 * q + 1] = v[q].y; }
    st_vec<KF>(p, t);
  }
}
template <int KF>
__device__ __forceinline__ void st_feat_scaled(float* p, const float2 (&v)[KF / 2], float s) {
  float2 t[KF / 2];
#pragma unroll
  for (int q = 0; q < KF / 2; ++q) t[q] = __fmul2_rn(v[q], f2(s));
  st_feat<KF, float>(p, t);
}

template <int W>
__device__ __forceinline__ void team_sync(int team) {
  if constexpr (W == 1) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(W * 32) : "memory");
  }
}

// Position of a thread in the work split shared by both directions.  A team serves one head for the
// whole kernel, so the weights and the weight-gradient sums of a lane stay in registers.
template <typename G, int LD, int W>
struct FeatThread {
  int lane, warp, team, wt;  // wt: warp of the team
  int sub, gw, s;            // lane of the position, group of the warp, slot of the group
  int c;                     // head
  long long first, step;     // units
  __device__ __forceinline__ explicit FeatThread(const FeatParams& p) {
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    team = warp / W;
    wt = warp - team * W;
    sub = lane & (LD - 1);
    const int slot = lane / LD;
    gw = slot / G::SEG;
    s = slot - gw * G::SEG;
    const int tpc = (int)(blockDim.x >> 5) / W;
    const long long gt = (long long)blockIdx.x * tpc + team;
    const long long tt = (long long)gridDim.x * tpc;  // a multiple of C (launch plan)
    c = (int)(gt % p.C);
    first = gt / p.C;
    step = tt / p.C;
  }
  __device__ __forceinline__ int pos(int r) const { return (wt * G::P + r) * G::SEG + s; }  // position of row r
  // row index of step j inside a lane of the warp that owns it, -1 in the other warps of the team (ALONE: there are none)
  template <bool ALONE>
  __device__ __forceinline__ int local_row(int j) const {
    if (ALONE) return j / G::SEG;
    const int row = j / G::SEG - wt * G::P;
    return (unsigned)row < (unsigned)G::P ? row : -1;
  }
};

// r of the activation for the feature pairs of a position.  BATCH > 1: shared reciprocals.
template <int ACT, int KP, int BATCH>
__device__ __forceinline__ void feat_act(const float2 (&ts)[KP], float2 (&rr)[KP]) {
  if constexpr (KP >= 2 && BATCH > 1) {
    act_r_all<ACT, KP, BATCH>(ts, rr);
  } else {
#pragma unroll
    for (int q = 0; q < KP; ++q) rr[q] = ActForm<ACT>::r(ts[q]);
  }
}

// Shared-memory exchange of KF features.  Conditional accesses are single predicated instructions: written as
// branches they split the step's basic block, and the scheduler could not overlap what lies on either side
// (backward of a two-warp team 1195 -> 1126 us at 1024 x 256 x 128).
__device__ __forceinline__ void sts_if(bool on, uint32_t a, float2 v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\t@p st.shared.v2.f32 [%0], {%1, %2};\n\t}" ::"r"(a), "f"(v.x), "f"(v.y), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void sts_if(bool on, uint32_t a, float2 v, float2 w) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"r"(a), "f"(v.x), "f"(v.y),
               "f"(w.x), "f"(w.y), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void sts_if(bool on, uint32_t a, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(a), "f"(v), "r"((int)on) : "memory");
}
template <int KF>
__device__ __forceinline__ void sts_row_if(bool on, uint32_t a, const float2 (&v)[KF / 2]) {
  if constexpr (KF % 4 == 0) {
#pragma unroll
    for (int q = 0; q < KF / 2; q += 2) sts_if(on, a + 8u * q, v[q], v[q + 1]);
  } else {
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) sts_if(on, a + 8u * q, v[q]);
  }
}
template <int KF>
__device__ __forceinline__ void lds_row(uint32_t a, float2 (&v)[KF / 2]) {
  if constexpr (KF % 4 == 0) {
#pragma unroll
    for (int q = 0; q < KF / 2; q += 2)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q + 1].x), "=f"(v[q + 1].y)
                   : "r"(a + 8u * q)
                   : "memory");
  } else {
#pragma unroll
    for (int q = 0; q < KF / 2; ++q) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[q].x), "=f"(v[q].y) : "r"(a + 8u * q) : "memory");
  }
}
template <int KF>
__device__ __forceinline__ void lds_row_if(bool on, uint32_t a, float2 (&v)[KF / 2]) {  // v keeps its value where !on
  if constexpr (KF % 4 == 0) {
#pragma unroll
    for (int q = 0; q < KF / 2; q += 2)
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                   : "+f"(v[q].x), "+f"(v[q].y), "+f"(v[q + 1].x), "+f"(v[q + 1].y)
                   : "r"(a + 8u * q), "r"((int)on)
                   : "memory");
  } else {
#pragma unroll
    for (int q = 0; q < KF / 2; ++q)
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %3, 0;\n\t@p ld.shared.v2.f32 {%0, %1}, [%2];\n\t}"
                   : "+f"(v[q].x), "+f"(v[q].y)
                   : "r"(a + 8u * q), "r"((int)on)
                   : "memory");
  }
}

// The lanes of position j hand its row to the team.
template <int P, int KP, int KF>
__device__ __forceinline__ void publish_row(uint32_t dst, const float2 (&X)[P][KP], int rj, bool mine) {
  float2 v[KP];
#pragma unroll
  for (int q = 0; q < KP; ++q) {
    v[q] = X[0][q];
#pragma unroll
    for (int r = 1; r < P; ++r)
      if (rj == r) v[q] = X[r][q];
  }
  sts_row_if<KF>(mine, dst, v);
}
// The same as a branch: the forward is short of issue slots rather than of overlap, and the selects of four rows cost
// more than the branch (1024 x 256 x 128, groups of 32: 540 against 571 us).
template <int P, int KP, int KF>
__device__ __forceinline__ void publish_row_branch(float* dst, const float2 (&X)[P][KP], int rj, bool mine) {
  if (mine) {
#pragma unroll
    for (int r = 0; r < P; ++r)
      if (rj == r) st_feat<KF, float>(dst, X[r]);
  }
}

// One forward step (k = steps done; SC: x = m^k X, a = m^k A): xj is the row of position j in the same scale.
//   Ts = sT (alpha x_i + sim_i x_j) ;  SC: A <- A + c m^-(k+1) F ;  X <- X + c A, else a <- m a + c F ;  x <- m x + c a
template <int LD, int KP, int P, int ACT, bool MASK, bool SC>
__device__ __forceinline__ void feat_forward_step(float2 (&X)[P][KP], float2 (&A)[P][KP], const float2 (&xj)[KP],
                                                  const float2 (&Wi)[KP], const float2 (&Wj)[KP], float alpha, int k, bool on) {
  using F = ActForm<ACT>;
  constexpr float sT = (float)F::sT;
  const float mk = SC ? kPow.pos[k] : 1.0f, imk1 = SC ? kPow.neg[k + 1] : 1.0f;
  const float2 al = f2(alpha * sT * mk);
  const float ss = sT * mk * mk;
  const float2 c1 = f2((float)((SC ? kFeatC : kCd) * F::f1) * imk1);
  [[maybe_unused]] const float2 c0 = f2((float)((SC ? kFeatC : kCd) * F::f0) * imk1);
  float2 accj = f2(0.0f);
#pragma unroll
  for (int q = 0; q < KP; ++q) accj = __ffma2_rn(xj[q], Wj[q], accj);
  const float cj = accj.x + accj.y;
#pragma unroll
  for (int r = 0; r < P; ++r) {
    float2 acc = f2(0.0f);
#pragma unroll
    for (int q = 0; q < KP; ++q) acc = __ffma2_rn(X[r][q], Wi[q], acc);
    const float2 sim = f2(red_sub<LD>(acc.x + acc.y + cj) * ss);
    float2 ts[KP], rr[KP];
#pragma unroll
    for (int q = 0; q < KP; ++q) ts[q] = __ffma2_rn(sim, xj[q], __fmul2_rn(X[r][q], al));
    feat_act<ACT, KP, 4>(ts, rr);
    if (!MASK || on) {
#pragma unroll
      for (int q = 0; q < KP; ++q) {
        if constexpr (SC) {
          if constexpr (F::f0 != 0.0) A[r][q] = __fadd2_rn(A[r][q], c0);
          A[r][q] = __ffma2_rn(rr[q], c1, A[r][q]);
          X[r][q] = __ffma2_rn(A[r][q], f2(kC), X[r][q]);
        } else {
          A[r][q] = __ffma2_rn(rr[q], c1, __ffma2_rn(A[r][q], f2(kM), c0));
          X[r][q] = __ffma2_rn(A[r][q], f2(kC), __fmul2_rn(X[r][q], f2(kM)));
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ forward
// p.mid: the fp32 state after every 16th step is also written, for a backward whose inverse chains then
// never exceed 16 steps.  p.ctxlen: a group takes group_steps() steps.
template <int NC, int LD, int KF, int W, int ACT, typename T, int MODE>
__global__ void __launch_bounds__(kFeatWarps * 32, FeatTune<FeatGeom<NC, LD, KF, W>::P>::fwd_blocks) feat_fwd_kernel(const FeatArgs<MODE> p) {
  using G = FeatGeom<NC, LD, KF, W>;
  constexpr int P = G::P, KP = G::KP, SEG = G::SEG;
  constexpr bool MASK = MODE == FM_MASK, EVEN = MODE == FM_CTX, CTX = MASK || EVEN || (MODE == FM_ANY && G::GPW == 1);
  constexpr bool MID = NC >= 16 && (MODE == FM_ANY || MODE == FM_STORED);
  constexpr bool SC = feat_fwd_scaled(MODE, NC, P, W);
  __shared__ __align__(16) float xs[G::TEAMS][2][G::XS];
  wait_for_inputs();
  const FeatThread<G, LD, W> th(p);
  const T* gx = static_cast<const T*>(p.in[0]);
  const T* ga = static_cast<const T*>(p.in[1]);
  T* gy = static_cast<T*>(p.out[0]);
  T* gya = static_cast<T*>(p.out[1]);
  float* const xrow = &xs[th.team][0][th.gw * G::D + th.sub * KF];

  float2 Wi[KP], Wj[KP];  // (1 - alpha) folded in
  {
    const float* wi = p.W + th.c * G::D + th.sub * KF;
    const float* wj = wi + p.E;
#pragma unroll
    for (int q = 0; q < KP; ++q) {
      Wi[q] = make_float2(wi[2 * q] * p.oma, wi[2 * q + 1] * p.oma);
      Wj[q] = make_float2(wj[2 * q] * p.oma, wj[2 * q + 1] * p.oma);
    }
  }
  int shift[P];  // (i * stride) mod m
#pragma unroll
  for (int r = 0; r < P; ++r) shift[r] = (int)((long long)th.pos(r) * p.stride % p.m);
  int par = 0;

  __shared__ int rows_before[EVEN ? kFeatCtxRows + 1 : 1], warp_sum[kFeatWarps];
  FeatUnits<EVEN> units;
  if constexpr (EVEN) units.init(p.ctxlen, (int)p.B, p.m, NC, rows_before, warp_sum);
  for (long long u = th.first; u < p.units; u += th.step) {
    long long b;
    int g;
    units.unit(u, p.mg, b, g);
    g = g * G::GPW + th.gw;
    const bool valid = G::GPW == 1 || g < p.m;
    float2 X[P][KP], A[P][KP];
    long long off[P];
#pragma unroll
    for (int r = 0; r < P; ++r) {
      int blk = g + shift[r];
      if (blk >= p.m) blk -= p.m;
      off[r] = ((b * p.N + (long long)blk * NC + th.pos(r)) * p.E) + th.c * G::D + th.sub * KF;
      if (valid) {
        ld_feat<KF, T>(gx + off[r], X[r]);
        ld_feat<KF, T>(ga + off[r], A[r]);
      } else {
#pragma unroll
        for (int q = 0; q < KP; ++q) X[r][q] = A[r][q] = f2(0.0f);
      }
    }
    int steps = NC, tsteps = NC;  // of this lane's group, of the team
    if constexpr (CTX) {
      if (p.ctxlen != nullptr) {
        steps = valid ? group_steps(p.ctxlen, b, g, NC) : 0;
        tsteps = MASK ? (int)__reduce_max_sync(0xffffffffu, (unsigned)steps) : steps;
      }
    }
    auto run_step = [&](int j) {
      float2 xj[KP];
      // x_j by shuffles where several lanes share a position (2048 x 256 x 128, groups of 8: 4 heads 334 against 342 us
      // through shared memory; 16 heads, one lane per position, 420 against 387)
      if constexpr (W == 1 && P == 1 && LD > 1) {
        const int src = (th.gw * SEG + j) * LD + th.sub;
#pragma unroll
        for (int q = 0; q < KP; ++q) xj[q] = shfl2(X[0][q], src);
      } else {
        const int rj = th.template local_row<W == 1>(j);
        float* const xb = xrow + par * G::XS;
        par ^= 1;
        publish_row_branch<P, KP, KF>(xb, X, rj, rj >= 0 && th.s == (j & (SEG - 1)));
        team_sync<W>(th.team);
        ld_feat<KF, float>(xb, xj);
      }
      feat_forward_step<LD, KP, P, ACT, MASK, SC>(X, A, xj, Wi, Wj, p.alpha, j, j < steps);
      if constexpr (MID) {
        if (p.mid != nullptr && ((j + 1) & 15) == 0 && (j + 1 < NC || p.mid_end) && valid) {
          float* mx = p.mid + (long long)(2 * ((j + 1) / 16 - 1)) * p.bne;
          const float sc = SC ? kPow.pos[j + 1] : 1.0f;
#pragma unroll
          for (int r = 0; r < P; ++r) {
            st_feat_scaled<KF>(mx + off[r], X[r], sc);
            st_feat_scaled<KF>(mx + p.bne + off[r], A[r], sc);
          }
        }
      }
    };
    if constexpr (feat_unrolled(NC, P, W)) {
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        if (CTX && j >= tsteps) break;
        run_step(j);
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < tsteps; ++j) run_step(j);
    }
    if (valid) {
      const float2 sc = f2(kPow.pos[steps]);
#pragma unroll
      for (int r = 0; r < P; ++r) {
#pragma unroll
        for (int q = 0; q < KP && SC; ++q) {
          X[r][q] = __fmul2_rn(X[r][q], sc);
          A[r][q] = __fmul2_rn(A[r][q], sc);
        }
        st_feat<KF, T>(gy + off[r], X[r]);
        st_feat<KF, T>(gya + off[r], A[r]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ backward
// From the stage OUTPUT (y, ya) and the cotangents (dy, dya): every step first rebuilds its input
// by the reversible inverse, then applies the closed-form vector-Jacobian product.  Per step j and
// position i (features k; sums over k are the dot products):
//     x_i = (y_i - c ya_i) / m ;  sim_i = (1-alpha)(x_i.Wi + x_j.Wj) ;  T = alpha x_i + sim_i x_j
//     a_i = (ya_i - c F(T)) / m
//     gA' = ga + c gy ;  gT = c gA' act'(T) ;  ga <- m gA' ;  gs_i = (1-alpha) gT_i.x_j
//     gx_i = m gy_i + alpha gT_i + gs_i Wi
//     gx_j += Wj sum_i gs_i + sum_i sim_i gT_i          (position j in its role as x_j)
//     dWi += sum_i gs_i x_i ;  dWj += (sum_i gs_i) x_j
// With k inverse steps done x = m^-k X, a = m^-k A, gy = m^k H, ga = m^k Gv; in these variables the
// step is (q = m^-(k+1), gT = c ds m^k gt)
//     X <- X - c A ;  Ts = sT (alpha q X_i + q^2 (X_i.Wi + X_j.Wj) X_j) ;  A <- A - c m^k F
//     Gv <- Gv + c H ;  g_i = (c ds / m) q gt_i.X_j ;  H_i <- H_i + (alpha c ds / m) gt_i + g_i Wi
//     H_j += sum_i [ g_i Wj + (c ds / m) q (X_i.Wi + X_j.Wj) gt_i ] ;  dWi += g_i X_i ;  dWj += g_i X_j
// The weight gradient is summed per lane over all its groups, then over the slots of the warp
// (fixed shuffle tree), the warps of the CTA that serve the same head (warp order) and the CTAs
// (dw_reduce_kernel): a fixed order for a given launch shape.
//
// Without the power (SC false; see feat_bwd_scaled) X, A, H and Gv are the true values, and m is applied in the step.
//
// REPLAY (saved = 1): the caller also kept the stage INPUT.  Every inverse step grows earlier rounding
// by 1/m, so a chain of NC = 32 steps from the output alone leaves the gradients at 1e-5 of their size;
// here the state half way is rebuilt exactly by running the forward over the first NC/2 steps from the
// input, so that no inverse chain is longer than NC/2 steps.  With bf16 storage the
// end state is replayed too: an inverse started from rounded outputs would amplify their rounding.
template <int NC, int LD, int KF, int W, int ACT, typename T, int MODE>
__global__ void __launch_bounds__(kFeatWarps * 32, FeatTune<FeatGeom<NC, LD, KF, W>::P>::bwd_blocks) feat_bwd_kernel(const FeatArgs<MODE> p) {
  using G = FeatGeom<NC, LD, KF, W>;
  using F = ActForm<ACT>;
  constexpr int P = G::P, SEG = G::SEG, KP = G::KP, D = G::D;
  constexpr bool REPLAY = MODE == FM_REPLAY, MASK = MODE == FM_MASK, EVEN = MODE == FM_CTX,
                 CTX = MASK || EVEN || (MODE == FM_ANY && G::GPW == 1);
  constexpr bool STORED = NC >= 16 && (MODE == FM_ANY || MODE == FM_STORED);
  constexpr bool SC = feat_bwd_scaled(MODE, NC, P, W, LD, ACT);
  // (bf16 with one row per lane comes out slower without the test that is always true: 2048 x 256 x 128, groups of 8 618 ->
  // 651 us, 256 x 256 x 128, heads of 16, groups of 16 158 -> 163; elsewhere it costs, four rows 1044 -> 1033, fp32 178 -> 175)
  constexpr bool ALONE = W == 1 && (P > 1 || sizeof(T) == 4);
  constexpr float sT = (float)F::sT;
  constexpr float cds = (float)(kCd * F::ds), cdsm = (float)(kFeatC * F::ds / kFeatM);
  constexpr bool COLS_SHFL = W == 1 && P == 1 && NC <= 4;  // (longer chains: 702 us by shared memory, 714 by shuffles)
  __shared__ __align__(16) float xs[G::TEAMS][2][G::XS];
  __shared__ __align__(16) float cs[G::TEAMS][2][W][G::XS];
  __shared__ float sdw[kFeatWarps][2][D];
  wait_for_inputs();
  const FeatThread<G, LD, W> th(p);
  const T* g_y = static_cast<const T*>(p.in[0]);
  const T* g_ya = static_cast<const T*>(p.in[1]);
  const T* g_dy = static_cast<const T*>(p.in[2]);
  const T* g_dya = static_cast<const T*>(p.in[3]);
  T* g_dx = static_cast<T*>(p.out[0]);
  T* g_dxa = static_cast<T*>(p.out[1]);
  T* g_xr = static_cast<T*>(p.out[2]);
  T* g_xar = static_cast<T*>(p.out[3]);
  const int frow = th.gw * D + th.sub * KF;
  const uint32_t xrow = smem_u32(&xs[th.team][0][frow]);
  const uint32_t crow = smem_u32(&cs[th.team][0][0][frow]);

  // Column sums over the slots: halving exchange (each round a lane keeps one half of its values and
  // receives the partner's sums for that half), then the remaining slots by plain exchanges.
  constexpr int HALV = KF == 6 ? 1 : ilog2(KF);
  constexpr int ROUNDS = HALV < ilog2(SEG) ? HALV : ilog2(SEG);
  constexpr int LEFT = KF >> ROUNDS;  // values a lane still holds
  int cfirst = 0;                     // the first of them
#pragma unroll
  for (int t = 0; t < ROUNDS; ++t) cfirst += ((th.s >> t) & 1) * (KF >> (t + 1));
  const uint32_t ccol = crow + 4u * (uint32_t)(th.wt * G::XS + cfirst);
  const bool cwriter = (th.s >> ROUNDS) == 0;

  float2 Wi[KP], Wj[KP];  // (1 - alpha) folded in
  {
    const float* wi = p.W + th.c * D + th.sub * KF;
    const float* wj = wi + p.E;
#pragma unroll
    for (int q = 0; q < KP; ++q) {
      Wi[q] = make_float2(wi[2 * q] * p.oma, wi[2 * q + 1] * p.oma);
      Wj[q] = make_float2(wj[2 * q] * p.oma, wj[2 * q + 1] * p.oma);
    }
  }
  const float2 alpha_g = f2(p.alpha * (SC ? cdsm : cds));
  // Block of row r: g + (i * stride) mod m, i = i_0 + r SEG.  The offsets are formed again where they are used: kept over
  // the steps they would cost the four-row kernels registers that are not there (1024 x 256 x 128, groups of 32: 1084 ->
  // 1067 us).
  const int shift0 = (int)((long long)th.pos(0) * p.stride % p.m), shift1 = (int)((long long)SEG * p.stride % p.m);
  float2 dwi[KP], dwj[KP];  // without the factor (1 - alpha)
#pragma unroll
  for (int q = 0; q < KP; ++q) dwi[q] = dwj[q] = f2(0.0f);
  int par = 0;

  __shared__ int rows_before[EVEN ? kFeatCtxRows + 1 : 1], warp_sum[kFeatWarps];
  FeatUnits<EVEN> units;
  if constexpr (EVEN) units.init(p.ctxlen, (int)p.B, p.m, NC, rows_before, warp_sum);
  for (long long u = th.first; u < p.units; u += th.step) {
    long long b;
    int g;
    units.unit(u, p.mg, b, g);
    g = g * G::GPW + th.gw;
    const bool valid = G::GPW == 1 || g < p.m;
    float2 X[P][KP], A[P][KP], H[P][KP], Gv[P][KP];
    auto offsets = [&](long long (&off)[P]) {
      asm volatile("" : "+r"(g));  // (or the compiler keeps the first result after all)
      int blk = g + shift0;
      if (blk >= p.m) blk -= p.m;
#pragma unroll
      for (int r = 0; r < P; ++r) {
        off[r] = ((b * p.N + (long long)blk * NC + th.pos(r)) * p.E) + th.c * D + th.sub * KF;
        blk += shift1;
        if (blk >= p.m) blk -= p.m;
      }
    };
    // (stored end state or full replay: y, ya are not read)
    bool from_output = true;
    if constexpr (REPLAY) from_output = sizeof(T) == 4;
    if constexpr (STORED) from_output = !(p.saved == 3 && p.mid_end);
    long long off0[P];
    offsets(off0);
#pragma unroll
    for (int r = 0; r < P; ++r) {
#pragma unroll
      for (int q = 0; q < KP; ++q) X[r][q] = A[r][q] = H[r][q] = Gv[r][q] = f2(0.0f);
      if (valid) {
        if (from_output) {
          ld_feat<KF, T>(g_y + off0[r], X[r]);
          ld_feat<KF, T>(g_ya + off0[r], A[r]);
        }
        ld_feat<KF, T>(g_dy + off0[r], H[r]);
        ld_feat<KF, T>(g_dya + off0[r], Gv[r]);
        // the stored state is needed half a stage from now: towards L2 already
        if constexpr (STORED && NC > 16) {
          if (p.saved == 3 && (th.sub & 3) == 0) {
            const float* mx = p.mid + off0[r];
            asm volatile("prefetch.global.L2 [%0];" ::"l"(mx));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(mx + p.bne));
          }
        }
      }
    }
    int steps = NC, tsteps = NC;  // of this lane's group, of the team
    if constexpr (CTX) {
      if (p.ctxlen != nullptr) {
        steps = valid ? group_steps(p.ctxlen, b, g, NC) : 0;
        tsteps = MASK ? (int)__reduce_max_sync(0xffffffffu, (unsigned)steps) : steps;
      }
    }
    // The steps go in runs of RUN; what replaces the rebuilt state (stored by the forward, or replayed from
    // the saved input) is dealt with between the runs, outside the step loop.  A run ends in true scale.
    constexpr int RUN = REPLAY ? NC / 2 : STORED && NC > 16 ? 16 : NC;
#pragma unroll 1
    for (int j0 = tsteps - 1; j0 >= 0; j0 -= j0 % RUN + 1) {
      if constexpr (REPLAY) {
        if (j0 == NC / 2 - 1 || sizeof(T) != 4) {
          constexpr bool SCF = feat_fwd_scaled(FM_PLAIN, NC, P, W);
          // the state after step j0, exactly: the forward over steps 0..j0 from the saved input
          const T* g_x = static_cast<const T*>(p.xin[0]);
          const T* g_xa = static_cast<const T*>(p.xin[1]);
          if (valid) {
            long long off[P];
            offsets(off);
#pragma unroll
            for (int r = 0; r < P; ++r) {
              ld_feat<KF, T>(g_x + off[r], X[r]);
              ld_feat<KF, T>(g_xa + off[r], A[r]);
            }
          }
#pragma unroll 1
          for (int jf = 0; jf <= j0; ++jf) {
            const int rf = th.template local_row<ALONE>(jf);
            float2 xf[KP];
            if constexpr (W == 1) {  // (bf16, 1024 x 256 x 128, groups of 32: 1553 us, through shared memory 1702)
              const int src = (th.gw * SEG + (jf & (SEG - 1))) * LD + th.sub;
#pragma unroll
              for (int q = 0; q < KP; ++q) {
                float2 v = X[0][q];
#pragma unroll
                for (int r = 1; r < P; ++r)
                  if (rf == r) v = X[r][q];
                xf[q] = shfl2(v, src);
              }
            } else {
              const uint32_t xb = xrow + 4u * (uint32_t)(par * G::XS);
              par ^= 1;
              publish_row<P, KP, KF>(xb, X, rf, rf >= 0 && th.s == (jf & (SEG - 1)));
              team_sync<W>(th.team);
              lds_row<KF>(xb, xf);
            }
            feat_forward_step<LD, KP, P, ACT, false, SCF>(X, A, xf, Wi, Wj, p.alpha, jf, true);
          }
          const float2 sc = f2(kPow.pos[j0 + 1]);
#pragma unroll
          for (int r = 0; r < P; ++r)
#pragma unroll
            for (int q = 0; q < KP && SCF; ++q) {
              X[r][q] = __fmul2_rn(X[r][q], sc);
              A[r][q] = __fmul2_rn(A[r][q], sc);
            }
        }
      } else if constexpr (STORED) {
        // the state after step j0 as the forward stored it
        if (p.saved == 3 && ((j0 + 1) & 15) == 0 && (j0 + 1 < NC || p.mid_end) && valid) {
          const float* mx = p.mid + (long long)(2 * ((j0 + 1) / 16 - 1)) * p.bne;
          long long off[P];
          offsets(off);
#pragma unroll
          for (int r = 0; r < P; ++r) {
            ld_feat<KF, float>(mx + off[r], X[r]);
            ld_feat<KF, float>(mx + p.bne + off[r], A[r]);
          }
        }
      }
      const int jend = j0 - j0 % RUN;
      // first step of this lane's group in the run (MASK: groups of a warp start at different steps)
      const int jtop = MASK && steps - 1 < j0 ? steps - 1 : j0;
      int rprev = -1;  // row and slot test of the step whose column sums are still in `cs`
      bool sprev = false;
      auto take_columns = [&]() {  // H_j += the team's column sums of the previous step (buffer par ^ 1)
        const bool mine = rprev >= 0 && sprev;
        const uint32_t cb = crow + 4u * (uint32_t)((par ^ 1) * W * G::XS);
        float2 add[KP];
#pragma unroll
        for (int q = 0; q < KP; ++q) add[q] = f2(0.0f);
        lds_row_if<KF>(mine, cb, add);
#pragma unroll
        for (int w = 1; w < W; ++w) {
          float2 t[KP];
#pragma unroll
          for (int q = 0; q < KP; ++q) t[q] = f2(0.0f);
          lds_row_if<KF>(mine, cb + 4u * (uint32_t)(w * G::XS), t);
#pragma unroll
          for (int q = 0; q < KP; ++q) add[q] = __fadd2_rn(add[q], t[q]);
        }
#pragma unroll
        for (int r = 0; r < P; ++r)
#pragma unroll
          for (int q = 0; q < KP; ++q)
            if (P == 1 || rprev == r) H[r][q] = __fadd2_rn(H[r][q], add[q]);
      };
      auto run_step = [&](int j, int kk) {  // kk steps of the run done
        const bool on = !MASK || j <= jtop;
        const int k = MASK ? (on ? jtop - j : 0) : kk;
        const float mk = SC ? kPow.pos[k] : 1.0f, iq = SC ? kPow.neg[k + 1] : 1.0f;
        if (on) {
#pragma unroll
          for (int r = 0; r < P; ++r)
#pragma unroll
            for (int q = 0; q < KP; ++q) {
              if constexpr (SC) X[r][q] = __ffma2_rn(A[r][q], f2(-kC), X[r][q]);
              else X[r][q] = __ffma2_rn(A[r][q], f2(-kCoverM), __fmul2_rn(X[r][q], f2(kInvM)));
            }
        }
        const int rj = th.template local_row<ALONE>(j);
        const bool sj = on && th.s == (j & (SEG - 1));
        float2 xj[KP];
        if constexpr (W == 1) {  // (shuffles: shorter than the way through shared memory)
          if constexpr (!COLS_SHFL) {
            team_sync<W>(th.team);
            take_columns();
          }
          const int src = (th.gw * SEG + (j & (SEG - 1))) * LD + th.sub;
#pragma unroll
          for (int q = 0; q < KP; ++q) {
            float2 v = X[0][q];
#pragma unroll
            for (int r = 1; r < P; ++r)
              if (rj == r) v = X[r][q];
            xj[q] = shfl2(v, src);
          }
        } else {
          const uint32_t xb = xrow + 4u * (uint32_t)(par * G::XS);
          publish_row<P, KP, KF>(xb, X, rj, rj >= 0 && th.s == (j & (SEG - 1)));
          team_sync<W>(th.team);
          take_columns();
          lds_row<KF>(xb, xj);
        }
        float2 accj = f2(0.0f);
#pragma unroll
        for (int q = 0; q < KP; ++q) accj = __ffma2_rn(xj[q], Wj[q], accj);
        const float cj = accj.x + accj.y;
        const float2 al = f2(p.alpha * sT * iq);
        const float ss = sT * iq * iq, sg = SC ? cdsm * iq : cds;
        constexpr double ca = SC ? kFeatC : kCd / kMd;
        const float2 a1 = f2((float)(-ca * F::f1) * mk);
        [[maybe_unused]] const float2 a0 = f2((float)(-ca * F::f0) * mk);
        float gs[P];
        float2 uu[KP];  // sum_i sim_i gT_i of this lane's positions, per feature
#pragma unroll
        for (int r = 0; r < P; ++r) {
          float2 acc = f2(0.0f);
#pragma unroll
          for (int q = 0; q < KP; ++q) acc = __ffma2_rn(X[r][q], Wi[q], acc);
          const float sim = red_sub<LD>(acc.x + acc.y + cj);
          const float2 sim_s = f2(sim * ss), simg = f2(sim * sg);
          float2 ts[KP], rr[KP];
#pragma unroll
          for (int q = 0; q < KP; ++q) ts[q] = __ffma2_rn(sim_s, xj[q], __fmul2_rn(X[r][q], al));
          feat_act<ACT, KP, feat_bwd_batch(MODE, P, W)>(ts, rr);
          float2 gacc = f2(0.0f);
#pragma unroll
          for (int q = 0; q < KP; ++q) {
            const float2 gap = __ffma2_rn(f2(kC), H[r][q], Gv[r][q]);
            const float2 gt = F::gt(gap, ts[q], rr[q]);
            gacc = __ffma2_rn(gt, xj[q], gacc);
            uu[q] = r == 0 ? __fmul2_rn(simg, gt) : __ffma2_rn(simg, gt, uu[q]);
            if (on) {  // (gs_i Wi is added to H below)
              if constexpr (SC) {
                if constexpr (F::f0 != 0.0) A[r][q] = __fadd2_rn(A[r][q], a0);
                A[r][q] = __ffma2_rn(rr[q], a1, A[r][q]);
                Gv[r][q] = gap;
                H[r][q] = __ffma2_rn(gt, alpha_g, H[r][q]);
              } else {
                A[r][q] = __ffma2_rn(rr[q], a1, __ffma2_rn(A[r][q], f2(kInvM), a0));
                Gv[r][q] = __fmul2_rn(gap, f2(kM));
                H[r][q] = __ffma2_rn(gt, alpha_g, __fmul2_rn(H[r][q], f2(kM)));
              }
            }
          }
          gs[r] = red_sub<LD>(gacc.x + gacc.y) * sg;
        }
        float sl = 0.0f;
#pragma unroll
        for (int r = 0; r < P; ++r) {
          const float2 gsv = f2(gs[r]);
          sl += gs[r];
          if (on) {
#pragma unroll
            for (int q = 0; q < KP; ++q) {
              H[r][q] = __ffma2_rn(gsv, Wi[q], H[r][q]);
              dwi[q] = __ffma2_rn(gsv, X[r][q], dwi[q]);
            }
          }
        }
        float v[KF];
#pragma unroll
        for (int q = 0; q < KP; ++q) {
          if (on) dwj[q] = __ffma2_rn(f2(sl), xj[q], dwj[q]);
          const float2 t = __ffma2_rn(f2(sl), Wj[q], uu[q]);  // + sum_i gs_i Wj
          v[2 * q] = t.x; v[2 * q + 1] = t.y;
        }
#pragma unroll
        for (int t = 0; t < ROUNDS; ++t) {
          const int half = KF >> (t + 1);
          const bool up = ((th.s >> t) & 1) != 0;
#pragma unroll
          for (int i = 0; i < half; ++i) {
            const float keep = up ? v[i + half] : v[i];
            const float send = up ? v[i] : v[i + half];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, LD << t);
          }
        }
#pragma unroll
        for (int o = LD << ROUNDS; o < LD * SEG; o <<= 1)
#pragma unroll
          for (int i = 0; i < LEFT; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
        if constexpr (COLS_SHFL) {  // straight to the lanes of position j
          const int base = th.lane - ((th.s & ((1 << ROUNDS) - 1)) * LD);
          float col[KF];
#pragma unroll
          for (int f = 0; f < KF; ++f) {
            int owner = 0;  // slot bits of the lane that ends up with feature f
#pragma unroll
            for (int t = 0; t < ROUNDS; ++t) owner |= ((f / (KF >> (t + 1))) & 1) << t;
            col[f] = __shfl_sync(0xffffffffu, v[f % LEFT], base + owner * LD);
          }
#pragma unroll
          for (int q = 0; q < KP; ++q)
            if (sj) H[0][q] = __fadd2_rn(H[0][q], make_float2(col[2 * q], col[2 * q + 1]));
        } else {
#pragma unroll
          for (int i = 0; i < LEFT; ++i) sts_if(cwriter, ccol + 4u * (uint32_t)(par * W * G::XS + i), v[i]);
          rprev = rj;
          sprev = sj;
          par ^= 1;
        }
      };
      if constexpr (feat_bwd_unrolled(NC, P, W, LD)) {
#pragma unroll
        for (int kk = 0; kk < NC; ++kk) {
          if (CTX && kk > j0) break;
          run_step(j0 - kk, kk);
        }
      } else {
#pragma unroll 1
        for (int j = j0; j >= jend; --j) run_step(j, j0 - j);
      }
      if constexpr (!COLS_SHFL) {
        team_sync<W>(th.team);
        take_columns();
      }
      // true scale: k steps done
      const float2 up = f2(kPow.neg[jtop - jend + 1]), dn = f2(kPow.pos[jtop - jend + 1]);
#pragma unroll
      for (int r = 0; r < P; ++r)
#pragma unroll
        for (int q = 0; q < KP && SC; ++q) {
          X[r][q] = __fmul2_rn(X[r][q], up);
          A[r][q] = __fmul2_rn(A[r][q], up);
          H[r][q] = __fmul2_rn(H[r][q], dn);
          Gv[r][q] = __fmul2_rn(Gv[r][q], dn);
        }
    }  // runs
    if (valid) {
      long long off[P];
      offsets(off);
#pragma unroll
      for (int r = 0; r < P; ++r) {
        st_feat<KF, T>(g_dx + off[r], H[r]);
        st_feat<KF, T>(g_dxa + off[r], Gv[r]);
        if (g_xr) {
          st_feat<KF, T>(g_xr + off[r], X[r]);
          st_feat<KF, T>(g_xar + off[r], A[r]);
        }
      }
    }
  }

  // ---- weight gradient: slots of the warp, warps of the same head, then the CTA's partial
#pragma unroll
  for (int q = 0; q < KP; ++q) {
#pragma unroll
    for (int o = LD; o < 32; o <<= 1) {
      dwi[q].x += __shfl_xor_sync(0xffffffffu, dwi[q].x, o);
      dwi[q].y += __shfl_xor_sync(0xffffffffu, dwi[q].y, o);
      dwj[q].x += __shfl_xor_sync(0xffffffffu, dwj[q].x, o);
      dwj[q].y += __shfl_xor_sync(0xffffffffu, dwj[q].y, o);
    }
  }
  if (th.lane < LD) {
#pragma unroll
    for (int q = 0; q < KP; ++q) {
      sdw[th.warp][0][th.sub * KF + 2 * q] = dwi[q].x * p.oma;
      sdw[th.warp][0][th.sub * KF + 2 * q + 1] = dwi[q].y * p.oma;
      sdw[th.warp][1][th.sub * KF + 2 * q] = dwj[q].x * p.oma;
      sdw[th.warp][1][th.sub * KF + 2 * q + 1] = dwj[q].y * p.oma;
    }
  }
  __syncthreads();
  const int nwarp = blockDim.x >> 5, tpc = nwarp / W;
  for (int idx = threadIdx.x; idx < 2 * p.E; idx += blockDim.x) {
    const int which = idx / p.E, f = idx - which * p.E;
    const int c = f / D, k = f - c * D;
    float acc = 0.0f;
    for (int w = 0; w < nwarp; ++w) {
      const long long gt = (long long)blockIdx.x * tpc + w / W;
      if ((int)(gt % p.C) == c) acc += sdw[w][which][k];
    }
    p.partials[(long long)blockIdx.x * 2 * p.E + idx] = acc;
  }
}

}  // namespace ncn
