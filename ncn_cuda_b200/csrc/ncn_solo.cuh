// Fused row kernels with one group per thread (one feature per position): groups of 16, and the rows of groups of 8 that
// ncn_lanes.cuh does not take (an odd number of blocks, or too many idle lanes).
//
// A pair of 16-position groups does not fit a thread's registers in four streams (ncn_lanes.cuh packs two groups per fp32x2
// instruction), and the kernels that held one kept two warps per scheduler busy.  Here the packed pairs are two positions of
// ONE group: 64 registers of state in the reverse sweep, so that 16 warps fit an SM (forward: 32).
//
//   * Rows come and go by 1-D TMA copies through one tile buffer.  A thread's group at stride 0 is NG contiguous positions:
//     128-bit accesses that start at a lane-dependent slot (LaneChunk) touch all banks.
//   * Between two stages of different stride a thread writes its values to stage-local slots o m + block (all streams of a
//     position in 8 or 16 bytes, consecutive threads consecutive slots) and reads those of the next stride behind one CTA
//     barrier; the slots a thread read are the ones it writes next, so one barrier is enough.  Offset 0 never moves.
//   * Stored states ([o m + g] per row, (x, a) pairs, the order of ncn_rows.cuh) are read from global memory where they are
//     needed; where one follows, x and a are not exchanged at all.
//
// Any number of blocks up to 512 per row, any stride; R rows side by side in a CTA.
//
// Measured on a B200 (forward + backward, before = ncn_pairs.cuh forward and ncn_rows.cuh backward): 25000 x 2048 fp32, groups of
// 16, 3 stages 1447 + 1947 -> 945 + 1660 us; 65536 x 8192 bf16, 4 stages 9.93 + 16.2 -> 9.23 + 15.7 ms.  Cycles per
// warp, position and step: fp32 13.9 + 24.2, arithmetic alone 11.5 + 19.2; bf16 10.0 + 17.0, alone 8.3 + 12.6 (rows of 8192: one
// CTA of 512 threads per SM, whose boundaries nothing overlaps).
#pragma once
#include "ncn_lanes.cuh"
#include "ncn_solo_launch.h"

namespace ncn {

// Steps in the scaled variables of ncn_common.cuh, two positions of the group per instruction; constants of LaneStage.
template <int NG, int ACT, int J>
struct SoloFwd {
  static __device__ __forceinline__ void run(float2 (&X)[NG / 2], float2 (&A)[NG / 2], float owi, float owj, float alpha) {
    using F = ActForm<ACT>;
    using S = LaneStage<NG, ACT>;
    constexpr float mk = (float)cpow(kMd, J), mkDk = (float)(cpow(kMd, J) * fwd_D(J, F::f0));
    constexpr float cA = (float)S::cA(J);
    const float XJ = (J & 1) ? X[J / 2].y : X[J / 2].x;
    const float xj = J == 0 ? XJ : fmaf(XJ, mk, mkDk);
    const float pp = fmaf(owi, xj, alpha);  // sT (alpha + (1-alpha) wi xj)
    float q = (owj * xj) * xj;
    if constexpr (mkDk != 0.0f) q = fmaf(pp, mkDk, q);  // (no product by zero: pp may be infinite)
    const float2 P = f2(pp * mk), Q = f2(q);
    float2 ts[NG / 2], r[NG / 2];
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) ts[i] = __ffma2_rn(X[i], P, Q);
    act_r_all<ACT, NG / 2, 4>(ts, r);
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) {
      A[i] = __ffma2_rn(r[i], f2(cA), A[i]);
      X[i] = __ffma2_rn(A[i], f2(kC), X[i]);
    }
    SoloFwd<NG, ACT, J + 1>::run(X, A, owi, owj, alpha);
  }
};
template <int NG, int ACT>
struct SoloFwd<NG, ACT, NG> {
  static __device__ __forceinline__ void run(float2 (&)[NG / 2], float2 (&)[NG / 2], float, float, float) {}
};

template <int NG, int ACT, int J>
struct SoloBwd {
  static __device__ __forceinline__ void run(float2 (&X)[NG / 2], float2 (&A)[NG / 2], float2 (&H)[NG / 2], float2 (&G)[NG / 2],
                                             float owi, float owj, float owjs, float alpha, float& dwi, float& dwj) {
    using F = ActForm<ACT>;
    using S = LaneStage<NG, ACT>;
    constexpr int k = NG - 1 - J;
    constexpr double mkd = cpow(kMd, k), DX = bwd_DX(k + 1, F::f0);
    constexpr float imk1 = (float)(1.0 / cpow(kMd, k + 1)), DX1 = (float)DX, imk1DX1 = (float)(DX / cpow(kMd, k + 1));
    constexpr float cAr = (float)S::cAr(J);
    constexpr float sTimk1 = (float)(F::sT / cpow(kMd, k + 1)), cdsm = (float)(kCd * F::ds / kMd);
    constexpr float K1 = (float)(kCd * F::ds / kMd / cpow(kMd, k + 1)), K2 = (float)(2.0 * kCd * F::ds / kMd);
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) X[i] = __ffma2_rn(f2(-kC), A[i], X[i]);
    const float XJ = (J & 1) ? X[J / 2].y : X[J / 2].x;
    const float xj = fmaf(XJ, imk1, imk1DX1);
    const float pp = fmaf(owi, xj, alpha), ps = pp * sTimk1;
    const float2 Ps = f2(ps), Qs = f2(fmaf(ps, DX1, (owjs * xj) * xj)), PH = f2(pp * cdsm);
    float2 ts[NG / 2], r[NG / 2], aI, aS;
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) ts[i] = __ffma2_rn(X[i], Ps, Qs);
    act_r_all<ACT, NG / 2, 2>(ts, r);
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) {
      A[i] = __ffma2_rn(r[i], f2(cAr), A[i]);
      G[i] = __ffma2_rn(f2(kC), H[i], G[i]);
      const float2 gt = F::gt(G[i], ts[i], r[i]);
      H[i] = __ffma2_rn(gt, PH, H[i]);
      aI = i == 0 ? __fmul2_rn(gt, X[0]) : __ffma2_rn(gt, X[i], aI);
      aS = i == 0 ? gt : __fadd2_rn(aS, gt);
    }
    // sums in raw units (as LBwdSteps): dwi gains xj u, dwj m^k xj v; their factors are lane_dw_scale_i / _j
    const float sS = aS.x + aS.y, u = fmaf(DX1, sS, aI.x + aI.y), v = xj * sS;
    const float add = fmaf(owj * v, K2, (owi * u) * K1);
    if (J & 1) H[J / 2].y += add; else H[J / 2].x += add;
    dwi = fmaf(xj, u, dwi);
    dwj = fmaf(xj * v, (float)mkd, dwj);
    SoloBwd<NG, ACT, J - 1>::run(X, A, H, G, owi, owj, owjs, alpha, dwi, dwj);
  }
};
template <int NG, int ACT>
struct SoloBwd<NG, ACT, -1> {
  static __device__ __forceinline__ void run(float2 (&)[NG / 2], float2 (&)[NG / 2], float2 (&)[NG / 2], float2 (&)[NG / 2], float,
                                             float, float, float, float&, float&) {}
};

// a group's NG contiguous positions <-> its pairs; slot (t + k) mod S in round k (LaneChunk: no bank conflicts)
template <int NG, typename T>
__device__ __forceinline__ void solo_ld(const T* chunk, float2 (&v)[NG / 2], int t) {
  float2 g[1][NG / 2];
  lane_ld_native<NG / 2, 2, T>(chunk, g, t);  // read as two halves of a pair: g[o] = (value o, value NG/2 + o)
  float q[NG];
#pragma unroll
  for (int o = 0; o < NG / 2; ++o) { q[o] = g[0][o].x; q[NG / 2 + o] = g[0][o].y; }
#pragma unroll
  for (int i = 0; i < NG / 2; ++i) v[i] = make_float2(q[2 * i], q[2 * i + 1]);
}
template <int NG, typename T>
__device__ __forceinline__ void solo_st(T* chunk, const float2 (&v)[NG / 2], int t) {
  float q[NG];
#pragma unroll
  for (int i = 0; i < NG / 2; ++i) { q[2 * i] = v[i].x; q[2 * i + 1] = v[i].y; }
  float2 g[1][NG / 2];
#pragma unroll
  for (int o = 0; o < NG / 2; ++o) g[0][o] = make_float2(q[o], q[NG / 2 + o]);
  lane_st_native<NG / 2, 2, T>(chunk, g, t);
}
template <int NG>
__device__ __forceinline__ float solo_get(const float2 (&v)[NG / 2], int o) { return (o & 1) ? v[o >> 1].y : v[o >> 1].x; }
template <int NG>
__device__ __forceinline__ void solo_set(float2 (&v)[NG / 2], int o, float x) {
  if (o & 1) v[o >> 1].y = x; else v[o >> 1].x = x;
}

// ------------------------------------------------------------------------------------------ forward
template <int NG, int ACT, typename T, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) solo_fwd_kernel(const __grid_constant__ SoloParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  using F = ActForm<ACT>;
  using S = LaneStage<NG, ACT>;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int N = p.N, m = p.m, R = p.R, L = p.L;
  const int RN = R * N;
  T* win = reinterpret_cast<T*>(smem);               // native x at win, xa at win + RN; (x, a) slots of 8 bytes
  T* sres = reinterpret_cast<T*>(smem + p.off_res);  // F_RESIDUAL: native x of the tile
  StageRec* recs = reinterpret_cast<StageRec*>(smem + p.off_w);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + p.off_bar);
  int* abort_flag = reinterpret_cast<int*>(bar + 2);
  int* wild = abort_flag + 1;  // a row did not come out finite (ncn_terms.cuh)
  const T* gx_in = static_cast<const T*>(p.in[0]);
  const T* ga_in = static_cast<const T*>(p.in[1]);
  T* gy_out = static_cast<T*>(p.out[0]);
  T* gya_out = static_cast<T*>(p.out[1]);
  float2* ckpt = reinterpret_cast<float2*>(p.ckpt);
  const bool residual = (p.flags & F_RESIDUAL) != 0;
  const long long BN = p.B * (long long)N;

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    *abort_flag = 0;
    *wild = 0;
    fence_mbar_init();
  }
  wait_for_inputs();
  fill_stage_table(recs, p.W, p.oma, p.l0, m, L, p.ckpt_every, p.flags, ckpt != nullptr, tid, nthr, &p.list);
  __syncthreads();

  const int r = tid / m, g = tid - r * m;  // row of the tile, group
  const int base = r * N;
  const uint32_t row = smem_u32(smem) + 8u * (uint32_t)base;
  constexpr float sT = (float)F::sT;
  const float alpha = p.alpha * sT;
  uint32_t phase = 0;

  for (long long tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    const long long row0 = tile * R;
    const int rows = (int)min((long long)R, p.B - row0);
    const uint32_t bytes = (uint32_t)(rows * N * sizeof(T));
    if (tid == 0) {
      bulk_wait_read0();  // the previous tile's stores have left the buffer
      mbar_expect_tx(&bar[0], (residual ? 3 : 2) * bytes);
      bulk_g2s(win, gx_in + row0 * N, bytes, &bar[0]);
      bulk_g2s(win + RN, ga_in + row0 * N, bytes, &bar[0]);
      if (residual) bulk_g2s(sres, gx_in + row0 * N, bytes, &bar[0]);
    }
    if (!mbar_wait_bounded(&bar[0], phase)) *abort_flag = 1;
    phase ^= 1;
    __syncthreads();
    if (*abort_flag) break;
    const bool active = r < rows;

    float2 X[NG / 2], A[NG / 2];
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) X[i] = A[i] = f2(0.0f);
    if (active) {
      solo_ld<NG, T>(win + base + g * NG, X, g);
      solo_ld<NG, T>(win + RN + base + g * NG, A, g);
    }
    __syncthreads();  // native inputs are in registers; the buffer may take slots
    if (tid == 0 && tile + gridDim.x < p.tiles) {  // next tile towards L2 while this one is worked on
      const long long nrow0 = (tile + gridDim.x) * R;
      const uint32_t nbytes = (uint32_t)(min((long long)R, p.B - nrow0) * N * sizeof(T));
      l2_prefetch(gx_in + nrow0 * N, nbytes);
      l2_prefetch(ga_in + nrow0 * N, nbytes);
    }
    int s_cur = 0;
    auto exchange = [&](int s) {  // from stride s_cur to stride s
      if (s == s_cur) return;
      if (active) {
        int blk = g;
#pragma unroll
        for (int o = 1; o < NG; ++o) {
          blk = wrap_add(blk, s_cur, m);
          sts64(row + 8u * (uint32_t)(o * m + blk), solo_get<NG>(X, o), solo_get<NG>(A, o));
        }
      }
      __syncthreads();
      if (active) {
        int blk = g;
#pragma unroll
        for (int o = 1; o < NG; ++o) {
          blk = wrap_add(blk, s, m);
          const float2 v = lds64(row + 8u * (uint32_t)(o * m + blk));
          solo_set<NG>(X, o, v.x);
          solo_set<NG>(A, o, v.y);
        }
      }
      s_cur = s;
    };
    for (int l = 0; l < L; ++l) {
      const StageRec rec = recs[l];
      exchange(rec.s);
      SoloFwd<NG, ACT, 0>::run(X, A, rec.owi * sT, rec.owj * sT, alpha);
#pragma unroll
      for (int i = 0; i < NG / 2; ++i) {
        X[i] = __ffma2_rn(X[i], f2((float)S::mN), f2((float)S::mND));
        A[i] = __ffma2_rn(A[i], f2((float)S::mN), f2((float)S::mNC));
      }
      if (rec.ck >= 0 && active) {
        float2* ck = ckpt + (long long)rec.ck * BN + (row0 + r) * N + g;
#pragma unroll
        for (int o = 0; o < NG; ++o) ck[o * m] = make_float2(solo_get<NG>(X, o), solo_get<NG>(A, o));
      }
    }
    if constexpr (act_shares<ACT>()) {
      float2 q = f2(0.0f);
#pragma unroll
      for (int i = 0; i < NG / 2; ++i) q = __ffma2_rn(X[i], X[i], q);
      if (active && !finite(q)) *wild = 1;
    }
    exchange(0);
    __syncthreads();  // every slot has been read; the buffer may take the native results
    if (active) {
      if (residual) {
        float2 xin[NG / 2];
        solo_ld<NG, T>(sres + base + g * NG, xin, g);
#pragma unroll
        for (int i = 0; i < NG / 2; ++i) X[i] = __fadd2_rn(X[i], xin[i]);
      }
      solo_st<NG, T>(win + base + g * NG, X, g);
      solo_st<NG, T>(win + RN + base + g * NG, A, g);
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(gy_out + row0 * N, win, bytes);
      bulk_s2g(gya_out + row0 * N, win + RN, bytes);
      bulk_commit();
    }
  }
  if constexpr (act_shares<ACT>()) wild_rows_by_terms<NG, ACT, T, /*PAIRS=*/false>(p, wild, abort_flag, recs, reinterpret_cast<float*>(win));
  if (tid == 0) {
    bulk_wait_all0();
    if (*abort_flag) atomicExch(p.status, DEV_WAIT_TIMEOUT);
  }
}

// ------------------------------------------------------------------------------------------ backward
// From the net output (reversible inverse), from stored states (checkpoints, F_TAPE), F_RESIDUAL; no forward replay.
//
// AHEAD (not with F_RESIDUAL, nor where the rebuilt input is asked for): the streams of the next tile are copied to a buffer of their
// own while this one is worked on, and with F_TAPE the state it starts from is read into x and a as soon as they are done with.  (A
// kernel of its own: the choice at run time costs the plain one 5 to 10 per cent, in registers.)
template <int NG, int ACT, typename T, int MAXT, int MINB, int AHEAD>
__global__ void __launch_bounds__(MAXT, MINB) solo_bwd_kernel(const SoloParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  using F = ActForm<ACT>;
  using S = LaneStage<NG, ACT>;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarp = nthr >> 5;
  const int N = p.N, m = p.m, R = p.R, L = p.L;
  const int RN = R * N;
  T* win = reinterpret_cast<T*>(smem);  // native streams q at win + q*RN; (gx, ga, x, a) slots of 16 bytes
  T* sdy = reinterpret_cast<T*>(smem + p.off_res);  // F_RESIDUAL: native dy of the tile
  float* red = reinterpret_cast<float*>(smem + p.off_red);  // [L][nwarp][2]
  StageRec* recs = reinterpret_cast<StageRec*>(smem + p.off_w);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + p.off_bar);
  int* abort_flag = reinterpret_cast<int*>(bar + 2);
  const T* g_in[4] = {static_cast<const T*>(p.in[0]), static_cast<const T*>(p.in[1]), static_cast<const T*>(p.in[2]),
                      static_cast<const T*>(p.in[3])};
  const float2* ckpt = reinterpret_cast<const float2*>(p.ckpt);
  const bool want_rec = !AHEAD && p.out[2] != nullptr;
  const bool residual = !AHEAD && (p.flags & F_RESIDUAL) != 0;
  // the last stage's output state comes from its checkpoint
  const bool tape = AHEAD ? AHEAD == SOLO_AHEAD_TAPE : (p.flags & F_TAPE) != 0;
  const long long BN = p.B * (long long)N;

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  wait_for_inputs();
  fill_stage_table(recs, p.W, p.oma, p.l0, m, L, p.ckpt_every, p.flags, ckpt != nullptr, tid, nthr);
  for (int i = tid; i < 2 * L * nwarp; i += nthr) red[i] = 0.0f;
  __syncthreads();

  const int r = tid / m, g = tid - r * m;
  const int base = r * N;
  const uint32_t row = smem_u32(smem) + 16u * (uint32_t)base;
  constexpr float sT = (float)F::sT;
  const float dsi = lane_dw_scale_i<ACT>(p.oma), dsj = lane_dw_scale_j<ACT>(p.oma);
  uint32_t phase = 0;

  constexpr int Q0 = AHEAD == SOLO_AHEAD_TAPE ? 2 : 0;  // AHEAD: the first stream that is read, at land
  T* const land = reinterpret_cast<T*>(smem + p.off_land);
  auto copy_ahead = [&](long long tl) {
    const uint32_t nbytes = (uint32_t)(min((long long)R, p.B - tl * R) * N * sizeof(T));
    mbar_expect_tx(&bar[0], (4 - Q0) * nbytes);
#pragma unroll
    for (int q = Q0; q < 4; ++q) bulk_g2s(land + (q - Q0) * RN, g_in[q] + tl * R * N, nbytes, &bar[0]);
  };
  float2 X[NG / 2], A[NG / 2];
  auto load_state = [&](long long tl, int ck) {
    const float2* c = ckpt + (long long)ck * BN + (tl * R + r) * N + g;
#pragma unroll
    for (int o = 0; o < NG; ++o) {
      const float2 v = __ldg(c + o * m);
      solo_set<NG>(X, o, v.x);
      solo_set<NG>(A, o, v.y);
    }
  };
  if (AHEAD) {
    if (tid == 0) copy_ahead(blockIdx.x);  // (there is a tile for every CTA)
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) X[i] = A[i] = f2(0.0f);
    if (AHEAD == SOLO_AHEAD_TAPE && r < min((long long)R, p.B - (long long)blockIdx.x * R)) load_state(blockIdx.x, recs[L - 1].ck);
  }

  for (long long tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
    const long long row0 = tile * R;
    const int rows = (int)min((long long)R, p.B - row0);
    const uint32_t bytes = (uint32_t)(rows * N * sizeof(T));
    if (!AHEAD && tid == 0) {
      bulk_wait_read0();  // the previous tile's stores have left the buffer
      mbar_expect_tx(&bar[0], (tape ? 2 : 4) * bytes + (residual ? bytes : 0));
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q >= 2 || !tape) bulk_g2s(win + q * RN, g_in[q] + row0 * N, bytes, &bar[0]);
      if (residual) bulk_g2s(sdy, g_in[2] + row0 * N, bytes, &bar[0]);
    }
    if (!mbar_wait_bounded(&bar[0], phase)) *abort_flag = 1;
    phase ^= 1;
    __syncthreads();
    if (*abort_flag) break;
    const bool active = r < rows;

    float2 H[NG / 2], G[NG / 2];
#pragma unroll
    for (int i = 0; i < NG / 2; ++i) {
      H[i] = G[i] = f2(0.0f);
      if (AHEAD != SOLO_AHEAD_TAPE) X[i] = A[i] = f2(0.0f);
    }
    if (active) {
      const T* c = (AHEAD ? land - Q0 * RN : win) + base + g * NG;
      if (!tape) {
        solo_ld<NG, T>(c, X, g);
        solo_ld<NG, T>(c + RN, A, g);
      }
      solo_ld<NG, T>(c + 2 * RN, H, g);
      solo_ld<NG, T>(c + 3 * RN, G, g);
    }
    if (AHEAD && tid == 0) bulk_wait_read0();  // the previous tile's stores have left the buffer
    __syncthreads();  // native inputs are in registers; the buffer may take slots
    if (AHEAD && tid == 0 && tile + gridDim.x < p.tiles) copy_ahead(tile + gridDim.x);
    if (tid == 0 && tile + gridDim.x < p.tiles) {  // next tile towards L2 while this one is worked on
      const long long nrow0 = (tile + gridDim.x) * R;
      const int nrows = (int)min((long long)R, p.B - nrow0);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (!AHEAD && (q >= 2 || !tape)) l2_prefetch(g_in[q] + nrow0 * N, (uint32_t)(nrows * N * sizeof(T)));
      for (int k = 0; k < p.n_ckpt; ++k) l2_prefetch(ckpt + (long long)k * BN + nrow0 * N, (uint32_t)(nrows * N * sizeof(float2)));
    }
    int s_cur = 0;
    auto exchange = [&](int s, bool state) {  // from stride s_cur to stride s; state: x, a as well
      if (s == s_cur) return;
      if (active) {
        int blk = g;
#pragma unroll
        for (int o = 1; o < NG; ++o) {
          blk = wrap_add(blk, s_cur, m);
          const uint32_t a = row + 16u * (uint32_t)(o * m + blk);
          if (state) sts128(a, solo_get<NG>(H, o), solo_get<NG>(G, o), solo_get<NG>(X, o), solo_get<NG>(A, o));
          else sts64(a, solo_get<NG>(H, o), solo_get<NG>(G, o));
        }
      }
      __syncthreads();
      if (active) {
        int blk = g;
#pragma unroll
        for (int o = 1; o < NG; ++o) {
          blk = wrap_add(blk, s, m);
          const uint32_t a = row + 16u * (uint32_t)(o * m + blk);
          if (state) {
            const float4 v = lds128(a);
            solo_set<NG>(H, o, v.x); solo_set<NG>(G, o, v.y); solo_set<NG>(X, o, v.z); solo_set<NG>(A, o, v.w);
          } else {
            const float2 v = lds64(a);
            solo_set<NG>(H, o, v.x); solo_set<NG>(G, o, v.y);
          }
        }
      }
      s_cur = s;
    };
    for (int l = L - 1; l >= 0; --l) {
      const StageRec rec = recs[l];
      exchange(rec.s, rec.ck < 0);
      // a state saved after stage l replaces the rebuilt one
      if (rec.ck >= 0 && active && (AHEAD != SOLO_AHEAD_TAPE || l < L - 1)) load_state(tile, rec.ck);
      float dwi = 0.0f, dwj = 0.0f;
      SoloBwd<NG, ACT, NG - 1>::run(X, A, H, G, rec.owi, rec.owj, rec.owj * sT, p.alpha, dwi, dwj);
#pragma unroll
      for (int i = 0; i < NG / 2; ++i) {
        X[i] = __ffma2_rn(X[i], f2((float)S::imN), f2((float)S::imNDX));
        A[i] = __ffma2_rn(A[i], f2((float)S::imN), f2((float)S::imNCA));
        H[i] = __fmul2_rn(H[i], f2((float)S::mN));
        G[i] = __fmul2_rn(G[i], f2((float)S::mN));
      }
      // ---- weight-gradient partial of this stage: fixed-order warp tree, one slot per warp
      {
        const float di = active ? dwi * dsi : 0.0f, dj = active ? dwj * dsj : 0.0f;
        const bool hi = (lane & 16) != 0;
        const float give = hi ? di : dj;
        float keep = hi ? dj : di;
        keep += __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
        if ((lane & 15) == 0) red[(l * nwarp + warp) * 2 + (hi ? 1 : 0)] += keep;
      }
    }
    if (AHEAD == SOLO_AHEAD_TAPE && r < min((long long)R, p.B - (tile + gridDim.x) * R)) load_state(tile + gridDim.x, recs[L - 1].ck);
    exchange(0, want_rec);
    __syncthreads();  // every slot has been read; the buffer may take the native results
    if (active) {
      if (residual) {
        float2 gin[NG / 2];
        solo_ld<NG, T>(sdy + base + g * NG, gin, g);
#pragma unroll
        for (int i = 0; i < NG / 2; ++i) H[i] = __fadd2_rn(H[i], gin[i]);
      }
      T* c = win + base + g * NG;
      solo_st<NG, T>(c, H, g);
      solo_st<NG, T>(c + RN, G, g);
      if (want_rec) {
        solo_st<NG, T>(c + 2 * RN, X, g);
        solo_st<NG, T>(c + 3 * RN, A, g);
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(static_cast<T*>(p.out[0]) + row0 * N, win, bytes);
      bulk_s2g(static_cast<T*>(p.out[1]) + row0 * N, win + RN, bytes);
      if (want_rec) {
        bulk_s2g(static_cast<T*>(p.out[2]) + row0 * N, win + 2 * RN, bytes);
        bulk_s2g(static_cast<T*>(p.out[3]) + row0 * N, win + 3 * RN, bytes);
      }
      bulk_commit();
    }
  }
  // ---- per-CTA partial: sum the warp slots in warp order
  __syncthreads();
  for (int i = tid; i < 2 * L; i += nthr) {
    const int l = i >> 1, c = i & 1;
    float acc = 0.0f;
    for (int w2 = 0; w2 < nwarp; ++w2) acc += red[(l * nwarp + w2) * 2 + c];
    p.partials[(long long)blockIdx.x * 2 * L + i] = acc;
  }
  if (tid == 0) {
    bulk_wait_all0();
    if (*abort_flag) atomicExch(p.status, DEV_WAIT_TIMEOUT);
  }
}

}  // namespace ncn
