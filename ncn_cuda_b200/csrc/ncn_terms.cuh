// Rows of a forward that did not come out finite, once more by the plain formula.
//
// Where the positions of a group share reciprocals (act_r_all), a NaN in one of them becomes a NaN in the others, and infinities in the
// scaled variables meet products and sums that the formula does not have.  The row kernels leave it at that while they run, look at their
// results, and take the rows with a NaN or an infinity in x again, here: a position sees its own NaN and x_j's, and T is formed as
// alpha x + (owi x + owj xj) xj.  A NaN or an infinity in x or in a, and a NaN in T, stay in x to the end of a net (x' = m x + c a',
// a' = m a + c F, and the shared reciprocals lose no NaN), so no row that met one is missed; the others keep their values.
//
// Forward before and with it, B200: 65536 x 4096, groups of 4, 6 stages 2891 -> 2909 us; 32768 x 4096, groups of 8, 4 stages 1664 -> 1698;
// bf16 with sigmoid 0.4 %; where the steps looked for a NaN in x_j before (rows that do not fill their warps, rows of 8192 positions,
// one group per thread) 1 to 3 % faster.  Tried in its place: the plain formula as a branch of every stage 2949 us, a test of the
// inputs before the stages 3030 us, a NaN in x_j carried through the constant of each step 2977 us.
#pragma once
#include "ncn_rows.cuh"

namespace ncn {

// Whether positions of a group share reciprocals.
template <int ACT>
__host__ __device__ constexpr bool act_shares() { return ACT == ACT_TANH || ACT == ACT_SIGMOID; }

// Whether the values whose squares q sums up are finite (false also beyond 1e18: such a row only goes the longer way).
__device__ __forceinline__ bool finite(float2 q) { return q.x + q.y < __int_as_float(0x7f800000); }

// The rows of a CTA that did not come out finite, behind its tile loop: *wild says that there are any, the stored results which.  By all
// threads of the CTA.  buf: 2N floats, the tile buffer.  PAIRS: stored states in the order of ncn_lanes.cuh, else in that of
// ncn_rows.cuh.  Not after a wait that was given up, when loads may be on their way to the buffer, and not where the results have
// replaced the input (F_OVERLAP): there a NaN stays in all the positions that shared its reciprocals.
//
// One loop over what a thread does next: the compiler weighs code by the depth of its loops, and with a loop
// each for rows, stages and steps it took registers from the tile loop (groups of 8: 3 % of the forward).
template <int NG, int ACT, typename T, bool PAIRS, typename P>
__device__ __forceinline__ void wild_rows_by_terms(const P& p, const int* wild, const int* gave_up, const StageRec* recs, float* buf) {
  using F = ActForm<ACT>;
  constexpr float sT = (float)F::sT;
  __syncthreads();
  if (!*wild || *gave_up || (p.flags & F_OVERLAP)) return;
  const int tid = threadIdx.x, nthr = blockDim.x, N = p.N, m = p.m;
  if (tid == 0) bulk_wait_all0();
  __syncthreads();
  const T* const x_in = static_cast<const T*>(p.in[0]);
  const T* const xa_in = static_cast<const T*>(p.in[1]);
  T* const y = static_cast<T*>(p.out[0]);
  T* const ya = static_cast<T*>(p.out[1]);
  const float al = p.alpha * sT;
  long long row = (long long)blockIdx.x * p.R;
  int l = -1, j = 0, pos = tid;  // stage (-1: the look, L: the results), step, position or group of this thread
  float q = 0.0f;
  while (row < p.B) {
    const long long at = row * N;
    if (l < 0) {
      if (pos < N) {
        q = fmaf(0.0f, Store<T>::ld(y + at + pos), q);  // NaN where one of them is not finite
        buf[pos] = Store<T>::ld(x_in + at + pos);
        buf[N + pos] = Store<T>::ld(xa_in + at + pos);
      }
    } else if (l < p.L) {
      if (pos < m) {  // (the groups of a stage share no position)
        const StageRec rec = recs[l];
        const float owi = rec.owi * sT, xj = buf[(int)((pos + (long long)j * rec.s) % m) * NG + j], oj = rec.owj * sT * xj;
        float* const ck = rec.ck >= 0 && j == NG - 1 ? p.ckpt + 2 * (rec.ck * p.B * N + at) : nullptr;
        int blk = pos;
#pragma unroll
        for (int i = 0; i < NG; ++i) {
          float* const xi = buf + blk * NG + i;
          const float sim = __fadd_rn(__fmul_rn(owi, xi[0]), oj);  // (products of equal size and opposite sign leave 0)
          const float ts = fmaf(sim, xj, al * xi[0]);
          const float a = fmaf(kM, xi[N], kC * fmaf((float)F::f1, F::r(make_float2(ts, ts)).x, (float)F::f0));
          const float x = fmaf(kM, xi[0], kC * a);
          xi[0] = x;
          xi[N] = a;
          if (ck != nullptr) {
            ck[PAIRS ? i * m + pos : 2 * (i * m + pos)] = x;
            ck[PAIRS ? (NG + i) * m + pos : 2 * (i * m + pos) + 1] = a;
          }
          blk = wrap_add(blk, rec.s, m);
        }
      }
    } else if (pos < N) {
      Store<T>::st(y + at + pos, (p.flags & F_RESIDUAL) ? buf[pos] + Store<T>::ld(x_in + at + pos) : buf[pos]);
      Store<T>::st(ya + at + pos, buf[N + pos]);
    }
    pos += nthr;
    if (pos - tid < (l >= 0 && l < p.L ? m : N)) continue;
    pos = tid;
    if (l < 0) {
      l = __syncthreads_or(q != 0.0f) ? 0 : p.L + 1;
      q = 0.0f;
    } else {
      __syncthreads();
      if (l == p.L) ++l; else if (++j == NG) { j = 0; ++l; }
    }
    if (l > p.L) {  // next row
      l = -1;
      ++row;
      if (row % p.R == 0) row += (gridDim.x - 1) * (long long)p.R;
    }
  }
}

}  // namespace ncn
