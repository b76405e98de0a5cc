// Pose update of one Softassign inner iteration, shared by the matrix-free
// kernels (sm_103a): from the grid-reduced moments to the next pose
// (src/softassign.cu:772-798 then findRTfromS, src/findRTfromS.cpp:33-159).
#pragma once
#include "cesa_ops.cuh"
#include "cesa_pose.h"
#include "cesa_pose_dd.cuh"
#include "cesa_prep.cuh"

namespace cesa {

struct SaPoseScratch {
  float S[9], xcp[3], yd[3], xc[3], yc[3];
  float Sl[9], xcl[3], ydl[3];  // S, xcp and yd below FP32 (pairs only)
};

// sa_moments_to_S with the centres, alpha and beta as (hi, lo) pairs too. Two
// clouds of unequal counts give sum V a part that S must cancel, against which
// FP32 rounding of a centre shows.
__device__ __forceinline__ void sa_moments_to_S_dd(int tid, const df* s_tot, const float* oX, const float* oY,
                                                   const float* yh, SaPoseScratch& ps) {
  const df A1 = dd_fast(s_tot[0].hi, s_tot[0].lo);
  const float inv = dd_inv(A1);
  auto over = [&](int k) { return dd_div(dd_fast(s_tot[k].hi, s_tot[k].lo), A1, inv); };
  auto minus = [](df a, df b) {
    df_add(a, df{-b.hi, -b.lo});
    return dd_fast(a.hi, a.lo);
  };
  df rm = over(28);  // rho - 1
  df_add(rm, -1.f);
  rm = dd_fast(rm.hi, rm.lo);
  const int i = tid < 9 ? tid % 3 : tid - 9, j = tid < 9 ? tid / 3 : tid - 9;
  const df xi = over(1 + i);
  df yd = over(29 + j);  // Yc - oY = B2 / A1 + (rho - 1) oY
  df_add(yd, dd_mul(rm, df_make(oY[j])));
  yd = dd_fast(yd.hi, yd.lo);
  if (tid < 9) {
    const df al = dd_sum(yh[j], oY[j]), be = minus(df_make(yh[j]), yd);
    const df T3 = s_tot[13 + j], T5 = s_tot[19], T7 = s_tot[23], T9 = s_tot[27];
    const df P2 = minus(s_tot[16 + i], dd_mul(xi, T5)), P3 = minus(s_tot[20 + i], dd_mul(xi, A1));
    df sij = minus(s_tot[4 + i + 3 * j], dd_mul(xi, T3));
    df_add(sij, dd_mul(P2, al));
    df_add(sij, dd_mul(P3, be));
    const df o = df_make(oX[i]);
    df_add(sij, dd_mul(minus(s_tot[24 + j], T3), o));
    df_add(sij, dd_mul(dd_mul(minus(T9, T5), al), o));
    df_add(sij, dd_mul(dd_mul(minus(T7, A1), be), o));
    sij = dd_fast(sij.hi, sij.lo);
    ps.S[i + 3 * j] = sij.hi;
    ps.Sl[i + 3 * j] = sij.lo;
  } else {
    ps.xcp[i] = xi.hi;
    ps.xcl[i] = xi.lo;
    ps.yd[i] = yd.hi;
    ps.ydl[i] = yd.lo;
    df xc = xi, yc = yd;
    df_add(xc, oX[i]);
    df_add(yc, oY[i]);
    ps.xc[i] = df_val(xc);
    ps.yc[i] = df_val(yc);
  }
}

// The certified solve as a call of its own: one thread runs it while the
// block waits, and outside the kernel's inlined code it gets its own register
// allocation instead of the sweeps' spills.
static __device__ __noinline__ void horn_fast_call(const float* S, HornState<float>* st, float* q, float* gap,
                                                   float* lmax) {
  horn_quaternion_fast<float>(S, *st, q, gap, lmax);
}

// Block-wide (every thread calls it). s_tot: the 32 moments; s_hdr: oX, oY,
// mean(Y') (centring header). Threads 0..8 form S and threads 9..11 the
// centres; thread 0 then solves Horn's problem (warm-started eigenbasis in
// `horn`) and writes the next centred pose to s_pose. In the block that
// `leads`, it also writes the adjoint's record (tape_rec, kSaTape floats, when
// given), the trace record (trace_rec, 32 doubles, when given) and the step
// count. `fast` selects the certified inverse iteration (horn_quaternion_fast,
// no eigenbasis for an adjoint; the trace's gap is then -1) over the Jacobi
// solve that the taped kernels need; kPairs forms S from paired centres
// and, in the schedule's `last` update, refines the pose.
template <bool kPairs = false>
__device__ __forceinline__ void sa_pose_update(const df* s_tot, const float* s_hdr, SaPoseScratch& ps,
                                               HornState<float>& horn, float* s_pose, bool leads,
                                               float* tape_rec, double* trace_rec, int step, float T,
                                               Ctl* ctl, Timeline* tl = nullptr, bool fast = false,
                                               bool last = false) {
  const int tid = threadIdx.x;
  if (kPairs) {
    if (tid < 12)
      sa_moments_to_S_dd(tid, s_tot, &s_hdr[0], &s_hdr[3], &s_hdr[6], ps);
  } else if (tid < 12) sa_moments_to_S(tid, s_tot, &s_hdr[0], &s_hdr[3], &s_hdr[6], ps.S, ps.xcp, ps.yd, ps.xc, ps.yc);
  __syncthreads();
  if (tl) tl->mark(13);
  if (tid == 0) {
    const float* oX = &s_hdr[0];
    const float* oY = &s_hdr[3];
    float S[9], Xc[3], Yc[3], Xcp[3], Yd[3];
    for (int k = 0; k < 9; ++k) S[k] = ps.S[k];
    for (int i = 0; i < 3; ++i) {
      Xc[i] = ps.xc[i];
      Yc[i] = ps.yc[i];
      Xcp[i] = ps.xcp[i];
      Yd[i] = ps.yd[i];
    }
    float q[4], gap = 0.f, lmax = 0.f, Rn[9], tn[3];
    if (fast)
      horn_fast_call(S, &horn, q, &gap, &lmax);
    else
      horn_quaternion<float>(S, horn, q, &gap, &lmax);
    // centred-frame translation t' = Xc' - R (Yc - oY)
    quat_to_pose<float>(q, Xcp, Yd, Rn, tn);
    if (kPairs && last) horn_refine_dd(ps.S, ps.Sl, ps.xcp, ps.xcl, ps.yd, ps.ydl, q, Rn, tn);
    for (int k = 0; k < 9; ++k) s_pose[k] = Rn[k];
    for (int k = 0; k < 3; ++k) s_pose[9 + k] = tn[k];
    if (leads) {
      if (tape_rec) {  // the update's solve, for the adjoint
        tape_rec[12] = s_tot[0].hi;
        tape_rec[13] = s_tot[0].lo;
        for (int i = 0; i < 3; ++i) {
          tape_rec[14 + i] = Xc[i];
          tape_rec[17 + i] = Yc[i];
          tape_rec[20 + i] = Xcp[i];
          tape_rec[23 + i] = Yd[i];
        }
        for (int i = 0; i < 9; ++i) tape_rec[26 + i] = S[i];
        for (int i = 0; i < 4; ++i) tape_rec[35 + i] = q[i];
        for (int i = 0; i < 4; ++i)
          for (int j = 0; j < 4; ++j) tape_rec[39 + 4 * i + j] = horn.V[i][j];
      }
      if (trace_rec) {
        double* rec = trace_rec;
        float to[3];
        pose_from_centred(Rn, tn, oX, oY, to);
        rec[0] = step;
        rec[1] = T;
        rec[2] = df_dbl(s_tot[0]);
        for (int i = 0; i < 3; ++i) {
          rec[3 + i] = Xc[i];
          rec[6 + i] = Yc[i];
          rec[27 + i] = to[i];
        }
        for (int k = 0; k < 9; ++k) {
          rec[9 + k] = S[k];
          rec[18 + k] = Rn[k];
        }
        rec[30] = gap;
        rec[31] = lmax;
      }
      ctl->steps_done = step + 1;
    }
  }
  __syncthreads();
}

}  // namespace cesa
