// Fused, streaming EM-ICP for sm_103a: the whole sigma schedule of emicp()
// (src/emicp.cu:441-669) in one persistent cooperative launch, with the N x M
// matrix A never materialised.
//
// Reference step (src/emicp.cu:453-635), rows r = Y points, columns c = X:
//   A_rc = exp(-|x_c - (R y_r + t)|^2 / sigma_p2)               (updateA)
//   C_r  = sum_c A_rc + exp(-d_02 / sigma_p2)                    (Sgemv + Saxpy)
//   A_rc <- sqrt(A_rc / C_r)   if C_r > 1e-6, else 1/N           (normalizeRowsOfA)
//   lambda_r = sum_c A_rc,  X'_r = sum_c A_rc x_c / lambda_r     (Sgemv, Sgemm, division)
//   Xc = sum lambda X' / sum lambda,  Yc = sum lambda y / sum lambda
//   S  = sum_r lambda_r (X'_r - Xc)(y_r - Yc)^T,  pose = findRTfromS(Xc, Yc, S)
// One-pass restatement used here: with e_rc = exp(-d^2 / (2 sigma_p2)) we have
// A = e^2 and sqrt(A / C) = e / sqrt(C). Per row, three running sums over the
// columns give everything: sum e^2, sum e, sum e*x. Then
//   C_r = sum e^2 + outlier,  lambda_r = sum e / sqrt(C_r),  lambda_r X'_r = sum e x / sqrt(C_r).
// Three forms, by size (plan_emicp):
//   small clouds    whole rows to a block, X in shared memory, one grid barrier a
//                   step: direct differences on scaled coordinates, 11 FP32 pipe ops
//                   + 1 MUFU per element;
//   large clouds    the local sweep: Y sorted, every unit about a centre of its
//                   own, 8 ops + 1 MUFU;
//   what is left    (lopsided clouds, single steps) direct differences over (row
//                   block, column slice) units with a scale, 12 ops + 1 MUFU, or
//                   over task ranges on scaled copies of X, 11.
//
// Coordinates are centred on the device (FP32 offsets oX, oY) before the
// loop. EM-ICP's S is translation invariant, so only Xc, Yc and t are shifted
// back; the pose enters and leaves in the caller's frame.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/cesa.h"
#include "cesa_kernels.h"
#include "cesa_ops.cuh"
#include "cesa_pose.h"
#include "cesa_pose_dd.cuh"
#include "cesa_prep.cuh"

namespace cesa {

struct EmicpArgs {
  const float4* rows;  // Y' centred (owned), M
  const float4* cols;  // X' centred (streamed), N
  int M, N;
  SweepGeom geo;
  float sigma0, sigma_factor, d_02;
  int nsteps;
  const CenterHdr* hdr;
  float* dRt;           // PoseIO in/out, caller frame
  float* part;          // row partials [5][S][Mp] (accumulator, column slice, row); ranged: [5][nblk][kmax][kBlockPts]
  const float4* xs;     // direct sweeps over ranges: two copies of X' scaled by a step's sc (step parity)
  const float4* blk;    // local sweeps: centre and radius of every owned block's rows (NaN: not compact)
  int refine;           // teams: refine every step's pose
  int Mp;
  df* rbpart;           // [2][grid][kEmNV] moments per block (step parity)
  Ctl* ctl;
  unsigned* pair_tab;   // SM pairs (geo.pair_num): [2 kPairCap + 1], zero at launch
  float* pair_t;        // SM pairs: [grid] sweep time of each virtual block, ns
  double* trace;
  int trace_cap;
  float* row_out;       // optional [M][5] (centred-frame u)
  float* tape;          // optional [nsteps][kEmTape]
  float* row_tape;      // optional [nsteps][M][5]
  int* d_status;
  unsigned long long* tl;
  int tl_cap;
  uint64_t timeout_ns;
};

// ---------------------------------------------------------------- local sweep
// The E-step sweep on clouds scaled by sc = sqrt(log2(e) / (2 sigma_p2)), each
// owned block about a centre c' of its own (its posed box centre, scaled):
//   e = 2^-|x' - z'|^2 = 2^-|z~|^2 2^(2 z~.x~ - |x~|^2),  x~ = x' - c', z~ = z' - c'.
// The prepare step streams (x~, -|x~|^2), lanes own 2 z~, and the row factor
// 2^-|z~|^2 multiplies a row's sums once: 3 FFMA for the exponent in place of
// 3 FADD + FMUL + 2 FFMA, 8 FP32 ops per element in place of 11. It is taken
// while the block's scaled radius is at most sqrt(kLocalR2), where 2^|z~|^2
// cannot overflow a sum of e^2; otherwise the block sweeps direct differences
// (EmicpElemScaled). The exponent is rounded at the size of |x~|^2 (of affinities that
// count, |x~| < 6 + radius), not of d^2: at small sigma a row's sum of e^2 is further
// off FP64 than by direct differences (10,007 x 9001, rms: 2.5e-7 -> 3.4e-7 at sigma_p2 =
// 3e-4, 2.2e-7 -> 3.8e-7 at 1e-4, 9.7e-7 -> 1.25e-6 at 1.06e-5). Refined poses more than make
// up for that in poses and gradients. Y is sorted
// along a Hilbert curve so that blocks are compact: at N = M = 40,097 98% of the
// default schedule's affinities take the short form, at 8171 points 91%.
// Bound by the FP32 pipe as before (72% of it busy where every block is short,
// 23.0 instructions per 128 elements against 29.5): N = M = 40,097 36.3 -> 31.5
// ms (poses refined), 17,000 8.75 -> 7.57. Not kept: 8 owned points a
// lane (256 per unit 33.0 ms, or 128 over half-warps 33.4, at their best pair
// splits), records stored as packed duplicates (35.4), kLocalR2 = 16 (32.1).
constexpr float kLocalR2 = 48.f;

// The poses of the local form are refined (horn_refine_dd), and those of the last
// steps on small clouds: the short form's rounding is then more than made up for,
// and gradients, which see the poses' noise most, come out closer to FP64 than with
// FP32 solves. At 10,007 x 9001 and 7000 x 7500, 16 pairs, gradients are 0.9e-6 -
// 2.6e-6 off with all 66 steps refined, 0.8e-6 - 4.6e-6 with the last 30, 0.9e-6 -
// 5.7e-6 with 16, 2.1e-6 - 1.1e-5 with none and direct differences. ~2 us a
// step, a third of a small clouds' step: they take the second half only.
constexpr int kSmallRefine = 32;

struct EmicpElemLocal {  // q = 2 z~ of two owned points; s = (x~, -|x~|^2)
  __device__ __forceinline__ void operator()(float2 (&acc)[5], const float2 (&q)[3], float4 s) const {
    float2 t = __ffma2_rn(q[2], dup2(s.z), dup2(s.w));
    t = __ffma2_rn(q[1], dup2(s.y), t);
    const float2 e = ex2_pair(__ffma2_rn(q[0], dup2(s.x), t));
    acc[0] = __ffma2_rn(e, e, acc[0]);
    acc[1] = __fadd2_rn(acc[1], e);
    acc[2] = __ffma2_rn(e, dup2(s.x), acc[2]);
    acc[3] = __ffma2_rn(e, dup2(s.y), acc[3]);
    acc[4] = __ffma2_rn(e, dup2(s.z), acc[4]);
  }
};

struct LocalSmem {
  float rho[2][kBlockPts];  // the owned points' |z~|^2, by unit parity
};

// As sweep_units (deferred), for the EM-ICP E-step: every unit's partial sums
// of e^2, e and e x' (scaled frame) are stored per (row, slice or slot).
template <int kLayout>
__device__ __forceinline__ bool em_local_sweep(const int& bid, const int& G, SweepSmem& sm, LocalSmem& ls, Pipe& pipe, const SweepGeom& g,
                                               const StreamSrc& src, const float4* own, const float4* blkinfo,
                                               const float (&R)[9], const float (&tc)[3], float sc, float* part,
                                               int part_ld, Ctl* ctl, uint64_t timeout_ns, int where, Timeline& tl,
                                               OwnCache& oc, const RangedShare* rs) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool ranged = kLayout == 1;
  pipe.cur = -1;
  auto task_range = [&](int uu, int ch, int& first, int& len) -> bool {  // as in sweep_units
    if (ranged) {
      const int o = rs->o_first + uu;
      const int o_last = rs->o_last;
      if (o > o_last) return false;
      const int c = (uu == 0 ? rs->c_first : 0) + ch;
      if (c >= (o == o_last ? rs->c_end : g.nch)) return false;
      first = c * kChunk;
      len = min(kChunk, g.n_stream - first);
      return true;
    }
    if (uu >= g.units) return false;
    const int sl = uu % g.slices;
    const int sb = sl * g.slice_len;
    const int se = min(sb + g.slice_len, g.n_stream);
    first = sb + ch * kChunk;
    if (first >= se) return false;
    len = min(kChunk, se - first);
    return true;
  };
  const int ustep = ranged ? 1 : G;
  int u = ranged ? 0 : bid;
  int cur_first = 0, cur_len = 0, cur_ch = 0, cur_stage = 0;
  unsigned cur_par = 0;
  bool cur_wait = false;
  int par = 0, upar = 0;
  bool have = task_range(u, 0, cur_first, cur_len);
  if (have) {
    cur_stage = pipe_issue(pipe, sm, src, cur_first, cur_first, cur_len, cur_wait);
    cur_par = (pipe.uses[cur_stage] - 1u) & 1u;
  }
  while (have) {
    const int blk = ranged ? rs->o_first + u : u / g.slices, sl = ranged ? u : u % g.slices;
    float4 ow[kOwnPerLane];
    load_owned_cached(oc, own, g.n_own, blk, ow);
    const float4 bi = __ldg(blkinfo + blk);
    const float cx = R[0] * bi.x + R[1] * bi.y + R[2] * bi.z + tc[0];
    const float cy = R[3] * bi.x + R[4] * bi.y + R[5] * bi.z + tc[1];
    const float cz = R[6] * bi.x + R[7] * bi.y + R[8] * bi.z + tc[2];
    const bool local = bi.w * bi.w * sc * sc <= kLocalR2;  // false for NaN; the same in every thread
    float2 q[kPairs][3];
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
      float p[2][3];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = 2 * k + h, i = lane + 32 * j;
        p[h][0] = R[0] * ow[j].x + R[1] * ow[j].y + R[2] * ow[j].z + tc[0];
        p[h][1] = R[3] * ow[j].x + R[4] * ow[j].y + R[5] * ow[j].z + tc[1];
        p[h][2] = R[6] * ow[j].x + R[7] * ow[j].y + R[8] * ow[j].z + tc[2];
        if (local) {
          const bool in = blk * kBlockPts + i < g.n_own;  // padding rows sit at the centre
          p[h][0] = in ? p[h][0] - cx : 0.f;
          p[h][1] = in ? p[h][1] - cy : 0.f;
          p[h][2] = in ? p[h][2] - cz : 0.f;
          if (warp == 0) ls.rho[upar][i] = fmaf(p[h][2], p[h][2], fmaf(p[h][1], p[h][1], p[h][0] * p[h][0]));
        }
      }
      const float f = local ? 2.f : -1.f;  // the scaled element takes the negated coordinates
#pragma unroll
      for (int c = 0; c < 3; ++c) q[k][c] = make_float2(f * p[0][c], f * p[1][c]);
    }
    float2 acc[kPairs][5];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
#pragma unroll
      for (int a = 0; a < 5; ++a) acc[k][a] = make_float2(0.f, 0.f);

    for (;;) {
      int n_first = 0, n_len = 0, n_u = u, n_ch = cur_ch + 1, n_stage = 0;
      unsigned n_par = 0;
      bool n_wait = false;
      bool have_n = task_range(n_u, n_ch, n_first, n_len);
      if (!have_n) {
        n_u = u + ustep;
        n_ch = 0;
        have_n = task_range(n_u, 0, n_first, n_len);
      }
      pipe.cur = cur_stage;
      if (have_n) {
        n_stage = pipe_issue(pipe, sm, src, n_first, n_first, n_len, n_wait);
        n_par = (pipe.uses[n_stage] - 1u) & 1u;
      }
      const bool bad = cur_wait && !mbar_wait(&sm.full[cur_stage], cur_par, ctl, timeout_ns, where);
      if (cur_ch == 0 && u == bid) tl.mark(2);
      // prepare: double-buffered, one block barrier per chunk (a stage that
      // timed out is read as it is; the block leaves after the barrier)
      float4* buf = par ? sm.prep2 : sm.prep;
      par ^= 1;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = tid + h * kThreads;
        if (c < cur_len) {
          const float4 x = sm.raw[cur_stage][c];
          float4 o;
          if (local) {
            o.x = fmaf(x.x, sc, -cx);
            o.y = fmaf(x.y, sc, -cy);
            o.z = fmaf(x.z, sc, -cz);
            o.w = -fmaf(o.z, o.z, fmaf(o.y, o.y, o.x * o.x));
          } else {
            o = make_float4(x.x * sc, x.y * sc, x.z * sc, 0.f);
          }
          buf[c] = o;
        }
      }
      if (__syncthreads_or(bad)) {
        // leave only after the prefetched copy (if any) has landed
        if (have_n && n_wait) mbar_wait(&sm.full[n_stage], n_par, ctl, timeout_ns, where + 1);
        return false;
      }
      if (local) {
        const EmicpElemLocal elem{};
#pragma unroll 8
        for (int c = warp; c < cur_len; c += kWarps) {
          const float4 a = buf[c];
#pragma unroll
          for (int k = 0; k < kPairs; ++k) elem(acc[k], q[k], a);
        }
      } else {
        const EmicpElemScaled elem{};
#pragma unroll 8
        for (int c = warp; c < cur_len; c += kWarps) {
          const float4 a = buf[c];
#pragma unroll
          for (int k = 0; k < kPairs; ++k) elem(acc[k], q[k], a, a);
        }
      }
      const bool unit_done = !(have_n && n_u == u);
      cur_first = n_first;
      cur_len = n_len;
      cur_ch = n_ch;
      cur_stage = n_stage;
      cur_par = n_par;
      cur_wait = n_wait;
      have = have_n;
      if (unit_done) break;
    }
    tl.mark(3);
    float tot[5];
    reduce_warps<5>(sm, acc, tot);
    const int i = blk * kBlockPts + tid;
    if (tid < kBlockPts && i < g.n_own) {
      if (local) {  // the row factor, and x~ back to x'
        const float rho = ex2_approx(-ls.rho[upar][tid]);
        tot[0] *= rho * rho;
        tot[1] *= rho;
        tot[2] = fmaf(tot[1], cx, tot[2] * rho);
        tot[3] = fmaf(tot[1], cy, tot[3] * rho);
        tot[4] = fmaf(tot[1], cz, tot[4] * rho);
      }
      if (ranged) {  // slot (owned block, j): this block is the j-th to cover it
        const int j = sl == 0 ? rs->j_first : 0;
        if (j < g.kmax) {
#pragma unroll
          for (int a = 0; a < 5; ++a) __stcg(part + (((size_t)a * g.nblk + blk) * g.kmax + j) * kBlockPts + tid, tot[a]);
        } else {
          set_status(ctl, kStatusInternal, where + 3);  // the plan's kmax is inconsistent
        }
      } else {
#pragma unroll
        for (int a = 0; a < 5; ++a) __stcg(part + ((size_t)a * g.slices + sl) * part_ld + i, tot[a]);
      }
    }
    upar ^= 1;
    tl.mark(4);
    u += ustep;
    cur_ch = 0;
  }
  return true;
}

// ---------------------------------------------------------------- small clouds
// A step of small clouds is a chain of latencies, of which the general path's
// two grid barriers are the largest. Here a block owns whole rows (up to 32)
// and holds all of X in shared memory: its rows' sums are complete within the
// block, and a step has one grid barrier (for the moments). A thread takes every
// 256th pair of columns against 4 rows at a time: direct differences, 11
// FP32 ops per element (the scale rides on the difference's FFMA). Bound by that
// chain (about 5.7 us a step) up to 2000 points, by the FP32 pipe from 5000 on:
// N = M = 1007 591 -> 493 us, 8171 x 6007 1897 -> 1739 (device call, poses of the
// second half refined).
constexpr int kRowsOwn = 32;                // most rows of a block
constexpr int kRowsMaxN = 8192;             // X in shared memory, two blocks to an SM
constexpr int kRowsPad = 2 * kThreads;      // columns are padded to this
struct RowsSmem {
  float4 y[kRowsOwn];                       // this block's rows
  float4 nz[kRowsOwn];                      // -z of the step, scaled
  float part[kRowsOwn / 4][kWarps][4][5];   // per-warp sums of (pass, row, accumulator)
  df mom[kEmNV][kRowsOwn + 1];
};
__host__ __device__ constexpr size_t rows_smem(int N) {
  return sizeof(RowsSmem) + sizeof(float) * 3 * (size_t)((N + kRowsPad - 1) / kRowsPad * kRowsPad);
}

__device__ __forceinline__ void rows_load(const EmicpArgs& A, RowsSmem& rs, float* xs, int r0, int nrows) {
  const int Np = (A.N + kRowsPad - 1) / kRowsPad * kRowsPad;
  for (int i = threadIdx.x; i < Np; i += kThreads) {
    // padding columns: so far away that their affinity is 0 at every finite sigma_p2
    // (the scale is 4.6e-20 and more: formed without 2 sigma_p2, which overflows)
    const float4 x = i < A.N ? ld_cg(A.cols + i) : make_float4(3e38f, 3e38f, 3e38f, 0.f);
    xs[i] = x.x;
    xs[Np + i] = x.y;
    xs[2 * Np + i] = x.z;
  }
  if ((int)threadIdx.x < kRowsOwn)
    rs.y[threadIdx.x] = (int)threadIdx.x < nrows ? ld_cg(A.rows + r0 + threadIdx.x) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Every row's sums of e^2, e and e x over all columns, per warp, into rs.part.
__device__ __forceinline__ void rows_sweep(const EmicpArgs& A, RowsSmem& rs, const float* xs, float sc, int nrows) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Np2 = (A.N + kRowsPad - 1) / kRowsPad * kThreads;  // pairs of columns
  const float2* x2 = reinterpret_cast<const float2*>(xs);
  const float2 sc2 = make_float2(sc, sc);
  for (int p = 0; 4 * p < nrows; ++p) {
    float2 q[4][3], acc[4][5];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 z = rs.nz[4 * p + r];
      q[r][0] = dup2(z.x);
      q[r][1] = dup2(z.y);
      q[r][2] = dup2(z.z);
#pragma unroll
      for (int a = 0; a < 5; ++a) acc[r][a] = make_float2(0.f, 0.f);
    }
#pragma unroll 2
    for (int i = tid; i < Np2; i += kThreads) {
      const float2 x = x2[i], y = x2[Np2 + i], z = x2[2 * Np2 + i];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 dx = __ffma2_rn(x, sc2, q[r][0]), dy = __ffma2_rn(y, sc2, q[r][1]), dz = __ffma2_rn(z, sc2, q[r][2]);
        const float2 e = ex2_neg_pair(__ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx))));
        acc[r][0] = __ffma2_rn(e, e, acc[r][0]);
        acc[r][1] = __fadd2_rn(acc[r][1], e);
        acc[r][2] = __ffma2_rn(e, x, acc[r][2]);
        acc[r][3] = __ffma2_rn(e, y, acc[r][3]);
        acc[r][4] = __ffma2_rn(e, z, acc[r][4]);
      }
    }
    // the warp's sums: lanes 8 r .. 8 r + 7 end with row r's
    float v[4][5], w[2][5], u[5];
    const bool up = (lane & 16) != 0, od = (lane & 8) != 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int a = 0; a < 5; ++a) v[r][a] = acc[r][a].x + acc[r][a].y;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int a = 0; a < 5; ++a) {
        const float give = up ? v[r][a] : v[r + 2][a], keep = up ? v[r + 2][a] : v[r][a];
        w[r][a] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
      }
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      const float give = od ? w[0][a] : w[1][a], keep = od ? w[1][a] : w[0][a];
      u[a] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)
#pragma unroll
      for (int a = 0; a < 5; ++a) u[a] += __shfl_xor_sync(0xffffffffu, u[a], off);
    if ((lane & 7) == 0)
#pragma unroll
      for (int a = 0; a < 5; ++a) rs.part[p][warp][lane >> 3][a] = u[a];
  }
}

// The rows completed (by warp 0, after a block barrier) and their 16 moments,
// added in row order by halves, stored as this block's record.
__device__ __forceinline__ void rows_finish(const EmicpArgs& A, RowsSmem& rs, int r0, int nrows, float outlier,
                                            const float* hdr, float* row_tape, df* rec) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return;
  df v[kEmNV];
#pragma unroll
  for (int k = 0; k < kEmNV; ++k) v[k] = df_make(0.f);
  if (lane < nrows) {
    float tot[5];
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      float t = rs.part[lane >> 2][0][lane & 3][a];
#pragma unroll
      for (int w = 1; w < kWarps; ++w) t += rs.part[lane >> 2][w][lane & 3][a];
      tot[a] = t;
    }
    const float xm[3] = {hdr[6], hdr[7], hdr[8]}, oX[3] = {hdr[0], hdr[1], hdr[2]};
    const float4 y = rs.y[lane];
    emicp_row_finish(r0 + lane, __float_as_int(y.w), tot, y, outlier, xm, A.row_out, oX, row_tape, v);
#pragma unroll
    for (int k = 0; k < kEmNV; ++k) rs.mom[k][lane] = v[k];
  }
  __syncwarp();
  const int k = lane & 15;
  df s = df_make(0.f);
  for (int i = lane >> 4; i < nrows; i += 2) df_add(s, rs.mom[k][i]);
  const df o = df_shfl_down(s, 16);
  df_add(s, o);
  if (lane < 16) __stcg(reinterpret_cast<float2*>(rec + k), make_float2(s.hi, s.lo));
}

// One registration by blocks 0 .. G - 1, this one block bid; false after a
// failure (status set). kPlain: local sweeps (A.blk) or direct differences over
// slices. kRanges: direct differences over task ranges, in a kernel of its own
// (beside the local sweeps it made them 1% slower). kTeams: one of several in the
// launch (local sweeps, no tape); the caller has initialised the stage barriers
// and the pipe. kSmall: small clouds, whole rows to a block (sm and pipe unused);
// kSmallOut: the same for a caller that wants the rows.
constexpr int kPlain = 0, kTeams = 1, kSmall = 2, kRanges = 3, kSmallOut = 4;
template <int kMode>
__device__ __forceinline__ bool emicp_run(const EmicpArgs& A, SweepSmem& sm, Pipe& pipe, const int& bid, const int& G,
                                          RowsSmem* rs = nullptr, float* xs = nullptr) {
  constexpr bool kTeam = kMode == kTeams, kRows = kMode == kSmall || kMode == kSmallOut;
  __shared__ float s_pose[12];
  __shared__ df s_red[kThreads];
  __shared__ OwnCache oc_rows;
  __shared__ LocalSmem s_local;
  __shared__ RangedShare rs_rows;  // this block's share of a ranged sweep
  __shared__ int s_pair[3];        // SM pairs: pair index (-1: none), role, parts swapped
  __shared__ uint64_t s_tsweep;    // SM pairs: start of the step's sweep
  __shared__ df s_tot[kEmNV];
  __shared__ float s_emS[30];  // S, Xc, Yc of the step; their parts below FP32
  __shared__ float s_hdr[12];

  const int tid = threadIdx.x;

  if (tid == 0) {
    if (!kTeam && !kRows) {
      for (int s = 0; s < kStages; ++s) mbar_init(&sm.full[s], 1);
      mbar_init_fence();
    }
    for (int k = 0; k < 3; ++k) {
      s_hdr[k] = A.hdr->oX[k];
      s_hdr[3 + k] = A.hdr->oY[k];
      s_hdr[6 + k] = A.hdr->xmean[k];
    }
    float R[9], t[3], tc[3];
    for (int k = 0; k < 9; ++k) R[k] = A.dRt[k];
    for (int k = 0; k < 3; ++k) t[k] = A.dRt[9 + k];
    pose_to_centred(R, t, &s_hdr[0], &s_hdr[3], tc);
    for (int k = 0; k < 9; ++k) s_pose[k] = R[k];
    for (int k = 0; k < 3; ++k) s_pose[9 + k] = tc[k];
    if (!kRows) oc_rows.blk = -1;
    int vb = bid;  // the virtual block whose share this block sweeps
    s_pair[0] = -1;
    if (kTeam && A.geo.pair_num) {  // ranks 2 d and 2 d + 1 share an SM
      s_pair[0] = bid >> 1;
      s_pair[1] = bid & 1;
      s_pair[2] = 0;
    } else if (!kRows && A.geo.pair_num) {
      const int2 pr = join_sm_pair(A.pair_tab, A.timeout_ns);
      if (pr.x >= 0 && pr.x < G / 2) {
        s_pair[0] = pr.x;
        s_pair[1] = pr.y;
        s_pair[2] = 0;
        vb = 2 * pr.x + pr.y;
      } else {
        set_status(A.ctl, kStatusInternal, 23);  // the launch ends at its first grid barrier
      }
    }
    if (!kRows) rs_rows = A.geo.pair_num && s_pair[0] < 0 ? RangedShare{0, -1, 0, 0, 0} : ranged_share(A.geo, vb, G);
  }
  __syncthreads();

  __shared__ HornState<float> horn;       // the pose's solver state (thread 0)
  __shared__ HornState<float> horn_tape;  // block 0 with a tape: the eigenbasis for the adjoint
  if (tid == 0) {
    horn.reset();
    horn_tape.reset();
  }
  if (!kTeam && !kRows) pipe_init(pipe);
  unsigned epoch = 0;
  const StreamSrc src{A.cols, nullptr, true};
  float s2 = A.sigma0;
  Timeline tl{kTeam ? nullptr : A.tl, A.tl_cap, 0};
  bool good = true;
  // Direct sweeps over ranges stream X' scaled by sc (and scale the owned rows alike),
  // so that an element needs no scale of its own. Each step's copy is written by
  // all blocks during the previous step's row completion.
  constexpr bool copies = kMode == kRanges;
  auto scale_x = [&](int par, float f) {
    float4* dst = const_cast<float4*>(A.xs) + (size_t)par * A.N;
    for (int i = bid * kThreads + tid; i < A.N; i += G * kThreads) {
      const float4 x = ld_cg(A.cols + i);
      __stcg(dst + i, make_float4(x.x * f, x.y * f, x.z * f, 0.f));
    }
  };
  if (copies && A.nsteps > 0) {
    scale_x(0, sqrtf(kLog2e / (2.f * s2)));
    good = grid_sync(A.ctl, epoch, (unsigned)G, A.timeout_ns, 22);
  }
  const int own_rows = kRows ? A.geo.slice_len : 0;  // small clouds: rows of a block
  const int own_r0 = bid * own_rows, own_n = max(0, min(own_rows, A.M - own_r0));
  if (kRows) rows_load(A, *rs, xs, own_r0, own_n);
  for (int step = 0; step < A.nsteps && good; ++step) {
    tl.mark(1);
    // the scaled X' was written by other blocks' ordinary stores, ahead of a
    // grid barrier; the bulk copies that stream it read through the async proxy
    if (copies && tid == 0) asm volatile("fence.proxy.async.global;" ::: "memory");
    const float outlier = expf(-A.d_02 / s2);  // src/emicp.cu:489
    float R[9], tc[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] = s_pose[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) tc[k] = s_pose[9 + k];
    if (kRows) {
      __syncthreads();  // (the first step: the rows are there)
      const float scr = sqrtf(0.5f * kLog2e / s2);
      if (kMode == kSmallOut) {
        // The rows are asked for: -z scaled is rounded once (warp i: coordinate i). Rounded before
        // the scale as well, as below, the rows' sums of e^2 are 1.15 times further off FP64
        // than with direct differences unscaled, so 0.7 times. A registration, whose
        // refined poses make up for it, keeps the shorter chain (0.15 us a step).
        const int i = tid >> 5, row = tid & 31;
        static_assert(kRowsOwn == 32, "a warp per coordinate");
        if (i < 3) {
          const float4 y = rs->y[row];
          df z = df_make(s_pose[9 + i]);
          df_add_prod(z, s_pose[3 * i], y.x);
          df_add_prod(z, s_pose[3 * i + 1], y.y);
          df_add_prod(z, s_pose[3 * i + 2], y.z);
          z = dd_fast(z.hi, z.lo);
          reinterpret_cast<float*>(&rs->nz[row])[i] = -__fmaf_rn(scr, z.hi, __fmul_rn(scr, z.lo));
        }
      } else if (tid < kRowsOwn) {
        const float4 y = rs->y[tid];
        rs->nz[tid] = make_float4(-scr * (R[0] * y.x + R[1] * y.y + R[2] * y.z + tc[0]),
                                  -scr * (R[3] * y.x + R[4] * y.y + R[5] * y.z + tc[1]),
                                  -scr * (R[6] * y.x + R[7] * y.y + R[8] * y.z + tc[2]), 0.f);
      }
    }
    __syncthreads();

    // e = exp(-d2 / (2 s2)) = 2^(nk d2). Every unit stores its rows' partial
    // sums over its column slice (deferred: no completion counter).
    const float sc = kRows ? sqrtf(0.5f * kLog2e / s2) : sqrtf(kLog2e / (2.f * s2));
    if (kRows) {
      rows_sweep(A, *rs, xs, sc, own_n);
      tl.mark(4);
      __syncthreads();
    } else if (kTeam || copies || A.blk) {
      float Rs[9], tcs[3];
#pragma unroll
      for (int k = 0; k < 9; ++k) Rs[k] = R[k] * sc;
#pragma unroll
      for (int k = 0; k < 3; ++k) tcs[k] = tc[k] * sc;
      if (tid == 0 && s_pair[0] >= 0) s_tsweep = global_ns();
      const bool ok = copies
                          ? sweep_units<5, EmicpElemScaled, NoPrep, NoFin, true, 1>(
                                sm, pipe, A.geo, StreamSrc{A.xs + (size_t)(step & 1) * A.N, nullptr, false}, A.rows, true,
                                Rs, tcs, 0u, A.part, nullptr, EmicpElemScaled{}, NoPrep{}, NoFin{}, A.ctl, A.timeout_ns,
                                10, tl, A.Mp, &oc_rows, &rs_rows)
                      : kTeam || A.geo.ranged
                          ? em_local_sweep<1>(bid, G, sm, s_local, pipe, A.geo, src, A.rows, A.blk, Rs, tcs, sc, A.part, A.Mp,
                                              A.ctl, A.timeout_ns, 10, tl, oc_rows, &rs_rows)
                          : em_local_sweep<0>(bid, G, sm, s_local, pipe, A.geo, src, A.rows, A.blk, Rs, tcs, sc, A.part, A.Mp,
                                              A.ctl, A.timeout_ns, 10, tl, oc_rows, nullptr);
      if (!ok) {
        good = false;
        break;
      }
      if (tid == 0 && s_pair[0] >= 0)
        A.pair_t[2 * s_pair[0] + (s_pair[1] ^ s_pair[2])] = (float)(global_ns() - s_tsweep);
    } else {
      const EmicpElem elem{-kLog2e / (2.f * s2)};
      if (!sweep_units<5, EmicpElem, NoPrep, NoFin, true, 0>(sm, pipe, A.geo, src, A.rows, true, R, tc, 0u, A.part,
                                                           nullptr, elem, NoPrep{}, NoFin{}, A.ctl, A.timeout_ns, 10,
                                                           tl, A.Mp, &oc_rows)) {
        good = false;
        break;
      }
    }
    if (!kRows) {
      if (!grid_sync(A.ctl, epoch, (unsigned)G, A.timeout_ns, 20)) {
        good = false;
        break;
      }
      tl.mark(5);
      if (tid == 0 && s_pair[0] >= 0) {  // SM pairs: the parts change blocks when the times show the other favoured
        long lo = 0, sp = 0, hi = 0;
        ranged_tasks(A.geo, 2 * s_pair[0], G, lo, sp);
        ranged_tasks(A.geo, 2 * s_pair[0] + 1, G, sp, hi);
        if (pair_swap(lo, sp, hi, A.pair_t, s_pair[0])) {
          s_pair[2] ^= 1;
          rs_rows = ranged_share(A.geo, 2 * s_pair[0] + (s_pair[1] ^ s_pair[2]), G);
        }
      }
    }
    // the next step's scaled X' (its buffer was last read by the previous step's sweep)
    if (copies && step + 1 < A.nsteps) scale_x((step + 1) & 1, sqrtf(kLog2e / (2.f * (s2 * A.sigma_factor))));
    // ---- rows completed, each block a contiguous share of them; its 16
    // moments are one record. Thread t first sums the slice partials of
    // (row, accumulator) pairs t, t + kThreads, ... (loads in flight together),
    // then row threads finish their rows (emicp_row_finish).
    df* rb = A.rbpart + (size_t)(step & 1) * G * kEmNV;
    if (kRows) {
      rows_finish(A, *rs, own_r0, own_n, outlier, s_hdr, A.row_tape ? A.row_tape + (size_t)step * A.M * 5 : nullptr,
                  rb + (size_t)bid * kEmNV);
    } else {
      const int S = A.geo.slices;
      const float inv_sc = kTeam || copies || A.blk ? 1.f / sc : 1.f;  // the e x sums are sc times too large
      const int rpc = (A.M + G - 1) / G;
      const int r0 = bid * rpc;
      const int nrows = max(0, min(rpc, A.M - r0));
      float* stot = reinterpret_cast<float*>(&sm.raw2[0][0]);  // [kThreads][5]; raw2 carries no stream here
      static_assert(sizeof(sm.raw2) >= sizeof(float) * 5 * kThreads, "row sums scratch");
      static_assert(offsetof(SweepSmem, full) - offsetof(SweepSmem, prep) >= sizeof(df) * (kEmNV + 1) * kThreads,
                    "moment scratch");
      const float xm[3] = {s_hdr[6], s_hdr[7], s_hdr[8]};
      const float oX[3] = {s_hdr[0], s_hdr[1], s_hdr[2]};
      float* row_tape = A.row_tape ? A.row_tape + (size_t)step * A.M * 5 : nullptr;
      df v[kEmNV];
#pragma unroll
      for (int k = 0; k < kEmNV; ++k) v[k] = df_make(0.f);
      for (int c0 = 0; c0 < nrows; c0 += kThreads) {  // rows [c0, c0 + kThreads) of the share
        const int nr = min(kThreads, nrows - c0);
        for (int pq = tid; pq < 5 * nr; pq += kThreads) {
          const int a = pq % 5, rr = pq / 5;
          if (kTeam || A.geo.ranged) {  // the kmax slots of the row's owned block, in task order
            const int kmax = A.geo.kmax;
            const float* P = A.part + (size_t)a * A.geo.nblk * kmax * kBlockPts + ranged_slot0(r0 + c0 + rr, kmax);
            float sum = 0.f;
            for (int j = 0; j < kmax; j += 4) {  // 4 loads in flight, then added in slot order
              float w[4];
#pragma unroll
              for (int q = 0; q < 4; ++q) w[q] = j + q < kmax ? __ldcg(P + (size_t)(j + q) * kBlockPts) : 0.f;
#pragma unroll
              for (int q = 0; q < 4; ++q) sum += w[q];
            }
            stot[rr * 5 + a] = a >= 2 ? sum * inv_sc : sum;
            continue;
          }
          const float* P = A.part + (size_t)a * S * A.Mp + r0 + c0 + rr;
          float sum = 0.f;
          int k = 0;
          for (; k + 16 <= S; k += 16) {
            float w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = __ldcg(P + (size_t)(k + j) * A.Mp);
#pragma unroll
            for (int j = 0; j < 16; ++j) sum += w[j];
          }
          if (k < S) {
            float w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = k + j < S ? __ldcg(P + (size_t)(k + j) * A.Mp) : 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) sum += w[j];  // adding the zeros leaves the sum unchanged
          }
          stot[rr * 5 + a] = a >= 2 ? sum * inv_sc : sum;
        }
        __syncthreads();
        if (tid < nr) {
          const int r = r0 + c0 + tid;
          const float tot[5] = {stot[tid * 5], stot[tid * 5 + 1], stot[tid * 5 + 2], stot[tid * 5 + 3],
                                stot[tid * 5 + 4]};
          const float4 y = ld_cg(A.rows + r);
          emicp_row_finish(r, __float_as_int(y.w), tot, y, outlier, xm, A.row_out, oX, row_tape, v);
        }
        __syncthreads();
      }
      em_block_moments(v, min(nrows, kThreads), reinterpret_cast<df*>(sm.prep), rb + (size_t)bid * kEmNV);
    }
    if (!grid_sync(A.ctl, epoch, (unsigned)G, A.timeout_ns, 21)) {
      good = false;
      break;
    }
    tl.mark(8);

    // ---- grid-wide moments -> pose (every block computes the same pose)
    reduce_block_partials<kEmNV>(rb, G, s_red, s_tot);
    tl.mark(6);
    const bool refine = kRows ? step + kSmallRefine >= A.nsteps : kTeam ? A.refine != 0 : (!copies && A.blk != nullptr);
    em_moments_to_S_block(s_tot, s_emS, refine);
    if (tid == 0) {
      float Xc[3], Yc[3], S[9];
      for (int k = 0; k < 9; ++k) S[k] = s_emS[k];
      for (int k = 0; k < 3; ++k) {
        Xc[k] = s_emS[9 + k];
        Yc[k] = s_emS[12 + k];
      }
      float q[4], gap = 0.f, lmax = 0.f, Rn[9], tn[3];
      // the pose: certified inverse iteration (Jacobi fallback); the same with
      // and without a tape, so that both forwards agree bitwise
      horn_quaternion_fast<float>(S, horn, q, &gap, &lmax);
      quat_to_pose<float>(q, Xc, Yc, Rn, tn);
      if (refine)
        horn_refine_dd(s_emS, s_emS + 15, s_emS + 9, s_emS + 24, s_emS + 12, s_emS + 27, q, Rn, tn);
      if (!kTeam && A.tape && bid == 0) {  // the step's inputs and solve for the adjoint
        // the adjoint's eigenbasis, from a Jacobi solve of the same S on its own
        // state (it does not feed back into the pose)
        float qj[4], gj = 0.f, lj = 0.f;
        horn_quaternion<float>(S, horn_tape, qj, &gj, &lj);
        float* rec = A.tape + (size_t)step * kEmTape;
        for (int k = 0; k < 12; ++k) rec[k] = s_pose[k];
        rec[12] = s2;
        for (int k = 0; k < kEmNV; ++k) {
          rec[16 + 2 * k] = s_tot[k].hi;
          rec[17 + 2 * k] = s_tot[k].lo;
        }
        for (int i = 0; i < 4; ++i)
          for (int j = 0; j < 4; ++j) rec[48 + 4 * i + j] = horn_tape.V[i][j];
        for (int k = 0; k < 4; ++k) rec[64 + k] = q[k];
      }
      for (int k = 0; k < 9; ++k) s_pose[k] = Rn[k];
      for (int k = 0; k < 3; ++k) s_pose[9 + k] = tn[k];
      if (bid == 0) {
        if (!kTeam && A.trace && step < A.trace_cap) {
          double* rec = A.trace + (size_t)step * 32;
          float to[3];
          pose_from_centred(Rn, tn, &s_hdr[0], &s_hdr[3], to);
          rec[0] = step;
          rec[1] = s2;
          rec[2] = df_dbl(s_tot[0]);
          for (int i = 0; i < 3; ++i) {
            rec[3 + i] = (double)Xc[i] + (double)s_hdr[i];
            rec[6 + i] = (double)Yc[i] + (double)s_hdr[3 + i];
            rec[27 + i] = to[i];
          }
          for (int k = 0; k < 9; ++k) {
            rec[9 + k] = S[k];
            rec[18 + k] = Rn[k];
          }
          rec[30] = gap;
          rec[31] = lmax;
        }
        A.ctl->steps_done = step + 1;
      }
    }
    __syncthreads();
    tl.mark(7);
    s2 *= A.sigma_factor;  // FP32, src/emicp.cu:668
  }

  if (bid == 0 && tid == 0) {
    const int st = ld_status(A.ctl);
    if (st == kStatusOk) {
      float R[9], tc[3], t[3];
      for (int k = 0; k < 9; ++k) R[k] = s_pose[k];
      for (int k = 0; k < 3; ++k) tc[k] = s_pose[9 + k];
      pose_from_centred(R, tc, &s_hdr[0], &s_hdr[3], t);
      for (int k = 0; k < 9; ++k) A.dRt[k] = R[k];
      for (int k = 0; k < 3; ++k) A.dRt[9 + k] = t[k];
    }
    if (A.d_status) *A.d_status = st;
    if (A.tl) A.ctl->pad[0] = (unsigned)tl.n;
  }
  return good;
}

__global__ void __launch_bounds__(kThreads, 2) emicp_kernel(const EmicpArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Pipe pipe;
  emicp_run<kPlain>(A, *reinterpret_cast<SweepSmem*>(smem_raw), pipe, (int)blockIdx.x, (int)gridDim.x);
}

__global__ void __launch_bounds__(kThreads, 2) emicp_ranges_kernel(const EmicpArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Pipe pipe;
  emicp_run<kRanges>(A, *reinterpret_cast<SweepSmem*>(smem_raw), pipe, (int)blockIdx.x, (int)gridDim.x);
}

template <int kMode>
__global__ void __launch_bounds__(kThreads, 2) emicp_rows_kernel(const EmicpArgs A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Pipe pipe;
  emicp_run<kMode>(A, *reinterpret_cast<SweepSmem*>(smem_raw), pipe, (int)blockIdx.x, (int)gridDim.x,
                    reinterpret_cast<RowsSmem*>(smem_raw), reinterpret_cast<float*>(smem_raw + sizeof(RowsSmem)));
}

// Many registrations in one cooperative launch, each by a team of blocks of
// its own: a team goes through its registrations one after the other and waits
// for nobody else, so that pairs of any sizes fill the chip without a step of
// one being a step of all (cesa_teams.cpp). All sweeps are local and ranged: one
// sweep loop (with the slice layout beside it ptxas made it 8% slower), its
// arguments in shared memory. In lock step over all pairs, with direct
// differences, a step paid two grid barriers and a last wave of units; lock step
// -> teams: one pair of 600 x 500 1.58 -> 1.00 ms, 20 of 2000 x 2000 4.47 ->
// 3.04, 60 9.43 -> 6.97, 20 of 6000 x 6000 20.8 -> 17.2, 20 of 500-20,000 points
// 8.8 / 16.3 / 12.3 -> 6.2 / 13.4 / 9.9 (three sets). Bound by the FP32 pipe and, in
// small pairs, by a step's latency; the teams' sizes are even numbers of
// blocks, which leaves up to 8% of the chip idle (20 x 14 of 304 blocks).
__global__ void __launch_bounds__(kThreads, 2) emicp_teams_kernel(const EmicpArgs* __restrict__ jobs,
                                                                  int njobs, const TeamBlock* __restrict__ blocks,
                                                                  Ctl* ctl, unsigned* pair_tab, uint64_t timeout_ns) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(smem_raw);
  __shared__ EmicpArgs s_args;
  static_assert(sizeof(EmicpArgs) % 4 == 0 && sizeof(EmicpArgs) / 4 <= kThreads, "copied by one word a thread");
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) mbar_init(&sm.full[s], 1);
    mbar_init_fence();
  }
  __shared__ int s_vb;
  __shared__ TeamBlock s_team;
  if (tid == 0) {  // SM pairs: virtual blocks 2 d and 2 d + 1 are an SM's two
    int vb = (int)blockIdx.x;
    if (pair_tab) {
      const int2 pr = join_sm_pair(pair_tab, timeout_ns);
      vb = pr.x >= 0 && pr.x < (int)gridDim.x / 2 ? 2 * pr.x + pr.y : -1;
      if (vb < 0) {  // every registration's blocks leave at their first barrier
        set_status(ctl, kStatusInternal, 25);
        for (int j = 0; j < njobs; ++j) set_status(jobs[j].ctl, kStatusInternal, 25);
      }
    }
    s_vb = vb;
  }
  Pipe pipe;
  pipe_init(pipe);
  __syncthreads();
  if (s_vb < 0) return;
  const int vb = s_vb;
  if (tid == 0) s_team = blocks[vb];
  for (;;) {
    __syncthreads();
    if (s_team.njobs <= 0) return;
    if (tid < (int)(sizeof(EmicpArgs) / 4))
      reinterpret_cast<unsigned*>(&s_args)[tid] = reinterpret_cast<const unsigned*>(jobs + s_team.first)[tid];
    __syncthreads();
    if (!emicp_run<kTeams>(s_args, sm, pipe, s_team.rank, s_team.size)) {
      if (tid == 0) set_status(ctl, ld_status(s_args.ctl), 24);
      return;
    }
    if (tid == 0) {
      s_team.first += 1;
      s_team.njobs -= 1;
    }
    for (int s = 0; s < kStages; ++s) pipe.tag[s] = -1;  // the next pair's chunks are others
  }
}

// ---------------------------------------------------------------- row order
// Index of a cell of the 32^3 grid along the Hilbert curve, by Skilling's
// transposition ("Programming the Hilbert curve", AIP Conf. Proc. 707, 2004).
// Consecutive cells are neighbours, so that 128 consecutive points are compact:
// at N = 40,097 98% of the default schedule's (block, step) pairs take the short
// form, against 96% along a Morton curve (8171 points: 91% against 86%).
__device__ __forceinline__ unsigned hilbert_index(unsigned (&x)[3]) {
#pragma unroll
  for (unsigned q = 16; q > 1; q >>= 1) {
    const unsigned p = q - 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (x[i] & q) {
        x[0] ^= p;
      } else {
        const unsigned t = (x[0] ^ x[i]) & p;
        x[0] ^= t;
        x[i] ^= t;
      }
    }
  }
  x[1] ^= x[0];
  x[2] ^= x[1];
  unsigned t = 0;
#pragma unroll
  for (unsigned q = 16; q > 1; q >>= 1)
    if (x[2] & q) t ^= q - 1;
  unsigned key = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    x[i] ^= t;
#pragma unroll
    for (int b = 0; b < 5; ++b) key |= ((x[i] >> b) & 1u) << (3 * b + 2 - i);
  }
  return key;
}

// Order of Y along a Hilbert curve of 32^3 cells over its bounding cube: a
// stable radix sort of 15-bit keys (two 8-bit digits) by one block, warp w on
// the w-th contiguous segment, so that the order does not depend on timing.
// perm receives it (tmp: scratch of M). One block, 5 to 7 ns a point: 0.8% of a
// registration of 40,097 points; emicp_sort_pays and emicp_team_sorts say where not.
__device__ __forceinline__ void em_sort(const float* __restrict__ Y, int M, unsigned* keys, int* perm, int* tmp) {
  constexpr int kW = 32, kDig = 256;
  __shared__ float s_lo[3][kW], s_hi[3][kW];
  __shared__ int s_cnt[kDig * kW];  // [digit][warp]
  __shared__ int s_sum[kW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = 3.0e38f;
    hi[k] = -3.0e38f;
  }
  for (int i = tid; i < M; i += 1024)
    for (int k = 0; k < 3; ++k) {
      const float y = Y[(size_t)k * M + i];
      lo[k] = fminf(lo[k], y);
      hi[k] = fmaxf(hi[k], y);
    }
  for (int k = 0; k < 3; ++k) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[k] = fminf(lo[k], __shfl_down_sync(0xffffffffu, lo[k], off));
      hi[k] = fmaxf(hi[k], __shfl_down_sync(0xffffffffu, hi[k], off));
    }
    if (lane == 0) {
      s_lo[k][warp] = lo[k];
      s_hi[k][warp] = hi[k];
    }
  }
  __syncthreads();
  float ext = 0.f;
  for (int k = 0; k < 3; ++k) {
    lo[k] = s_lo[k][0];
    hi[k] = s_hi[k][0];
    for (int w = 1; w < kW; ++w) {
      lo[k] = fminf(lo[k], s_lo[k][w]);
      hi[k] = fmaxf(hi[k], s_hi[k][w]);
    }
    ext = fmaxf(ext, hi[k] - lo[k]);
  }
  const float inv = ext > 0.f ? 32.f / ext : 0.f;
  for (int i = tid; i < M; i += 1024) {
    unsigned c[3];
    for (int k = 0; k < 3; ++k)  // (a coordinate that is not finite lands in some cell: only locality is at stake)
      c[k] = (unsigned)min(31, max(0, (int)((Y[(size_t)k * M + i] - lo[k]) * inv)));
    keys[i] = hilbert_index(c);
  }
  const int seg = ((M + kW - 1) / kW + 31) & ~31;
  const int sb = min(warp * seg, M), se = min(sb + seg, M);
  for (int pass = 0; pass < 2; ++pass) {
    const int shift = 8 * pass;
    const int* from = pass ? tmp : nullptr;  // pass 0 reads in index order
    int* to = pass ? perm : tmp;
    for (int i = tid; i < kDig * kW; i += 1024) s_cnt[i] = 0;
    __syncthreads();
    for (int i0 = sb; i0 < se; i0 += 32) {
      const bool in = i0 + lane < se;
      const unsigned act = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int id = from ? from[i0 + lane] : i0 + lane;
        const int d = (int)(keys[id] >> shift) & 255;
        const unsigned same = __match_any_sync(act, d);
        if (lane == __ffs((int)same) - 1) s_cnt[d * kW + warp] += __popc(same);
      }
      __syncwarp();
    }
    __syncthreads();
    // exclusive scan over (digit, warp): 8 entries a thread
    int v[8], sum = 0;
    for (int k = 0; k < 8; ++k) {
      v[k] = s_cnt[tid * 8 + k];
      sum += v[k];
    }
    int inc = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += n;
    }
    if (lane == 31) s_sum[warp] = inc;
    __syncthreads();
    int base = inc - sum;
    for (int w = 0; w < warp; ++w) base += s_sum[w];
    for (int k = 0; k < 8; ++k) {
      s_cnt[tid * 8 + k] = base;
      base += v[k];
    }
    __syncthreads();
    for (int i0 = sb; i0 < se; i0 += 32) {
      const bool in = i0 + lane < se;
      const unsigned act = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int id = from ? from[i0 + lane] : i0 + lane;
        const int d = (int)(keys[id] >> shift) & 255;
        const unsigned same = __match_any_sync(act, d);
        const int at = s_cnt[d * kW + warp] + __popc(same & ((1u << lane) - 1u));
        __syncwarp(act);
        if (lane == __ffs((int)same) - 1) s_cnt[d * kW + warp] += __popc(same);
        to[at] = id;
      }
      __syncwarp();
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024) em_sort_kernel(const float* __restrict__ Y, int M, unsigned* keys, int* perm,
                                                       int* tmp) {
  em_sort(Y, M, keys, perm, tmp);
}

// Y' in the order perm (null: as given): (y - o, index in the caller's order).
__device__ __forceinline__ void em_pack_rows(const float* __restrict__ Y, int M, const CenterHdr* hdr,
                                             const int* __restrict__ perm, float4* __restrict__ out) {
  const float* o = hdr->oY;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < M; r += gridDim.x * blockDim.x) {
    const int i = perm ? perm[r] : r;
    out[r] = make_float4(__fsub_rn(Y[i], o[0]), __fsub_rn(Y[M + i], o[1]), __fsub_rn(Y[2 * M + i], o[2]),
                         __int_as_float(i));
  }
}

__global__ void em_pack_rows_kernel(const float* __restrict__ Y, int M, const CenterHdr* hdr,
                                    const int* __restrict__ perm, float4* __restrict__ out) {
  em_pack_rows(Y, M, hdr, perm, out);
}

// Centre of an owned block's (blockIdx.x) bounding box and its points' largest
// distance from it (NaN where a coordinate is not finite).
__device__ __forceinline__ void em_block(const float4* __restrict__ rows, int M, float4* __restrict__ out) {
  constexpr int kW = kBlockPts / 32;
  __shared__ float s_lo[3][kW], s_hi[3][kW], s_r[kW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * kBlockPts + threadIdx.x;
  const float4 y = rows[min(r, M - 1)];  // the last block's padding repeats its last point
  float lo[3] = {y.x, y.y, y.z}, hi[3] = {y.x, y.y, y.z};
  for (int k = 0; k < 3; ++k) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], off));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], off));
    }
    if (lane == 0) {
      s_lo[k][warp] = lo[k];
      s_hi[k][warp] = hi[k];
    }
  }
  __syncthreads();
  float c[3];
  for (int k = 0; k < 3; ++k) {
    float l = s_lo[k][0], h = s_hi[k][0];
    for (int w = 1; w < kW; ++w) {
      l = fminf(l, s_lo[k][w]);
      h = fmaxf(h, s_hi[k][w]);
    }
    c[k] = 0.5f * (l + h);
  }
  const float dx = y.x - c[0], dy = y.y - c[1], dz = y.z - c[2];
  float d = sqrtf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)));
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_xor_sync(0xffffffffu, d, off);
    d = (o > d || o != o) ? o : d;
  }
  if (lane == 0) s_r[warp] = d;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kW; ++w) d = (s_r[w] > d || s_r[w] != s_r[w]) ? s_r[w] : d;
    out[blockIdx.x] = make_float4(c[0], c[1], c[2], d);
  }
}

__global__ void __launch_bounds__(kBlockPts) em_block_kernel(const float4* __restrict__ rows, int M,
                                                            float4* __restrict__ out) {
  em_block(rows, M, out);
}

// The same for the pairs of a batch.
struct TeamPrep {
  const float* Y;
  int M;
  const CenterHdr* hdr;
  unsigned* keys;
  int* perm;
  float4* rows;
  float4* blk;
};

__global__ void __launch_bounds__(1024) em_sort_teams_kernel(const TeamPrep* __restrict__ tab) {
  const TeamPrep P = tab[blockIdx.x];
  if (P.perm) em_sort(P.Y, P.M, P.keys, P.perm, P.perm + P.M);
}

__global__ void em_pack_teams_kernel(const TeamPrep* __restrict__ tab) {
  const TeamPrep P = tab[blockIdx.y];
  em_pack_rows(P.Y, P.M, P.hdr, P.perm, P.rows);
}

__global__ void __launch_bounds__(kBlockPts) em_block_teams_kernel(const TeamPrep* __restrict__ tab) {
  const TeamPrep P = tab[blockIdx.y];
  if ((int)blockIdx.x * kBlockPts >= P.M) return;
  if (!P.perm) {  // unsorted: no block counts as compact
    if (threadIdx.x == 0) P.blk[blockIdx.x] = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fc00000));
    return;
  }
  em_block(P.rows, P.M, P.blk);
}

// ------------------------------------------------------------------ host side

namespace {
struct Carve {
  char* p;
  size_t off = 0;
  explicit Carve(void* base) : p(static_cast<char*>(base)) {}
  template <class T>
  T* take(size_t n) {
    off = (off + 255) & ~size_t(255);
    T* r = p ? reinterpret_cast<T*>(p + off) : nullptr;
    off += n * sizeof(T);
    return r;
  }
};

struct EmicpPlan {
  int grid;
  SweepGeom geo;
  size_t smem;
  bool local;  // sorted Y, local sweeps, refined poses
  bool rows;   // small clouds: whole rows to a block, X in shared memory
};

size_t sweep_smem() { return sizeof(SweepSmem); }

constexpr int kEmPairNum = 208;  // SM pairs: the favoured block's share, 13 / 16

// The others take the local sweep, with the sort that it wants and refined poses,
// where that ends sooner over the whole schedule. Its shorter element saves 4.9e-5
// ns of an affinity (40,097^2: 5.2 ms of 36), a refined pose costs 1.7 us a step, the
// sort, by one block, 5 to 7 ns a row. Hence 4.6e7 affinities a step, and 1.35e5 columns
// over all steps for a row. Default schedule, direct / local (ms): 9000 x 4000 1.59 / 1.63, x 6000
// 2.11 / 2.07, 20,000 x 2000 1.71 / 1.73, x 3000 2.26 / 2.20, 2000 x 50,000 3.83 / 3.82, 2500 x 40,000
// 4.30 / 4.08, 1000 x 400,000 11.6 / 13.5, 30 x 10^6 8.2 / 16.0; 16 steps: 3500 x 30,000 1.07 /
// 1.10, 20,000 x 3000 0.60 / 0.59; one step of 40,097^2 0.78 / 0.91.
// (Never for a single step: it returns its rows, whose sums direct differences leave nearer to
// FP64 at small sigma: 2.2e-7 against 3.8e-7 rms at 10,007 x 9001, sigma_p2 = 1e-4; no refined
// pose makes up for them.)
bool emicp_sort_pays(int N, long nsteps) { return nsteps > 1 && (double)N * (double)nsteps >= 1.35e5; }
bool emicp_local_pays(int N, int M, long nsteps) {
  return (double)N * (double)M >= 4.6e7 && emicp_sort_pays(N, nsteps);
}

// A batch's pairs are sorted side by side, a block each: it is not worth it only
// for long thin ones (one pair alone, unsorted against sorted and lock step, ms: 10 x
// 32,000 1.05 / 1.40 / 1.30, 400 x 32,000 1.38 / 1.67 / 1.59, 129 x 190,001 2.72 / 3.87 / 3.17, 300 x 100,000
// 2.47 / 3.03 / 2.65; 20 pairs of 400 x 32,000 11.4 / 10.9 / 11.2, of 800 x 32,000 18.2 / 16.9 / 17.0).
bool emicp_team_sorts(int N, int M, long nsteps) {
  return M <= 8192 || (M <= 32768 && N >= 500) || emicp_sort_pays(N, nsteps);
}

// Rows of a block in the small clouds' form, 0 where it is not taken: X has to
// fit shared memory beside a second block's, and up to 6e7 affinities a step the
// barrier that it saves is worth more than the local sweep's shorter element
// (general or local form -> this, both without refined poses, us: 100^2 664 -> 379, 600 x
// 500 581 -> 410, 1007^2 591 -> 426, 2000^2 734 -> 568, 4001^2 1086 -> 996, 6000 x 5000
// 1475 -> 1386, 8171 x 6007 1897 -> 1679; 8000 x 9000 2401 -> 2420; the refinement
// adds about 60). A whole number of passes of 4 rows; 8 rather than 4 where that
// leaves one block to an SM (1007: 448 -> 426).
int emicp_small_rows(int N, int M, int limit) {
  if (N > kRowsMaxN || (double)N * (double)M >= 6e7) return 0;
  int own = (M + 4 * limit - 1) / (4 * limit) * 4;
  if (own == 4 && M > 2 * limit) own = 8;
  // many rows against few columns: a block's passes take longer than the slices' second
  // barrier (ms, slices against this: 16 x 7000 0.735 / 0.751, 100 x 9000 0.773 / 0.801, 200 x 9728 0.799
  // / 0.814, 600 x 9000 0.862 / 0.926, 1600 x 9728 1.104 / 1.159; but 16 x 5000 0.735 / 0.691, 300 x 9728
  // 0.857 / 0.815, 1000 x 8000 0.942 / 0.871, 2000 x 9700 1.206 / 1.169)
  const bool thin = (own > 20 && N < 64) || (own > 24 && N < 128) ||
                    (own > 28 && (N < 224 || (N > 512 && N < 2000)));
  return own <= kRowsOwn && !thin ? own : 0;
}

EmicpPlan plan_emicp_as(int N, int M, bool local, int device) {
  EmicpPlan P;
  P.smem = sweep_smem();
  const int limit = persistent_grid_limit(device, (const void*)emicp_kernel, P.smem);
  P.local = P.rows = false;
  const int own =
      emicp_small_rows(N, M, persistent_grid_limit(device, (const void*)emicp_rows_kernel<kSmall>, rows_smem(kRowsMaxN)));
  if (own > 0) {
    P.rows = true;
    P.smem = rows_smem(N);
    P.grid = (M + own - 1) / own;
    P.geo = SweepGeom{M, N, 0, 0, own, 0, 0, 0, 0, 0};
    return P;
  }
  P.local = local;
  const SweepGeomH h = plan_sweep(M, N, limit);
  P.geo = SweepGeom{h.n_own, h.n_stream, h.nblk, h.slices, h.slice_len, h.units, 0, 0, 0, 0};
  P.grid = h.units < limit ? h.units : limit;
  // Large clouds: contiguous task ranges, the same work per block to one
  // chunk of 512 streamed points, instead of units dealt in waves; with two
  // blocks on every SM, each SM's pair splits its range 13 : 3, the larger
  // part to the block the SM favours.
  // (The query also sets the kernel's shared-memory limit.)
  const bool ranges = ranged_pays(h.nblk, N, limit) &&
                      (P.local || persistent_grid_limit(device, (const void*)emicp_ranges_kernel, P.smem) >= limit);
  if (ranges) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const char* ev = getenv("CESA_SM_PAIRS");  // "0": equal shares (for comparisons)
    if (sms > 0 && limit == 2 * sms && !(ev && ev[0] == '0')) P.geo.pair_num = kEmPairNum;
    make_ranged(P.geo, limit);
    P.grid = limit;
  }
  return P;
}

struct EmicpCarved {
  Ctl* ctl;
  CenterHdr* hdr;
  float4* rows;
  float4* cols;
  float4* xs;
  float4* blk;
  unsigned* keys;
  int* perm;
  float* part;
  df* rbpart;
  unsigned* pair_tab;
  float* pair_t;
  int Mp;
};

EmicpCarved carve_emicp(void* base, const EmicpPlan& P, int N, int M, size_t* total) {
  Carve c(base);
  EmicpCarved w;
  w.Mp = (M + 3) & ~3;
  w.ctl = c.take<Ctl>(1);
  w.hdr = c.take<CenterHdr>(1);
  w.rows = c.take<float4>((size_t)M);
  w.cols = c.take<float4>((size_t)N);
  w.xs = c.take<float4>(P.geo.ranged && !P.local ? (size_t)2 * N : 0);
  w.blk = c.take<float4>(P.local ? (size_t)P.geo.nblk : 0);
  w.part = c.take<float>(P.geo.ranged ? (size_t)5 * P.geo.nblk * P.geo.kmax * kBlockPts
                                      : (size_t)5 * P.geo.slices * w.Mp);
  // the sort's keys (M) and orders (2 M) lie where the sweeps' partials, at least 5 M
  // words, are written later: a sorted registration takes no more than one that is not
  w.keys = reinterpret_cast<unsigned*>(w.part);
  w.perm = reinterpret_cast<int*>(w.part) + M;
  w.rbpart = c.take<df>((size_t)2 * P.grid * kEmNV);
  w.pair_tab = c.take<unsigned>(P.geo.pair_num ? 2 * kPairCap + 1 : 0);
  w.pair_t = c.take<float>(P.geo.pair_num ? (size_t)P.grid : 0);
  if (total) *total = c.off;
  return w;
}

// cap: the workspace at hand. Sorted rows over slices want 16 bytes a block more
// than unsorted ones; where only those fit, they run.
EmicpPlan plan_emicp(int N, int M, long nsteps, int device, size_t cap = SIZE_MAX) {
  EmicpPlan P = plan_emicp_as(N, M, emicp_local_pays(N, M, nsteps), device);
  size_t total = 0;
  carve_emicp(nullptr, P, N, M, &total);
  if (P.local && total > cap) P = plan_emicp_as(N, M, false, device);
  return P;
}
}  // namespace

void emicp_ws_views(void* ws, int N, int M, long nsteps, int device, CenterHdr** hdr, float4** rows, float4** cols) {
  const EmicpPlan P = plan_emicp(N, M, nsteps, device);
  EmicpCarved w = carve_emicp(ws, P, N, M, nullptr);
  *hdr = w.hdr;
  *rows = w.rows;
  *cols = w.cols;
}

int emicp_form(int N, int M, long nsteps, int device) {
  const EmicpPlan P = plan_emicp(N, M, nsteps, device);
  return P.rows         ? CESA_EMICP_FORM_ROWS
         : P.local      ? CESA_EMICP_FORM_LOCAL
         : P.geo.ranged ? CESA_EMICP_FORM_RANGES
                        : CESA_EMICP_FORM_SLICES;
}

size_t emicp_ws_need(int N, int M, long nsteps, int device, size_t cap) {
  const EmicpPlan P = plan_emicp(N, M, nsteps, device, cap);
  size_t total = 0;
  carve_emicp(nullptr, P, N, M, &total);
  return total;
}

int enqueue_emicp(const EmicpLaunch& L, void* ws, size_t ws_bytes, cudaStream_t st, int* grid_used) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const EmicpPlan P = plan_emicp(L.N, L.M, L.nsteps, device, ws_bytes);
  size_t total = 0;
  EmicpCarved w = carve_emicp(ws, P, L.N, L.M, &total);
  if (total > ws_bytes) return (int)cudaErrorInvalidValue;
  if (grid_used) *grid_used = P.grid;
  // the control block starts at zero every launch
  e = cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), st);
  if (e == cudaSuccess && P.geo.pair_num)
    e = cudaMemsetAsync(w.pair_tab, 0, sizeof(unsigned) * (2 * kPairCap + 1), st);
  if (e != cudaSuccess) return (int)e;
  prep_center_kernel<<<1, 1024, 0, st>>>(L.dX, L.N, L.dY, L.M, w.hdr);
  const int pb = 256, pg_x = (L.N + pb - 1) / pb, pg_y = (L.M + pb - 1) / pb;
  prep_pack_kernel<<<pg_x < 1024 ? pg_x : 1024, pb, 0, st>>>(L.dX, L.N, w.hdr, 0, 0.f, w.cols);
  if (P.local) {
    em_sort_kernel<<<1, 1024, 0, st>>>(L.dY, L.M, w.keys, w.perm, w.perm + L.M);
    em_pack_rows_kernel<<<pg_y < 1024 ? pg_y : 1024, pb, 0, st>>>(L.dY, L.M, w.hdr, w.perm, w.rows);
    em_block_kernel<<<P.geo.nblk, kBlockPts, 0, st>>>(w.rows, L.M, w.blk);
  } else {
    em_pack_rows_kernel<<<pg_y < 1024 ? pg_y : 1024, pb, 0, st>>>(L.dY, L.M, w.hdr, nullptr, w.rows);
  }
  e = cudaGetLastError();
  // ranged partial slots that no block writes must read as zero (after the sort,
  // which uses the same memory)
  if (e == cudaSuccess && P.geo.ranged)
    e = cudaMemsetAsync(w.part, 0, sizeof(float) * 5 * (size_t)P.geo.nblk * P.geo.kmax * kBlockPts, st);
  if (e != cudaSuccess) return (int)e;
  if (L.nsteps <= 0) return 0;

  EmicpArgs A;
  A.rows = w.rows;
  A.cols = w.cols;
  A.M = L.M;
  A.N = L.N;
  A.geo = P.geo;
  A.sigma0 = L.sigma_p2;
  A.sigma_factor = L.sigma_factor;
  A.d_02 = L.d_02;
  A.nsteps = L.nsteps;
  A.hdr = w.hdr;
  A.dRt = L.dRt;
  A.part = w.part;
  A.xs = w.xs;
  A.blk = P.local ? w.blk : nullptr;
  A.refine = 0;
  A.Mp = w.Mp;
  A.rbpart = w.rbpart;
  A.ctl = w.ctl;
  A.pair_tab = w.pair_tab;
  A.pair_t = w.pair_t;
  A.trace = L.trace;
  A.trace_cap = L.trace_cap;
  A.row_out = L.row_out;
  A.tape = L.tape;
  A.row_tape = L.row_tape;
  A.d_status = L.d_status;
  A.tl = L.timeline;
  A.tl_cap = L.timeline_cap;
  A.timeout_ns = L.timeout_ns;
  void* args[] = {(void*)&A};
  const void* kernel = P.rows                     ? (const void*)emicp_rows_kernel<kSmall>
                       : P.geo.ranged && !P.local ? (const void*)emicp_ranges_kernel
                                                  : (const void*)emicp_kernel;
  if (P.rows && L.row_out) {
    kernel = (const void*)emicp_rows_kernel<kSmallOut>;
    if (persistent_grid_limit(device, kernel, rows_smem(kRowsMaxN)) < P.grid) return (int)cudaErrorCooperativeLaunchTooLarge;
  }
  e = cudaLaunchCooperativeKernel(kernel, dim3(P.grid), dim3(kThreads), args, P.smem, st);
  return (int)e;
}

namespace {
struct TeamsCarved {
  Ctl* ctl;  // one per job; cleared, as are the ranged partials behind them
  unsigned* pair_tab;
  size_t zero_bytes, total;
  EmicpArgs* args;
  TeamPrep* prep;
  TeamBlock* blocks;
  std::vector<EmicpArgs> hargs;
  std::vector<TeamPrep> hprep;
};

TeamsCarved carve_teams(void* base, const EmTeamJob* jobs, int n, const TeamPlan& P, bool pairs,
                        uint64_t timeout_ns) {
  TeamsCarved w;
  Carve c(base);
  w.ctl = c.take<Ctl>((size_t)n);
  w.pair_tab = c.take<unsigned>(pairs ? 2 * kPairCap + 1 : 0);
  if (!pairs) w.pair_tab = nullptr;
  w.hargs.resize((size_t)n);
  w.hprep.resize((size_t)n);
  for (int j = 0; j < n; ++j) {
    const EmTeamJob& J = jobs[P.order[(size_t)j]];
    EmicpArgs& A = w.hargs[(size_t)j];
    A = EmicpArgs{};
    const int g = P.size[(size_t)j];
    const SweepGeomH h = plan_sweep(J.M, J.N, g);
    A.geo = SweepGeom{h.n_own, h.n_stream, h.nblk, h.slices, h.slice_len, h.units, 0, 0, 0, 0};
    {
      if (pairs && g % 2 == 0) A.geo.pair_num = kEmPairNum;
      make_ranged(A.geo, g);
    }
    A.cols = J.cols;
    A.M = J.M;
    A.N = J.N;
    A.sigma0 = J.sigma_p2;
    A.sigma_factor = J.sigma_factor;
    A.d_02 = J.d_02;
    A.nsteps = J.nsteps;
    A.hdr = J.hdr;
    A.dRt = J.dRt;
    A.Mp = (J.M + 3) & ~3;
    A.ctl = w.ctl ? w.ctl + j : nullptr;
    A.timeout_ns = timeout_ns;
    if (A.geo.ranged) A.part = c.take<float>((size_t)5 * A.geo.nblk * A.geo.kmax * kBlockPts);
  }
  w.zero_bytes = c.off;
  w.args = c.take<EmicpArgs>((size_t)n);
  w.prep = c.take<TeamPrep>((size_t)n);
  w.blocks = c.take<TeamBlock>(P.blocks.size());
  for (int j = 0; j < n; ++j) {
    const EmTeamJob& J = jobs[P.order[(size_t)j]];
    EmicpArgs& A = w.hargs[(size_t)j];
    if (!A.geo.ranged) A.part = c.take<float>((size_t)5 * A.geo.slices * A.Mp);
    A.rbpart = c.take<df>((size_t)2 * P.size[(size_t)j] * kEmNV);
    A.pair_t = c.take<float>((size_t)P.size[(size_t)j]);
    const bool sorted = emicp_team_sorts(J.N, J.M, J.nsteps);
    A.refine = sorted;
    float4* blk = c.take<float4>((size_t)A.geo.nblk);
    unsigned* keys = sorted ? c.take<unsigned>((size_t)J.M) : nullptr;
    int* perm = sorted ? c.take<int>((size_t)2 * J.M) : nullptr;
    float4* rows = c.take<float4>((size_t)J.M);
    A.rows = rows;
    A.blk = blk;
    w.hprep[(size_t)j] = TeamPrep{J.dY, J.M, J.hdr, keys, perm, rows, blk};
  }
  w.total = c.off;
  return w;
}

int teams_grid(int device, bool* pairs) {
  const int G = persistent_grid_limit(device, (const void*)emicp_teams_kernel, sweep_smem());
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  *pairs = sms > 0 && G == 2 * sms;
  return G;
}
}  // namespace

size_t emicp_teams_ws_need(const EmTeamJob* jobs, int n, int device, TeamPlan* plan) {
  if (n < 1) return 0;
  bool pairs = false;
  *plan = plan_teams(jobs, n, teams_grid(device, &pairs));
  return carve_teams(nullptr, jobs, n, *plan, pairs, 0).total;
}

int enqueue_emicp_teams(const EmTeamJob* jobs, int n, const TeamPlan& P, void* ws, size_t ws_bytes, void* ctl,
                        uint64_t timeout_ns, cudaStream_t st) {
  if (n < 1) return 0;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  bool pairs = false;
  const int G = teams_grid(device, &pairs);
  if ((int)P.order.size() != n) return (int)cudaErrorInvalidValue;
  TeamsCarved w = carve_teams(ws, jobs, n, P, pairs, timeout_ns);
  if (w.total > ws_bytes || (int)P.blocks.size() != G) return (int)cudaErrorInvalidValue;
  int max_blk = 1;
  for (const EmicpArgs& A : w.hargs) max_blk = A.geo.nblk > max_blk ? A.geo.nblk : max_blk;
  e = cudaMemsetAsync(ws, 0, w.zero_bytes, st);
  if (e == cudaSuccess)
    e = put_table(w.args, w.hargs.data(), sizeof(EmicpArgs) * (size_t)n, st);
  if (e == cudaSuccess)
    e = put_table(w.prep, w.hprep.data(), sizeof(TeamPrep) * (size_t)n, st);
  if (e == cudaSuccess)
    e = put_table(w.blocks, P.blocks.data(), sizeof(TeamBlock) * P.blocks.size(), st);
  if (e != cudaSuccess) return (int)e;
  em_sort_teams_kernel<<<n, 1024, 0, st>>>(w.prep);
  em_pack_teams_kernel<<<dim3(16, n), 256, 0, st>>>(w.prep);
  em_block_teams_kernel<<<dim3(max_blk, n), kBlockPts, 0, st>>>(w.prep);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  const EmicpArgs* jobs_d = w.args;
  const TeamBlock* blocks_d = w.blocks;
  Ctl* main_ctl = static_cast<Ctl*>(ctl);
  void* args[] = {(void*)&jobs_d, (void*)&n, (void*)&blocks_d, (void*)&main_ctl, (void*)&w.pair_tab, (void*)&timeout_ns};
  return (int)cudaLaunchCooperativeKernel((const void*)emicp_teams_kernel, dim3(G), dim3(kThreads), args, sweep_smem(),
                                          st);
}

int read_ws_status(void* ws, cudaStream_t st, int* status, int* steps, int* tl_written) {
  Ctl h;
  cudaError_t e = cudaMemcpyAsync(&h, ws, sizeof(Ctl), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return (int)e;
  if (status) *status = h.status;
  if (steps) *steps = h.steps_done;
  if (tl_written) *tl_written = (int)h.pad[0];
  return 0;
}

namespace {
struct TableChunk {
  unsigned w[896];
};
__global__ void table_chunk_kernel(unsigned* dst, int n, const __grid_constant__ TableChunk c) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = c.w[i];
}
}  // namespace

cudaError_t put_table(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
  if (cap != cudaStreamCaptureStatusActive) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  if (bytes % sizeof(unsigned)) return cudaErrorInvalidValue;
  for (size_t at = 0; at < bytes; at += sizeof(TableChunk)) {
    TableChunk c;
    const size_t len = bytes - at < sizeof(c) ? bytes - at : sizeof(c);
    memcpy(c.w, static_cast<const char*>(src) + at, len);
    table_chunk_kernel<<<1, 256, 0, st>>>(reinterpret_cast<unsigned*>(static_cast<char*>(dst) + at),
                                          (int)(len / sizeof(unsigned)), c);
  }
  return cudaGetLastError();
}

// Smem opt-in and occupancy for a persistent kernel: blocks per SM x SMs.
int persistent_grid_limit(int device, const void* kernel, size_t smem) {
  // SM count per device, filled on first use; each entry is written once with
  // its device's own value, so concurrent callers on other devices cannot mix
  // them up.
  static std::atomic<int> sms_of[64];
  int sms = 0;
  if (device >= 0 && device < 64) sms = sms_of[device].load(std::memory_order_relaxed);
  if (sms <= 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (device >= 0 && device < 64 && sms > 0) sms_of[device].store(sms, std::memory_order_relaxed);
  }
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 2) per_sm = 2;
  return per_sm * (sms > 0 ? sms : 1);
}

// Unit decomposition over the split S. Modelled time, in element
// evaluations of one block (~20 per ns): waves x (unit work + fixed cost per
// unit: streamed-chunk latency, reductions) + the completion of split owned
// blocks (partials written, the last unit loads S partials per accumulator,
// 16 in flight).
SweepGeomH plan_sweep(int n_own, int n_stream, int grid_limit) {
  SweepGeomH best{};
  const int nblk = (n_own + kBlockPts - 1) / kBlockPts;
#ifndef CESA_UNIT_FIXED_COST
#define CESA_UNIT_FIXED_COST 40000.0  // per-unit cost in element evaluations of one block
#endif
  const double fixed = CESA_UNIT_FIXED_COST;
  double best_cost = 1e300;
  const int smax_stream = (n_stream + 31) / 32;
  const int smax = smax_stream < 128 ? smax_stream : 128;
  for (int S = 1; S <= (smax > 0 ? smax : 1); ++S) {
    const int slice_len = (n_stream + S - 1) / S;
    const int s_eff = (n_stream + slice_len - 1) / slice_len;
    if (s_eff != S) continue;
    const long units = (long)nblk * S;
    const int grid = units < grid_limit ? (int)units : grid_limit;
    const long waves = (units + grid - 1) / grid;
    const double split = S > 1 ? 30000.0 + 15000.0 * ((S + 15) / 16) : 0.0;
    const double cost = (double)waves * ((double)kBlockPts * slice_len + fixed) + split;
    if (cost < best_cost * 0.999) {
      best_cost = cost;
      best = SweepGeomH{n_own, n_stream, nblk, S, slice_len, (int)units};
    }
  }
  if (best.units == 0) best = SweepGeomH{n_own, n_stream, nblk, 1, n_stream, nblk};
  return best;
}

}  // namespace cesa
