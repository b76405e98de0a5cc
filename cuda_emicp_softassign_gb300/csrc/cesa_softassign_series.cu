// Series form of the Softassign pose updates (sm_103a): while the temperature
// is high against the extent of the clouds, every Sinkhorn sum over the N x M
// affinities is a short polynomial, and a pose update costs O(N + M).
//
// With both clouds about their means (x = X' - cX, z = R (Y' - cY)) and
// delta = R cY + t' - cX,
//   K_rc = e^(alpha/T) / sqrt(T) e^(-|x_r - z_c - delta|^2 / T)
//        = 2^c0 F_r G_c e^(2 x_r.z_c / T),
//   F_r = e^(-|x_r - delta|^2 / T),  G_c = e^(-(|z_c|^2 + 2 z_c.delta) / T),
// and e^(u.v) = sum_|k|<=D u^k v^k / k! over the monomials of three variables.
// The truncation is at most q^(D+1)/(D+1)! e^q of a term, q = 2 max|x| max|z| / T
// (independent of the pose): D is the smallest degree (2..8, or up to what the
// caller gives: 6 beside the banded kernel, 4 there on unequal counts) for which
// that is below 2^-25, half an FP32 unit in the last place, or 2e-9 for clouds of
// unequal counts (kTolEqual, kTolUnequal). A row pass is then: the
// P = C(D+3, 3) moments sum_c b_c G_c v_c^k of the columns, and per row the
// polynomial sum_k (moment_k / k!) u_r^k; a column pass likewise. The default
// schedule on scans of 0.2 extent (alignScaleOnce's scale) has q from 4e-4 at
// T = 100 to 0.06 at T = 0.6: D = 2..4, P = 10..35, in place of 20,000 exponentials
// per row. An update whose q, exponents or offset leave the range (also NaN)
// ends the kernel; the affinity kernels take the schedule up from there
// (SeriesHand), so every input still runs.
//
// One thread-block cluster of 1-16 CTAs runs all updates. Rows and columns
// stay in shared memory, cut evenly over the CTAs; a pass's moments are summed
// per warp through shared memory, per CTA, pushed to every CTA's slots by
// remote stores and, after one cluster barrier, added in rank order by each CTA
// itself: 2 I1 + 2 exchanges an update. Scalings, slack, the moments of the
// final sweep and the pose are those of the affinity kernels
// (src/softassign.cu:494-798), the scalings and the slack as (hi, lo) pairs.
// What bounds it is latency: an update is a chain of ~8 exchanges and the
// fixed-order sums before and after each, up to some 2000 points, and from there on the
// points' polynomials too (2 P FMAs per point and pass). us an update at D = 2, 4 and 6:
// N = M = 100 10.4, 12.6, 16.6; 413 12.4, 14.6, 18.0; 2000 13.9, 17.3, 23.1; 7001 17.2, 22.9, 33.0; 20,000
// 25.0, 34.2, 51.4. Default schedule, affinity kernels -> this: N = M = 413 20.1 -> 6.6
// ms, 2000 12.9 -> 7.4, 20,000 461 -> 13.6; 30 updates from T = 0.1 at 7001 x 6007
// 4.25 -> 1.2 to 1.6, and 2.5 where a pair's extent leaves the last ones to the affinity
// kernels (8 pairs).
#include <mutex>
#include <vector>

#include "cesa_kernels.h"
#include "cesa_ops.cuh"
#include "cesa_pose.h"
#include "cesa_prep.cuh"
#include "cesa_sa_pose.cuh"

namespace cesa {

constexpr int kSerThreads = 512;
constexpr int kSerWarps = kSerThreads / 32;
constexpr int kSerMaxD = 8;
constexpr int kSerMaxCS = 16;
__host__ __device__ constexpr int ser_terms(int D) { return (D + 1) * (D + 2) * (D + 3) / 6; }
constexpr int kSerPs = (ser_terms(kSerMaxD) + 3) & ~3;       // 168: a polynomial's coefficients
constexpr int kSerPf = (ser_terms(kSerMaxD + 1) + 3) & ~3;  // 220: the final sweep's moments, one degree more
constexpr int kSerSets = 5;                    // the final sweep's weighted sums
constexpr int kSerRedRows = 16;                // a warp's transpose buffer: [16][36] floats
constexpr int kSerRedLd = 36;

struct SeriesArgs {
  const float4* rows;  // X' centred (N)
  const float4* cols;  // Y' centred (M)
  const CenterHdr* hdr;
  const float* dRt;    // the pose, caller frame (read)
  const float* s_in;   // initial slack, or null: moutlier
  const float* u_in;
  float* s_out;        // slack after the last update done here
  float* u_out;
  SeriesHand* hand;
  int N, M, nr, nc;    // nr, nc: rows and columns per CTA
  int JMAX, I0, I1;
  float alpha, T0, TFACTOR, moutlier;
  int max_degree;
  float* state;        // optional: pose (12, centred) and temperature reached
  float* dRt_out;      // optional: the final pose, when the whole schedule ran here
  Ctl* ctl;
  double* trace;
  int trace_cap;
};

// Dynamic shared memory, in floats from the base (every part 16-byte aligned):
// fixed parts, then the state of this CTA's points.
constexpr int kLPose = 0;                                // the pose (12), centred frame
constexpr int kLHdr = kLPose + 12;                       // oX, oY, mean(Y'), mean(X')
constexpr int kLTot = kLHdr + 12;                        // [32] dfs: the pose's moments
constexpr int kLRef = kLTot + 64;                        // reference weights: columns' G, their W, rows' W; then a
                                                         // pass's constant term (hi, lo)
constexpr int kLWtab = kLRef + 8;                        // [threads] dfs: 2^c0 of the coming temperatures
constexpr int kLCoef = kLWtab + 2 * kSerThreads;         // 1 / k!
constexpr int kLTab = kLCoef + kSerPs;                   // positions of k and k + e_x, e_y, e_z among the terms of one
                                                         // degree more, a byte each
constexpr int kLM = kLTab + kSerPs;                      // [5][kSerPs] coefficients of the polynomials being evaluated
constexpr int kLWsum = kLM + kSerSets * kSerPs;          // [2][warps][kSerPf] per-warp sums; zero for warps without points
constexpr int kLWd = kLWsum + 2 * kSerWarps * kSerPf;    // [warps][32] dfs, likewise
constexpr int kLSlot = kLWd + kSerWarps * 64;            // [2][16][kSerPs] every CTA's moments of a pass, by parity; zero
                                                         // for CTAs that are not there
constexpr int kLFin = kLSlot + 2 * kSerMaxCS * kSerPs;   // [2][kSerPf] this CTA's moments of the final sweep, read by the cluster
constexpr int kLRaw = kLFin + 2 * kSerPf;                // [2][kSerPf] the cluster's
constexpr int kLSlotD = kLRaw + 2 * kSerPf;              // [16][32] dfs: every CTA's moments of the pose
constexpr int kLRed = kLSlotD + kSerMaxCS * 64;          // [warps][16][36]
constexpr int kLState = kLRed + kSerWarps * kSerRedRows * kSerRedLd;
static_assert(kSerWarps == 16 && kSerMaxCS == 16, "sums of 16");

// State arrays: rows x', W, s; columns y', v, W, u, cs (W, s, u and cs as
// (hi, lo) pairs in two arrays each). A row's W is its scaling times its factor
// of K, 2^c0 a_r F_r, a column's b_c G_c: the weights that a pass sums, and what
// its sums are multiplied with.
constexpr int kRW = 3, kRs = 5, kRowArr = 7;
constexpr int kCv = 3, kCW = 6, kCu = 8, kCcs = 10, kColArr = 12;

namespace {

__device__ __forceinline__ void st_dsmem(const float* p, unsigned rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dsmem_addr(p, rank)), "f"(v) : "memory");
}
// (float2: the store wants 8-byte alignment)
__device__ __forceinline__ void st_dsmem2(const float2* p, unsigned rank, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dsmem_addr(p, rank)), "f"(a), "f"(b) : "memory");
}

// 16 bytes of shared memory; volatile, so that a loop over points does not keep
// every coefficient in a register (and spill the rest).
__device__ __forceinline__ float4 ld_smem4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

// Polynomial of degree D in (x, y, z) by nested Horner steps; m: coefficients
// in evaluation order (a, b, c descending), 16-byte aligned.
template <int D>
__device__ __forceinline__ float poly_eval(const float* m, float x, float y, float z) {
  const uint32_t m4 = smem_u32(m);
  float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
  int idx = 0;
  float r = 0.f;
#pragma unroll
  for (int a = D; a >= 0; --a) {
    float s = 0.f;
#pragma unroll
    for (int b = D - a; b >= 0; --b) {
      float t = 0.f;
#pragma unroll
      for (int c = D - a - b; c >= 0; --c) {
        if ((idx & 3) == 0) w = ld_smem4(m4 + 4u * (unsigned)idx);
        const float v = (idx & 3) == 0 ? w.x : (idx & 3) == 1 ? w.y : (idx & 3) == 2 ? w.z : w.w;
        t = c == D - a - b ? v : fmaf(t, z, v);
        ++idx;
      }
      s = b == D - a ? t : fmaf(s, y, t);
    }
    r = a == D ? s : fmaf(r, x, s);
  }
  return r;
}

// Position of monomial x^a y^b z^c in evaluation order: the terms of higher a,
// then of higher b, then of higher c (tetrahedral and triangular counts).
template <int D>
__host__ __device__ constexpr int mono_index(int a, int b, int c) {
  return (D - a) * (D - a + 1) * (D - a + 2) / 6 + (D - a - b) * (D - a - b + 1) / 2 + (D - a - b - c);
}

// acc[i - LO] += g x^a y^b z^c for the monomials of positions [LO, LO + NV);
// the constant term's addend is g0.
template <int D, int LO, int NV>
__device__ __forceinline__ void mono_add(float g, float g0, float x, float y, float z, float (&acc)[NV]) {
  float xa = g;
#pragma unroll
  for (int a = 0; a <= D; ++a) {
    float yb = xa;
#pragma unroll
    for (int b = 0; b <= D - a; ++b) {
      float zc = yb;
#pragma unroll
      for (int c = 0; c <= D - a - b; ++c) {
        const int i = mono_index<D>(a, b, c);
        if (i >= LO && i < LO + NV) acc[i - LO < 0 ? 0 : (i - LO >= NV ? NV - 1 : i - LO)] += i == ser_terms(D) - 1 ? g0 : zc;
        if (c < D - a - b) zc *= z;
      }
      if (b < D - a) yb *= y;
    }
    if (a < D) xa *= x;
  }
}

// Sums of NV <= 16 values over the warp's lanes, each in a fixed order, to
// dst[0 .. NV): through the warp's transpose buffer.
template <int NV>
__device__ __forceinline__ void warp_sum16(const float* v, float* buf, float* dst) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NV; ++k) buf[k * kSerRedLd + lane] = v[k];
  __syncwarp();
  constexpr int PER = NV > 8 ? 16 : 8;  // lane % PER: the value, lane / PER: its part of PER entries
  const int row = lane % PER, part = lane / PER;
  float s = 0.f;
  if (row < NV) {
    const float4* p = reinterpret_cast<const float4*>(buf + row * kSerRedLd + part * PER);
    float4 q[PER / 4];
#pragma unroll
    for (int k = 0; k < PER / 4; ++k) q[k] = p[k];
#pragma unroll
    for (int w = PER / 8; w >= 1; w >>= 1)
#pragma unroll
      for (int k = 0; k < w; ++k) {
        q[k].x += q[k + w].x;
        q[k].y += q[k + w].y;
        q[k].z += q[k + w].z;
        q[k].w += q[k + w].w;
      }
    s = (q[0].x + q[0].y) + (q[0].z + q[0].w);
  }
#pragma unroll
  for (int off = 16; off >= PER; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (lane < NV) dst[lane] = s;
  __syncwarp();
}

// Sums of NV (17..32) values over the warp's lanes: a first exchange leaves the
// low half-warp with values 0-15 and the high one with values 16-31, so that
// all of them fit the buffer at once.
template <int NV>
__device__ __forceinline__ void warp_sum32(const float* v, float* buf, float* dst) {
  const int lane = threadIdx.x & 31;
  const bool high = lane >= 16;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float a = v[k], b = k + 16 < NV ? v[k + 16] : 0.f;
    const float o = __shfl_xor_sync(0xffffffffu, high ? a : b, 16);
    buf[k * kSerRedLd + lane] = (high ? b : a) + o;
  }
  __syncwarp();
  const float4* p = reinterpret_cast<const float4*>(buf + (lane & 15) * kSerRedLd + (lane & 16));
  float4 q[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) q[k] = p[k];
#pragma unroll
  for (int w = 2; w >= 1; w >>= 1)
#pragma unroll
    for (int k = 0; k < w; ++k) {
      q[k].x += q[k + w].x;
      q[k].y += q[k + w].y;
      q[k].z += q[k + w].z;
      q[k].w += q[k + w].w;
    }
  const float s = (q[0].x + q[0].y) + (q[0].z + q[0].w);
  if (lane < NV) dst[lane] = s;
  __syncwarp();
}

// The same for any NV, up to 32 at a time.
template <int NV>
__device__ __forceinline__ void warp_sum(const float* v, float* buf, float* dst) {
  if constexpr (NV <= 16)
    warp_sum16<NV>(v, buf, dst);
  else
    warp_sum32<(NV > 32 ? 32 : NV)>(v, buf, dst);
  if constexpr (NV > 32) warp_sum<NV - 32>(v + 32, buf, dst + 32);
}

// delta = R cY + t' - cX: the means' distance under the pose.
__device__ __forceinline__ void series_delta(const float* pose, const float* hdr, float (&dl)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k)
    dl[k] = pose[3 * k] * hdr[6] + pose[3 * k + 1] * hdr[7] + pose[3 * k + 2] * hdr[8] + (pose[9 + k] - hdr[9 + k]);
}

// The block's dynamic shared memory.
__device__ __forceinline__ float* ser_mem() {
  extern __shared__ __align__(16) float ser_smem[];
  return ser_smem;
}

__device__ __forceinline__ float* at(int o) { return ser_mem() + o; }

// The block's context: this CTA's share of the points (state arrays of nrp and
// ncp entries).
struct Ser {
  int N, M, nr, nc;  // the clouds, this CTA's rows and columns
  int nrp, ncp;
  int nt;  // threads that hold points (whole warps)
  int CS;
  unsigned rank;
  unsigned par;  // parity of the next pass's slots
  __device__ __forceinline__ float* row(int k) const { return at(kLState + k * nrp); }
  __device__ __forceinline__ float* col(int k) const { return at(kLState + kRowArr * nrp + k * ncp); }
  // (hi, lo) state value k of point i
  __device__ __forceinline__ df rowd(int k, int i) const { return df{row(k)[i], row(k + 1)[i]}; }
  __device__ __forceinline__ df cold(int k, int i) const { return df{col(k)[i], col(k + 1)[i]}; }
  __device__ __forceinline__ void rowd(int k, int i, df v) const {
    row(k)[i] = v.hi;
    row(k + 1)[i] = v.lo;
  }
  __device__ __forceinline__ void cold(int k, int i, df v) const {
    col(k)[i] = v.hi;
    col(k + 1)[i] = v.lo;
  }
};

// The scalings and the slack are (hi, lo) pairs: a row's s is divided by its
// row sum in every pass of every update (1500 times in the default schedule),
// where the assignment is nearly uniform and only the variation of the
// scalings carries information. FP32 rounding of each sum would walk s away by
// far more than one pass's error.

// e^x, with the part below FP32 where x is small (e^x - 1 rounded once).
__device__ __forceinline__ df dd_exp(float x) {
  return fabsf(x) < 0.5f ? dd_fast(1.f, expm1f(x)) : df_make(expf(x));
}

// Per-warp moments of one set over the n points of this CTA, into
// wsum[warp][kSerPf]; pt(i, x, y, z, g0) gives point i's coordinates and its
// term of the constant moment, and returns its weight. Warps of the nt threads without a point write zeros.
// The terms are taken in groups of at most 60 accumulators.
template <int D, int LO, class Pt>
__device__ __forceinline__ void moments_group(const Ser& S, int n, float* wsum, const Pt& pt) {
  constexpr int P = ser_terms(D);
  constexpr int NV = P - LO > 60 ? 32 : P - LO;
  const int warp = threadIdx.x >> 5;
  float acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = 0.f;
  for (int i = threadIdx.x; i < n; i += S.nt) {
    float x, y, z, g0;
    const float g = pt(i, x, y, z, g0);
    mono_add<D, LO, NV>(g, g0, x, y, z, acc);
  }
  float* buf = at(kLRed) + warp * kSerRedRows * kSerRedLd;
  float* dst = wsum + warp * kSerPf + LO;
  warp_sum<NV>(acc, buf, dst);
  if constexpr (LO + NV < P) moments_group<D, LO + NV>(S, n, wsum, pt);
}

template <int D, class Pt>
__device__ __forceinline__ void warp_moments(const Ser& S, int n, float* wsum, const Pt& pt) {
  if ((int)threadIdx.x < S.nt) moments_group<D, 0>(S, n, wsum, pt);
}

// Sum of 16 values ld apart, fixed tree (the per-warp sums or the CTAs' slots;
// absent ones hold zeros).
__device__ __forceinline__ float sum16(const float* p, int ld) {
  float q[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) q[k] = p[k * ld];
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
    for (int k = 0; k < w; ++k) q[k] += q[k + w];
  return q[0];
}
__device__ __forceinline__ df sum16d(const float* p) {  // 16 dfs 64 floats apart
  df q[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float2 w = *reinterpret_cast<const float2*>(p + 64 * k);
    q[k] = df{w.x, w.y};
  }
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
    for (int k = 0; k < w; ++k) df_add(q[k], q[k + w]);
  return q[0];
}

__device__ __forceinline__ void ser_sync(const Ser& S) {
  if (S.CS > 1)
    cluster_sync_all();
  else
    __syncthreads();
}

// Threads that share a term's remote stores (each adds its sum itself).
__host__ __device__ constexpr int push_threads(int P) { return 2 * P <= kSerThreads ? 2 : 1; }

// Moments of one pass over this CTA's points, all CTAs' added in rank order
// and divided by k!: the polynomial's coefficients in L.m. The constant term is
// kept apart (returned; its place in L.m is 0) and to more than FP32: its
// addends are the weights' differences from a reference weight, ref[which],
// which every CTA knows and the nearly uniform weights are close to, and the
// ntot references are added back as a (hi, lo) pair. The mean weight is the
// next such pass's reference.
template <int D, class Pt>
__device__ __forceinline__ df pass_moments(Ser& S, int n, int ntot, int which, const Pt& pt) {
  constexpr int P = ser_terms(D);
  const int t = threadIdx.x;
  float* ws = at(kLWsum);
  warp_moments<D>(S, n, ws, pt);
  __syncthreads();
  float* slots = at(kLSlot) + S.par * kSerMaxCS * kSerPs;
  S.par ^= 1u;
  // into this CTA's slot of every CTA: kPush threads to a term, each for every
  // kPush-th CTA, as a loop: unrolled over 16 CTAs the stores were mostly code to
  // fetch (100 points 6.37 -> 5.45 ms, 413 7.09 -> 6.52, 2000 7.83 -> 7.40, 20,000
  // 14.1 -> 13.7; with 16 or 4 threads to a term 20,000 took 14.4 and 13.8)
  constexpr int kPush = push_threads(P);
  if (t < P * kPush) {
    const int k = t / kPush;
    const float s = sum16(ws + k, kSerPf);
    const float* dst = slots + S.rank * kSerPs + k;
#pragma unroll 1
    for (int r = t % kPush; r < S.CS; r += kPush) st_dsmem(dst, (unsigned)r, s);
  }
  ser_sync(S);
  float* m = at(kLM);
  if (t < P) {
    const float s = sum16(slots + t, kSerPs) * at(kLCoef)[t];
    m[t] = t == P - 1 ? 0.f : s;
  } else if (t == kSerThreads - 1) {  // the constant term, in a warp of its own
    float* ref = at(kLRef);
    const float c = ref[which], nf = (float)ntot;
    df k = df_make(0.f);
    df_add_prod(k, nf, c);
    df_add(k, sum16(slots + P - 1, kSerPs));
    k = dd_fast(k.hi, k.lo);
    ref[4] = k.hi;
    ref[5] = k.lo;
    const float mean = __fdividef(k.hi, nf);
    ref[which] = fabsf(mean) < 1e30f ? mean : 0.f;
  }
  __syncthreads();
  return df{at(kLRef)[4], at(kLRef)[5]};
}

// Tables of degree D: 1/(a! b! c!) in evaluation order, and where a term and
// its three neighbours of one degree more stand among the terms of degree D + 1.
template <int D>
__device__ __forceinline__ void fill_tables(float* coef, uint32_t* tab) {
  const int t = threadIdx.x;
  if (t < ser_terms(D)) {
    int idx = 0;
    for (int a = D; a >= 0; --a)
      for (int b = D - a; b >= 0; --b)
        for (int c = D - a - b; c >= 0; --c, ++idx)
          if (idx == t) {
            float f = 1.f;
            for (int k = 2; k <= a; ++k) f *= (float)k;
            for (int k = 2; k <= b; ++k) f *= (float)k;
            for (int k = 2; k <= c; ++k) f *= (float)k;
            coef[t] = 1.f / f;
            tab[t] = (uint32_t)mono_index<D + 1>(a, b, c) | (uint32_t)mono_index<D + 1>(a + 1, b, c) << 8 |
                     (uint32_t)mono_index<D + 1>(a, b + 1, c) << 16 | (uint32_t)mono_index<D + 1>(a, b, c + 1) << 24;
          }
  }
}

// Sums over the warp's lanes of 32 df values, 8 at a time (value lane % 8,
// part lane / 8).
__device__ __forceinline__ void warp_sum_df32(const df* v, float* buf, df* dst) {
  const int lane = threadIdx.x & 31;
  constexpr int LD = 34;  // dfs per row
  static_assert(8 * LD * 2 <= kSerRedRows * kSerRedLd, "transpose buffer");
  float2* b2 = reinterpret_cast<float2*>(buf);
  const int row = lane & 7, part = lane >> 3;
#pragma unroll
  for (int g = 0; g < 32; g += 8) {
#pragma unroll
    for (int k = 0; k < 8; ++k) b2[k * LD + lane] = make_float2(v[g + k].hi, v[g + k].lo);
    __syncwarp();
    const float4* p = reinterpret_cast<const float4*>(b2 + row * LD + part * 8);
    df q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 w = p[k];
      q[k] = df{w.x, w.y};
      df_add(q[k], df{w.z, w.w});
    }
    df_add(q[0], q[2]);
    df_add(q[1], q[3]);
    df_add(q[0], q[1]);
#pragma unroll
    for (int off = 16; off >= 8; off >>= 1) {
      const df o = df_shfl_down(q[0], off);
      df_add(q[0], o);
    }
    if (lane < 8) dst[g + lane] = q[0];
    __syncwarp();
  }
}

// One row's contribution to the 28 row-side moments (the slots of
// sa_row_moments), with w as a (hi, lo) pair: the unequal part of two clouds'
// counts leaves sum w x V a large term that w's FP32 rounding would not cancel.
// kFirst: v holds nothing yet, and the products are its values.
template <bool kFirst>
__device__ __forceinline__ void series_row_moments(df (&v)[32], df w, float mu, const float (&V)[3],
                                                   const float (&xp)[3]) {
  auto add = [&](int k, float x, float lo) {
    if (kFirst) {
      v[k] = df{x, lo};
    } else {
      df_add(v[k], x);
      v[k].lo = __fadd_rn(v[k].lo, lo);
    }
  };
  auto prod = [&](int k, float x, float xl, float y) {  // (x + xl) y
    const float p = __fmul_rn(x, y);
    add(k, p, __fmaf_rn(xl, y, __fmaf_rn(x, y, -p)));
  };
  const df w2 = dd_mul(w, w);
  const float wmu = w.hi * mu;
  add(0, w.hi, w.lo);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    prod(1 + i, w.hi, w.lo, xp[i]);
    const float wx = w.hi * xp[i];
#pragma unroll
    for (int j = 0; j < 3; ++j) prod(4 + i + 3 * j, wx, 0.f, V[j]);
    add(13 + i, V[i], 0.f);
    prod(16 + i, wmu, 0.f, xp[i]);
    prod(20 + i, w2.hi, w2.lo, xp[i]);
    prod(24 + i, w.hi, 0.f, V[i]);
  }
  add(19, mu, 0.f);
  add(23, w2.hi, w2.lo);
  prod(27, w.hi, 0.f, mu);
}

// One pose update up to its 32 moments (L.tot, every CTA the same).
template <int D>
__device__ __noinline__ void series_update(Ser& Sg, df wsc, int I1, float lam, float T) {
  Ser S = Sg;
  const int tid = threadIdx.x;
  const bool live = tid < S.nt;
  const float* pose = at(kLPose);
  const float* hdr = at(kLHdr);
  const float rT = 1.f / T;
  const float vs = 2.f / (T * lam);  // u = lam x, v = vs z: u.v = 2 x.z / T
  const float cx = hdr[9], cy = hdr[10], cz = hdr[11];
  const float yh0 = hdr[6], yh1 = hdr[7], yh2 = hdr[8];
  float *x0 = S.row(0), *x1 = S.row(1), *x2 = S.row(2);
  float *y0 = S.col(0), *y1 = S.col(1), *y2 = S.col(2), *v0 = S.col(kCv), *v1 = S.col(kCv + 1), *v2 = S.col(kCv + 2);
  const float* m = at(kLM);
  if (live) {
    float dl[3];
    series_delta(pose, hdr, dl);
    for (int i = tid; i < S.nr; i += S.nt) {
      const float x = x0[i] - cx - dl[0], y = x1[i] - cy - dl[1], z = x2[i] - cz - dl[2];
      S.rowd(kRW, i, dd_mul(dd_exp(-rT * fmaf(z, z, fmaf(y, y, x * x))), wsc));
    }
    for (int j = tid; j < S.nc; j += S.nt) {
      const float x = y0[j] - yh0, y = y1[j] - yh1, z = y2[j] - yh2;
      const float zx = pose[0] * x + pose[1] * y + pose[2] * z;
      const float zy = pose[3] * x + pose[4] * y + pose[5] * z;
      const float zz = pose[6] * x + pose[7] * y + pose[8] * z;
      const float e = fmaf(zx, fmaf(2.f, dl[0], zx), fmaf(zy, fmaf(2.f, dl[1], zy), zz * fmaf(2.f, dl[2], zz)));
      S.cold(kCW, j, dd_exp(-rT * e));
      v0[j] = zx * vs;
      v1[j] = zy * vs;
      v2[j] = zz * vs;
    }
  }
  // a point's sum over K, its weight W (constant + rest) + slack
  auto point_sum = [&](df W, df m0, float rest, df slack) {
    df p = dd_sum(m0.hi, rest);
    p.lo = __fadd_rn(p.lo, m0.lo);
    const df t = dd_mul(W, p);
    const df r = dd_sum(t.hi, slack.hi);
    return dd_fast(r.hi, __fadd_rn(r.lo, __fadd_rn(t.lo, slack.lo)));
  };
  // (each thread reads back only what it wrote itself, here and below)
  const float* ref = at(kLRef);
  for (int k = 0; k < I1; ++k) {
    // row pass k (normalizeMbySinkhorn_row + Saxpy, src/softassign.cu:538-561):
    // rs = a_old (row sum of K b) + s_old, a = a_old / rs, s = s_old / rs
    const float rc = ref[k == 0 ? 0 : 1];
    const df mr = pass_moments<D>(S, S.nc, S.M, k == 0 ? 0 : 1, [&](int j, float& x, float& y, float& z, float& g0) {
      x = v0[j];
      y = v1[j];
      z = v2[j];
      const df g = S.cold(kCW, j);
      g0 = (g.hi - rc) + g.lo;
      return g.hi;
    });
    if (live)
      for (int i = tid; i < S.nr; i += S.nt) {
        const float p = poly_eval<D>(m, (x0[i] - cx) * lam, (x1[i] - cy) * lam, (x2[i] - cz) * lam);
        const df W = S.rowd(kRW, i), so = S.rowd(kRs, i);
        const df sum = point_sum(W, mr, p, so);
        const float inv = dd_inv(sum);
        S.rowd(kRW, i, dd_div(W, sum, inv));
        S.rowd(kRs, i, dd_div(so, sum, inv));
      }
    // column pass k (src/softassign.cu:579-597), likewise
    const float rr = ref[2];
    const df mc = pass_moments<D>(S, S.nr, S.N, 2, [&](int i, float& x, float& y, float& z, float& g0) {
      x = (x0[i] - cx) * lam;
      y = (x1[i] - cy) * lam;
      z = (x2[i] - cz) * lam;
      const df g = S.rowd(kRW, i);
      g0 = (g.hi - rr) + g.lo;
      return g.hi;
    });
    if (live)
      for (int j = tid; j < S.nc; j += S.nt) {
        const float p = poly_eval<D>(m, v0[j], v1[j], v2[j]);
        const df W = S.cold(kCW, j), uo = S.cold(kCu, j);
        const df sum = point_sum(W, mc, p, uo);
        const float inv = dd_inv(sum);
        S.cold(kCW, j, dd_div(W, sum, inv));
        S.cold(kCu, j, dd_div(uo, sum, inv));
        S.cold(kCcs, j, sum);
      }
  }
  // The final sweep's sums (see FinalElem): over K b, K b (cs - 1) and
  // K b cs (y' - Yhat). With y' - Yhat = R^T z the last three are moments of one
  // degree more of b cs = b + b (cs - 1): two sets of moments of degree D + 1.
  const float rc = ref[1];
#pragma unroll 1
  for (int q = 0; q < 2; ++q) {
    warp_moments<D + 1>(S, S.nc, at(kLWsum) + q * kSerWarps * kSerPf,
                        [&](int j, float& x, float& y, float& z, float& g0) {
                          x = v0[j];
                          y = v1[j];
                          z = v2[j];
                          const df W = S.cold(kCW, j);
                          if (q == 0) {
                            g0 = (W.hi - rc) + W.lo;
                            return W.hi;
                          }
                          const df cs = S.cold(kCcs, j);
                          g0 = W.hi * ((cs.hi - 1.f) + cs.lo);
                          return g0;
                        });
  }
  __syncthreads();
  constexpr int P1 = ser_terms(D + 1);
  static_assert(2 * P1 <= kSerThreads, "one thread per moment");
  if (tid < 2 * P1) {
    const int q = tid >= P1, t = tid - q * P1;
    at(kLFin)[q * kSerPf + t] = sum16(at(kLWsum) + q * kSerWarps * kSerPf + t, kSerPf);
  }
  ser_sync(S);
  {
    float* raw = at(kLRaw);
    if (tid < 2 * P1) {
      const int q = tid >= P1, t = tid - q * P1;
      const float* src = at(kLFin) + q * kSerPf + t;
      float v[kSerMaxCS];
#pragma unroll
      for (int r = 0; r < kSerMaxCS; ++r) v[r] = r < S.CS ? ld_dsmem(src, (unsigned)r) : 0.f;
#pragma unroll
      for (int w = kSerMaxCS / 2; w >= 1; w >>= 1)
#pragma unroll
        for (int r = 0; r < w; ++r) v[r] += v[r + w];
      raw[q * kSerPf + t] = v[0];
    }
    __syncthreads();
    if (tid < ser_terms(D)) {
      const float c = at(kLCoef)[tid], cv = c / vs;
      const uint32_t w = reinterpret_cast<const uint32_t*>(at(kLTab))[tid];
      float* mo = at(kLM) + tid;
      const float r0 = raw[w & 255u];  // the constant term: see pass_moments
      mo[0] = tid == ser_terms(D) - 1 ? 0.f : r0 * c;
      mo[kSerPs] = raw[kSerPf + (w & 255u)] * c;
      if (tid == ser_terms(D) - 1) {
        df k = df_make(0.f);
        df_add_prod(k, (float)S.M, rc);
        df_add(k, r0);
        k = dd_fast(k.hi, k.lo);
        at(kLRef)[4] = k.hi;
        at(kLRef)[5] = k.lo;
      }
#pragma unroll
      for (int e = 1; e <= 3; ++e) {
        const uint32_t i = (w >> (8 * e)) & 255u;
        mo[(1 + e) * kSerPs] = (raw[i] + raw[kSerPf + i]) * cv;
      }
    }
    __syncthreads();
  }
  df v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = df_make(0.f);
  const df w0{at(kLRef)[4], at(kLRef)[5]};
  auto row_moments = [&](int i, auto first) {
    const float xp[3] = {x0[i], x1[i], x2[i]};
    const float x = (xp[0] - cx) * lam, y = (xp[1] - cy) * lam, z = (xp[2] - cz) * lam;
    float p5[kSerSets];
#pragma unroll
    for (int q = 0; q < kSerSets; ++q) p5[q] = poly_eval<D>(m + q * kSerPs, x, y, z);
    const df ad = S.rowd(kRW, i);
    df w = dd_sum(w0.hi, p5[0]);
    w.lo = __fadd_rn(w.lo, w0.lo);
    w = dd_mul(ad, w);
    const float ar = ad.hi;
    float V[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) V[k] = ar * (pose[k] * p5[2] + pose[3 + k] * p5[3] + pose[6 + k] * p5[4]);
    series_row_moments<decltype(first)::value>(v, w, ar * p5[1], V, xp);
  };
  if (live && tid < S.nr) row_moments(tid, std::true_type{});
#pragma unroll 1
  for (int i = tid + S.nt; live && i < S.nr; i += S.nt) row_moments(i, std::false_type{});
  for (int j = tid; live && j < S.nc; j += S.nt) {
    const float csv = S.col(kCcs)[j];
    const float csl = S.col(kCcs + 1)[j];
    const float yy[3] = {y0[j], y1[j], y2[j]};
    df_add(v[28], df{csv, csl});
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      df_add_prod(v[29 + k], csv, yy[k]);
      v[29 + k].lo = __fmaf_rn(csl, yy[k], v[29 + k].lo);
    }
  }
  float* wd = at(kLWd);
  if (live) {
    const int warp = tid >> 5;
    warp_sum_df32(v, at(kLRed) + warp * kSerRedRows * kSerRedLd, reinterpret_cast<df*>(wd) + warp * 32);
  }
  __syncthreads();
  float2* slotD = reinterpret_cast<float2*>(at(kLSlotD));
  static_assert(kLSlotD % 2 == 0, "pairs");
  if (tid < 32 * 4) {
    const int k = tid & 31;
    const df s = sum16d(wd + 2 * k);
#pragma unroll 1
    for (int r = tid >> 5; r < S.CS; r += 4) st_dsmem2(slotD + S.rank * 32 + k, (unsigned)r, s.hi, s.lo);
  }
  ser_sync(S);
  if (tid < 32) reinterpret_cast<df*>(at(kLTot))[tid] = sum16d(at(kLSlotD) + 2 * tid);
  __syncthreads();
  Sg.par = S.par;
}

// max that keeps a NaN.
__device__ __forceinline__ float nan_max(float a, float b) { return b > a || b != b ? b : a; }

// Smallest degree for which the truncated series stays within tol of every
// affinity (see the head of this file), 0 when none up to max_degree does.
__device__ __forceinline__ int series_degree(float q, int max_degree, float tol) {
  if (!(q < 2.f)) return 0;
  float term = q * q * q * (1.f / 6.f) * expf(q);
  for (int D = 2; D <= max_degree; ++D) {
    if (term <= tol) return D;
    term *= q / (float)(D + 2);
  }
  return 0;
}

}  // namespace

// Truncation, relative to an affinity: half an FP32 unit in the last place. Clouds
// of unequal counts leave part of every sum to the slack, which the pose's S has to
// cancel, and the truncation, of one sign in all terms, shows there: they take 1/15
// of it (7001 x 6007, 30 updates from T = 0.1, the worst of 12 pairs against FP64: 1.5e-6
// with the larger, 9.7e-7 with the smaller, 2.2e-6 with the affinity kernels; 1.33 and
// 1.55 ms).
constexpr float kTolEqual = 2.98e-8f, kTolUnequal = 2e-9f;

// The updates of one pair, by one cluster.
__device__ __forceinline__ void series_run(const SeriesArgs& A) {
  __shared__ float2 s_rad[kSerMaxCS];
  __shared__ float s_wr[2][kSerWarps];
  __shared__ SaPoseScratch ps;
  __shared__ HornState<float> horn;
  const int tid = threadIdx.x;
  Ser S;
  S.CS = (int)cluster_nctarank();
  S.rank = cluster_ctarank();
  // a cluster that does not hold the points' shares (the same answer in every
  // CTA) leaves before any cluster barrier or remote access
  if (S.CS > kSerMaxCS || (long)S.CS * A.nr < A.N || (long)S.CS * A.nc < A.M) {
    if (tid == 0) set_status(A.ctl, kStatusUnsupported, 80);
    return;
  }
  S.nrp = (A.nr + 3) & ~3;
  S.ncp = (A.nc + 3) & ~3;
  const int r0 = (int)S.rank * A.nr, c0 = (int)S.rank * A.nc;
  S.N = A.N;
  S.M = A.M;
  S.nr = max(0, min(A.nr, A.N - r0));
  S.nc = max(0, min(A.nc, A.M - c0));
  S.nt = 32 * min(kSerWarps, (max(A.nr, A.nc) + 31) >> 5);
  for (int i = tid; i < kLState - kLWsum; i += kSerThreads) at(kLWsum)[i] = 0.f;
  S.par = 0;
  float* s_pose = at(kLPose);
  float* s_hdr = at(kLHdr);
  if (tid == 0) {
    for (int k = 0; k < 3; ++k) {
      s_hdr[k] = A.hdr->oX[k];
      s_hdr[3 + k] = A.hdr->oY[k];
      s_hdr[6 + k] = A.hdr->ymean[k];
      s_hdr[9 + k] = A.hdr->xmean[k];
    }
    float R[9], t[3], tc[3];
    for (int k = 0; k < 9; ++k) R[k] = A.dRt[k];
    for (int k = 0; k < 3; ++k) t[k] = A.dRt[9 + k];
    pose_to_centred(R, t, &s_hdr[0], &s_hdr[3], tc);
    for (int k = 0; k < 9; ++k) s_pose[k] = R[k];
    for (int k = 0; k < 3; ++k) s_pose[9 + k] = tc[k];
    float* ref = at(kLRef);
    ref[0] = 1.f;
    ref[1] = ref[2] = 0.f;
    horn.reset();
  }
  __syncthreads();
  float rx = 0.f, ry = 0.f;  // largest squared distances from the means (NaN stays NaN)
  for (int i = tid; i < S.nr; i += kSerThreads) {
    const float4 p = ld_cg(A.rows + r0 + i);
    S.row(0)[i] = p.x;
    S.row(1)[i] = p.y;
    S.row(2)[i] = p.z;
    S.rowd(kRs, i, df_make(A.s_in ? A.s_in[r0 + i] : A.moutlier));
    const float x = p.x - s_hdr[9], y = p.y - s_hdr[10], z = p.z - s_hdr[11];
    const float d = fmaf(z, z, fmaf(y, y, x * x));
    rx = nan_max(rx, d);
  }
  for (int j = tid; j < S.nc; j += kSerThreads) {
    const float4 p = ld_cg(A.cols + c0 + j);
    S.col(0)[j] = p.x;
    S.col(1)[j] = p.y;
    S.col(2)[j] = p.z;
    S.cold(kCu, j, df_make(A.u_in ? A.u_in[c0 + j] : A.moutlier));
    const float x = p.x - s_hdr[6], y = p.y - s_hdr[7], z = p.z - s_hdr[8];
    const float d = fmaf(z, z, fmaf(y, y, x * x));
    ry = nan_max(ry, d);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float a = __shfl_xor_sync(0xffffffffu, rx, off), b = __shfl_xor_sync(0xffffffffu, ry, off);
    rx = nan_max(rx, a);
    ry = nan_max(ry, b);
  }
  if ((tid & 31) == 0) {
    s_wr[0][tid >> 5] = rx;
    s_wr[1][tid >> 5] = ry;
  }
  // the first remote stores wait until every CTA of the cluster has started
  ser_sync(S);
  if (tid == 0) {
    for (int w = 1; w < kSerWarps; ++w) {
      rx = nan_max(rx, s_wr[0][w]);
      ry = nan_max(ry, s_wr[1][w]);
    }
    for (int r = 0; r < S.CS; ++r) st_dsmem2(&s_rad[S.rank], (unsigned)r, rx, ry);
  }
  ser_sync(S);
  rx = s_rad[0].x;
  ry = s_rad[0].y;
  for (int r = 1; r < S.CS; ++r) {
    rx = nan_max(rx, s_rad[r].x);
    ry = nan_max(ry, s_rad[r].y);
  }
  rx = sqrtf(rx) * 1.0001f;
  ry = sqrtf(ry) * 1.0001f;

  float T = A.T0;
  int step = 0, Dc = 0, tit = 0, it0 = 0;
  bool on = true;
  for (tit = 0; tit < A.JMAX; ++tit) {
    const float kk = kLog2e / T;
    const float c0e = fmaf(A.alpha, kk, -0.5f * log2f(T));
    if (tit % kSerThreads == 0) {  // 2^c0 = e^(alpha / T) / sqrt(T) of the next temperatures, one per thread
      __syncthreads();
      if (tid < A.JMAX - tit) {
        float Tk = T;
        for (int k = 0; k < tid; ++k) Tk = Tk * A.TFACTOR;
        const double w = exp((double)A.alpha / (double)Tk) / sqrt((double)Tk);
        const float hi = (float)w;
        at(kLWtab)[2 * tid] = hi;
        at(kLWtab)[2 * tid + 1] = (float)(w - (double)hi);
      }
      __syncthreads();
    }
    const df wsc{at(kLWtab)[2 * (tit % kSerThreads)], at(kLWtab)[2 * (tit % kSerThreads) + 1]};
    const int D = series_degree(2.f * rx * ry / T, A.max_degree, A.N == A.M ? kTolEqual : kTolUnequal);
    // u = lam x and v = (2 / (T lam)) z have the same largest norm, sqrt(q) < 1.5
    const float lam = rx > 0.f && ry > 0.f ? sqrtf(2.f * ry / (T * rx)) : sqrtf(2.f / T);
    it0 = 0;
    on = D > 0 && fabsf(c0e) < 95.f && lam > 1e-30f && lam < 1e30f;
    if (!on) break;
    for (it0 = 0; it0 < A.I0; ++it0, ++step) {
      float dl[3];
      series_delta(s_pose, s_hdr, dl);
      // every exponent of F and G stays well inside FP32's range
      const float far = rx + ry + sqrtf(dl[0] * dl[0] + dl[1] * dl[1] + dl[2] * dl[2]);
      on = kk * far * far < 40.f;
      if (!on) break;
#define CESA_SERIES_CASE(d)                                                                \
  case d:                                                                                  \
    if (Dc != d) {                                                                         \
      __syncthreads();                                                                     \
      fill_tables<d>(at(kLCoef), reinterpret_cast<uint32_t*>(at(kLTab)));          \
      Dc = d;                                                                              \
    }                                                                                      \
    series_update<d>(S, wsc, A.I1, lam, T);                                                \
    break;
      switch (D) {
        CESA_SERIES_CASE(2)
        CESA_SERIES_CASE(3)
        CESA_SERIES_CASE(4)
        CESA_SERIES_CASE(5)
        CESA_SERIES_CASE(6)
        CESA_SERIES_CASE(7)
        CESA_SERIES_CASE(8)
      }
#undef CESA_SERIES_CASE
      double* trace_rec = (A.trace && step < A.trace_cap) ? A.trace + (size_t)step * 32 : nullptr;
      sa_pose_update<true>(reinterpret_cast<const df*>(at(kLTot)), s_hdr, ps, horn, s_pose, S.rank == 0, nullptr, trace_rec, step, T, A.ctl, nullptr, true,
                           tit == A.JMAX - 1 && it0 == A.I0 - 1);
    }
    if (!on) break;
    T = T * A.TFACTOR;  // FP32, src/softassign.cu:820
  }
  if (on) it0 = 0;  // the schedule ran to its end: tit == JMAX
  for (int i = tid; i < S.nr; i += kSerThreads) A.s_out[r0 + i] = S.row(kRs)[i];
  for (int j = tid; j < S.nc; j += kSerThreads) A.u_out[c0 + j] = S.col(kCu)[j];
  if (S.rank == 0 && tid == 0) {
    A.hand->titer = tit;
    A.hand->iter0 = it0;
    for (int k = 0; k < 12; ++k) A.hand->pose[k] = s_pose[k];
    if (A.state) {
      for (int k = 0; k < 12; ++k) A.state[k] = s_pose[k];
      A.state[12] = T;
    }
    if (A.dRt_out && on) {
      float R[9], t[3], tc[3];
      for (int k = 0; k < 9; ++k) R[k] = s_pose[k];
      for (int k = 0; k < 3; ++k) tc[k] = s_pose[9 + k];
      pose_from_centred(R, tc, &s_hdr[0], &s_hdr[3], t);
      for (int k = 0; k < 9; ++k) A.dRt_out[k] = R[k];
      for (int k = 0; k < 3; ++k) A.dRt_out[9 + k] = t[k];
    }
  }
  if (S.CS > 1) cluster_sync_all();  // no CTA leaves while a peer may still write its shared memory
}

__global__ void __launch_bounds__(kSerThreads, 1) softassign_series_kernel(const SeriesArgs A) { series_run(A); }

// A batch's launches (one per cluster size) run side by side: each may start
// once all CTAs of the one before have started, and none completes before it.
__global__ void __launch_bounds__(kSerThreads, 1) softassign_series_batch_kernel(const SeriesArgs* tab) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  series_run(tab[cluster_id_x()]);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ------------------------------------------------------------------ host side
namespace {
constexpr size_t kSerSmemMax = 220 * 1024;  // of 227 KB; the rest is static
constexpr int kSerBatchPts = 1536;          // most points per CTA in a batch
static_assert(sizeof(float) * ((size_t)kLState + (size_t)(kRowArr + kColArr) * kSerBatchPts) <= kSerSmemMax, "fits");

struct SeriesPlan {
  int CS = 0, nr = 0, nc = 0;
  size_t smem = 0;
};

// The least power of two of CTAs, up to max_cluster, that leaves each at most
// `pts` points of a cloud (0: the choice for one pair alone); CS = 0 where the
// points do not fit.
SeriesPlan plan_series(int N, int M, int max_cluster, int pts = 0) {
  SeriesPlan P;
  if (max_cluster < 1) return P;
  const int n = N > M ? N : M;
  int CS = 1;
  // one pair: 128 up to 512 points (7.0 against 7.2 ms with 256 at N = M =
  // 413), else 256 (7.7 against 7.7 with 128 and 9.0 with 512 at 2000)
  if (pts == 0) pts = n <= 512 ? 128 : 256;
  while (2 * CS <= max_cluster && (n + CS - 1) / CS > pts) CS *= 2;
  const int nr = (N + CS - 1) / CS, nc = (M + CS - 1) / CS;
  const size_t smem =
      sizeof(float) * ((size_t)kLState + (size_t)kRowArr * ((nr + 3) & ~3) + (size_t)kColArr * ((nc + 3) & ~3));
  if (smem > kSerSmemMax) return P;
  P.CS = CS;
  P.nr = nr;
  P.nc = nc;
  P.smem = smem;
  return P;
}
}  // namespace

int softassign_series_cluster(int N, int M, int max_cluster) {
  if (N < 1 || M < 1 || N >= (1 << 24) || M >= (1 << 24)) return 0;
  return plan_series(N, M, max_cluster).CS;
}

namespace {
cudaError_t series_limits(const void* k) {
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSerSmemMax);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

cudaLaunchAttribute cluster_attr(int CS) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CS;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  return at;
}

// The largest cluster that the device (or the partition of it) holds with the
// most shared memory that a CTA takes here, for both kernels; 0: none. Asked once
// per device.
int series_max_cluster(int device) {
  static std::mutex mu;
  static int cached[64];  // 1 + the answer
  std::lock_guard<std::mutex> lock(mu);
  if (device < 0 || device >= 64) return 0;
  if (cached[device] > 0) return cached[device] - 1;
  int best = 0;
  for (int CS = kSerMaxCS; CS >= 1 && best == 0; CS /= 2) {
    bool all = true;
    for (const void* k : {(const void*)softassign_series_kernel, (const void*)softassign_series_batch_kernel}) {
      cudaLaunchAttribute at[1] = {cluster_attr(CS)};
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(CS);
      cfg.blockDim = dim3(kSerThreads);
      cfg.dynamicSmemBytes = kSerSmemMax;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (series_limits(k) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      all = all && n > 0;
    }
    if (all) best = CS;
  }
  cached[device] = best + 1;
  return best;
}
}  // namespace

bool softassign_series_fits(int N, int M) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return softassign_series_cluster(N, M, series_max_cluster(device)) > 0;
}

namespace {
cudaError_t launch_series(const void* k, int clusters, int CS, size_t smem, void** args, cudaStream_t st,
                          bool beside = false) {
  const cudaError_t e = series_limits(k);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * CS);
  cfg.blockDim = dim3(kSerThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2] = {cluster_attr(CS), {}};
  cfg.attrs = at;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = beside ? 2 : 1;
  return cudaLaunchKernelExC(&cfg, k, args);
}
}  // namespace

int enqueue_softassign_series(const SoftassignLaunch& L, const float4* rows, const float4* cols, const CenterHdr* hdr,
                              float* s_out, float* u_out, SeriesHand* hand, int max_degree, void* ctl,
                              cudaStream_t st) {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const SeriesPlan P = plan_series(L.N, L.M, series_max_cluster(device));
  if (P.CS < 1) return (int)cudaErrorInvalidConfiguration;
  SeriesArgs A{};
  A.rows = rows;
  A.cols = cols;
  A.hdr = hdr;
  A.dRt = L.dRt;
  A.s_in = L.s_io;
  A.u_in = L.u_io;
  A.s_out = s_out;
  A.u_out = u_out;
  A.hand = hand;
  A.N = L.N;
  A.M = L.M;
  A.nr = P.nr;
  A.nc = P.nc;
  A.JMAX = L.JMAX;
  A.I0 = L.I0;
  A.I1 = L.I1;
  A.alpha = L.alpha;
  A.T0 = L.T_0;
  A.TFACTOR = L.TFACTOR;
  A.moutlier = L.moutlier;
  A.max_degree = max_degree < kSerMaxD ? max_degree : kSerMaxD;
  A.ctl = static_cast<Ctl*>(ctl);
  A.trace = L.trace;
  A.trace_cap = L.trace_cap;
  void* args[] = {(void*)&A};
  return (int)launch_series((const void*)softassign_series_kernel, 1, P.CS, P.smem, args, st);
}

size_t softassign_series_table_bytes(int njobs) { return sizeof(SeriesArgs) * (size_t)njobs; }

// Points per CTA for a batch: the fewest for which all clusters run at once.
// One pair (60 temperatures) takes little longer on fewer CTAs (its updates
// are latency: N = M = 1000 on 4 CTAs 4.6 ms, on 1 6.0; 4000 on 16 5.1, on 4
// 6.6), a second wave of clusters twice as long: 20 pairs of 500-20,000 points
// take 15.9 / 11.7 / 6.8 / 8.2 ms with 256 / 512 / 1024 / 1536 points (276 / 210
// / 129 / 105 CTAs) and 25 ms one cluster size after the other. Clusters of 16 leave SMs
// of their GPCs over, so 7/8 of the SMs count (154 CTAs did not fit 152 SMs:
// 12.5 ms; 129 did).
int batch_points(const SeriesJob* jobs, int njobs, int max_cluster, int sms) {
  for (int pts = 256; pts <= 1024; pts *= 2) {
    long ctas = 0;
    for (int i = 0; i < njobs; ++i) ctas += plan_series(jobs[i].N, jobs[i].M, max_cluster, pts).CS;
    if (ctas <= (long)sms * 7 / 8) return pts;
  }
  return kSerBatchPts;
}

int enqueue_softassign_series_batch(const SeriesJob* jobs, int njobs, void* dev_table, void* ctl, cudaStream_t st) {
  int device = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return (int)e;
  const int max_cluster = series_max_cluster(device);
  const int pts = batch_points(jobs, njobs, max_cluster, sms);
  // one launch per cluster size, its pairs in the order given
  std::vector<SeriesArgs> tab;
  tab.reserve((size_t)njobs);
  struct Group {
    int CS, first, n;
    size_t smem;
  };
  std::vector<Group> groups;
  for (int CS = kSerMaxCS; CS >= 1; CS /= 2) {
    Group g{CS, (int)tab.size(), 0, 0};
    for (int i = 0; i < njobs; ++i) {
      const SeriesJob& J = jobs[i];
      const SeriesPlan P = plan_series(J.N, J.M, max_cluster, pts);
      if (P.CS != CS) continue;
      SeriesArgs A{};
      A.rows = J.rows;
      A.cols = J.cols;
      A.hdr = J.hdr;
      A.dRt = J.dRt;
      A.s_out = J.s;
      A.u_out = J.u;
      A.hand = J.hand;
      A.N = J.N;
      A.M = J.M;
      A.nr = P.nr;
      A.nc = P.nc;
      A.JMAX = J.JMAX;
      A.I0 = J.I0;
      A.I1 = J.I1;
      A.alpha = J.alpha;
      A.T0 = J.T0;
      A.TFACTOR = J.TFACTOR;
      A.moutlier = J.moutlier;
      A.max_degree = kSerMaxD;
      A.state = J.state;
      A.dRt_out = J.dRt;
      A.ctl = static_cast<Ctl*>(ctl);
      tab.push_back(A);
      g.n += 1;
      g.smem = P.smem > g.smem ? P.smem : g.smem;
    }
    if (g.n > 0) groups.push_back(g);
  }
  if (tab.empty()) return 0;
  e = put_table(dev_table, tab.data(), sizeof(SeriesArgs) * tab.size(), st);
  for (size_t i = 0; i < groups.size() && e == cudaSuccess; ++i) {
    const SeriesArgs* t = static_cast<const SeriesArgs*>(dev_table) + groups[i].first;
    void* args[] = {(void*)&t};
    e = launch_series((const void*)softassign_series_batch_kernel, groups[i].n, groups[i].CS, groups[i].smem, args, st,
                      i > 0);
  }
  return (int)e;
}

}  // namespace cesa
