// mrf_bp.cu -- the BP hot loop over the incidence lists.
//
//   k_pair_prepare : per (camera, voxel) pair, the cavity probability
//                    q = P(empty) excluding the camera's own message
//                    (src/cuda/gvdbkernels.cu:764-773)
//   k_ray_bp       : per ray, Pre pass (tau accumulation with the reference's
//                    per-brick visibility reset, gvdbkernels.cu:689-819), the
//                    infinity term (gvdbkernels.cu:1196-1208) and the Post pass
//                    (ray->voxel messages, gvdbkernels.cu:824-1038), all as
//                    warp-wide log-domain prefix scans
//   k_pair_update  : per pair, the length-weighted message average, new
//                    log-odds message, total log-odds and belief
//                    (gvdbkernels.cu:457-479); a segmented sum over the
//                    pair-grouped permutation of the dynamic incidences --
//                    no atomics, fixed summation order
#include <cuda_fp16.h>

#include <algorithm>

#include "mrf_internal.h"

namespace mrf {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// kPrepPer pairs per thread, strided by the block so that every load stays
// coalesced and a thread keeps kPrepPer independent L gathers in flight
constexpr int kPrepThreads = 256;
constexpr int kPrepPer = 4;

__global__ void __launch_bounds__(kPrepThreads)
    k_pair_prepare(const uint32_t* __restrict__ pair_vox, const float* __restrict__ m,
                   const float* __restrict__ L, float* __restrict__ lnq, __half* __restrict__ lnq16,
                   float* __restrict__ dm, uint32_t p0, uint32_t p1) {
  const uint32_t base = p0 + blockIdx.x * (kPrepThreads * kPrepPer) + threadIdx.x;
  float eta[kPrepPer];
#pragma unroll
  for (int k = 0; k < kPrepPer; ++k) {
    const uint32_t p = base + k * kPrepThreads;
    eta[k] = p < p1 ? L[pair_vox[p]] - m[p] : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < kPrepPer; ++k) {
    const uint32_t p = base + k * kPrepThreads;
    if (p >= p1) break;
    float qq = clampf(1.0f / (1.0f + expf(eta[k])), kFEps, 1.0f - kFEps);
    if (lnq16)
      lnq16[p] = __float2half_rn(logf(qq));  // 16-bit streams: the ray kernel gathers halves
    else
      lnq[p] = logf(qq);
    if (dm) dm[p] = __int_as_float(0x7fc00000);  // Jacobi: NaN until the pair updates
  }
}

// the same over the views' loud pairs only (Jacobi, later iterations of a
// call): element i of the views' loud ranges back to back (prefix[v] the first
// of view v, whose pairs start at base[v])
__global__ void __launch_bounds__(kPrepThreads)
    k_pair_prepare_loud(const uint32_t* __restrict__ pair_vox, const float* __restrict__ m,
                        const float* __restrict__ L, float* __restrict__ lnq, __half* __restrict__ lnq16,
                        float* __restrict__ dm, const uint32_t* __restrict__ prefix,
                        const uint32_t* __restrict__ base, int nv) {
  const uint32_t n = prefix[nv];
  const uint32_t i0 = blockIdx.x * (kPrepThreads * kPrepPer) + threadIdx.x;
  int v = 0;
  for (int hi = nv; hi - v > 1;) {
    const int mid = (v + hi) >> 1;
    if (prefix[mid] <= i0) v = mid;
    else hi = mid;
  }
  float eta[kPrepPer];
  uint32_t p[kPrepPer];
#pragma unroll
  for (int k = 0; k < kPrepPer; ++k) {
    const uint32_t i = i0 + k * kPrepThreads;
    while (v + 1 < nv && i >= prefix[v + 1]) ++v;
    p[k] = base[v] + (i - prefix[v]);
    eta[k] = i < n ? L[pair_vox[p[k]]] - m[p[k]] : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < kPrepPer; ++k) {
    if (i0 + k * kPrepThreads >= n) break;
    const float qq = clampf(1.0f / (1.0f + expf(eta[k])), kFEps, 1.0f - kFEps);
    if (lnq16)
      lnq16[p[k]] = __float2half_rn(logf(qq));
    else
      lnq[p[k]] = logf(qq);
    dm[p[k]] = __int_as_float(0x7fc00000);
  }
}

// ---- ray messages ----------------------------------------------------------
// A group of kG lanes per ray, 32 / kG rays per warp.  Each lane owns kE = 4
// consecutive incidences of a chunk of 4 kG (ray offsets are padded to
// multiples of 4, so the streams load as 16-byte vectors).
//
// With k4 = k_dyn rounded down to 4, every potential before k4 is zero: the
// static prefix [0, k4) only contributes its sum of l ln q, which needs no
// scan: a lane-strided sum and one group reduction, split at r0 into la
// (before r0) and lb.  From k4 on, C_i = sum_{k4 <= j <= i} l_j ln q_j is a
// serial prefix inside the lane plus one group scan per chunk.  Pre
// visibility restarts at r0 (the reference restores its carried state only
// once the accumulated tau is non-zero, gvdbkernels.cu:708-715):
//   e_i = V^pre_i = exp(C_i + A_{k4-1} - A_{r0-1}),  V_i = exp(A_{r0-1}) e_i,
// so one exponential per incidence serves both passes.  r0 <= k_dyn on every
// ray in the queues; where it lies behind k4 it is in the first vector.
//
// Pass 1 forms the Pre total T = sum e_i (1 - q_i) mu_i.  Pass 2 turns
// (V_i mu_i, q_i, l_i) and T into the messages p_i * l_i of the dynamic
// range [k4, n_post) only: before k_dyn tau_i = 0, F_i = 0, mu1_i = 0 and p_i
// is exactly the clamp floor F_EPS (static messages, summed once per build
// into the pairs).  A warp whose rays all end inside their first chunk keeps
// it in registers for pass 2; otherwise pass 2 re-reads the dynamic range.
// On rays longer than kLongRay the Pre total T is summed across lanes in FP64
// and the running difference T - F of pass 2 is carried in FP64; each lane's
// share of T is a compensated FP32 sum.  (GB300 issues FP64 at 1/64 of the
// FP32 rate, so FP64 stays out of the per-incidence arithmetic.)
//
// The ln q gathers are the kernel's cost.  Pairs are numbered brick-major
// by first visit (mrf_build.cu), so consecutive incidences of a ray gather
// from nearby addresses and neighbouring rays from the same ones.
//
// Why groups of 8: a 1 cm ray holds about 60 incidences from k4 on and 30
// loud ones before it, so a whole warp per ray (chunks of 128) left half its
// lanes idle and paid the scans, reductions and the ticket once per ray: 850
// warp instructions a ray, bound by issue.  Four rays a warp take 300 and
// the kernel waits for memory (issue slots 30 % busy).  Whole Gauss-Seidel
// iteration, 8 x 640x480 at 1 cm, third iteration on: 2.61 ms with a warp
// per ray, 1.97 with 8 lanes, 2.25 with 16, 2.11 with 4; all rays in full
// 3.24, 2.92, 2.94, 3.20; Jacobi, 32 views at 2 cm: 1.86, 1.44, 1.60, 1.51.
// Eight incidences a lane (chunks of 64, fewer warps) and the next rays'
// records fetched a ray ahead: no faster.
constexpr int kRayWarps = 4;
constexpr int kG = 8;                    // lanes per ray
constexpr int kRaysPerWarp = 32 / kG;
constexpr int kE = 4;                    // incidences per lane of a chunk
constexpr int kChunk = kG * kE;
// Chunks of a full static prefix in flight, their pair ids a step ahead: the
// prefix is a chain of a load and a gather that depends on it, and registers
// hold the SM at 32 warps.  1 -> 2: five iterations over eight 640x480 views
// at 2 cm 5.55 -> 5.33 ms, eight at 1 cm 24.2 -> 23.6, five 160x120 views
// 1.137 -> 1.102; rays of endpoint bricks, shorter than a chunk, 7.62 -> 7.70.
// Two without the ids ahead: 5.57, 24.0; three: 5.42, 23.5 (spills).  One where
// more than 8 blocks share the registers (two would spill).
template <int kMinBlocks>
constexpr int kPrefixChunks = kMinBlocks > 8 ? 1 : 2;
constexpr int kLoudPer = 4;              // loud prefix incidences in flight per lane

// inclusive scan and sum over the lanes of a group (gl: lane in the group)
__device__ __forceinline__ float group_incl_scan(float v, int gl) {
#pragma unroll
  for (int o = 1; o < kG; o <<= 1) {
    const float u = __shfl_up_sync(kFull, v, o, kG);
    if (gl >= o) v += u;
  }
  return v;
}
template <typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = kG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// streamed incidence arrays: read-only path (kPol 0) or evict-first
// streaming loads (kPol 1) that leave L2 to the ln q gathers
template <int kPol, typename T>
__device__ __forceinline__ T ld_stream(const T* p) {
  if (kPol) return __ldcs(p);
  return __ldg(p);
}

// four consecutive values at element i (a multiple of 4) as one vector load,
// zeros when !ok
template <int kPol>
__device__ __forceinline__ void ld4(uint32_t (&out)[kE], const uint32_t* __restrict__ base, uint32_t i, bool ok) {
  uint4 u = make_uint4(0u, 0u, 0u, 0u);
  if (ok) u = ld_stream<kPol>(reinterpret_cast<const uint4*>(base + i));
  out[0] = u.x;
  out[1] = u.y;
  out[2] = u.z;
  out[3] = u.w;
}
template <int kPol>
__device__ __forceinline__ void ld4(float (&out)[kE], const float* __restrict__ base, uint32_t i, bool ok) {
  float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (ok) u = ld_stream<kPol>(reinterpret_cast<const float4*>(base + i));
  out[0] = u.x;
  out[1] = u.y;
  out[2] = u.z;
  out[3] = u.w;
}
template <int kPol>
__device__ __forceinline__ void ld4(float (&out)[kE], const __half* __restrict__ base, uint32_t i, bool ok) {
  uint2 u = make_uint2(0u, 0u);
  if (ok) u = ld_stream<kPol>(reinterpret_cast<const uint2*>(base + i));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  out[0] = a.x;
  out[1] = a.y;
  out[2] = b.x;
  out[3] = b.y;
}
__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }

// one lane's slice of a chunk from k4 on: lengths and potentials (zeros in
// the ray's padding and past its end), ln q, the prefix exponents C
struct Slice {
  float len[kE], mu[kE], lq[kE], C[kE];
};

// with the lane's pair ids: gathers ln q, loads potentials (and lengths
// unless kLenIn gave them), forms C from carry; returns the chunk's total
template <int kPol, bool kLenIn, typename TL, typename TQ>
__device__ __forceinline__ float load_slice(Slice& s, const uint32_t (&pid)[kE], uint32_t off, int i0, int n,
                                            float carry, int gl, const TL* __restrict__ inc_len,
                                            const float* __restrict__ inc_mu, const TQ* __restrict__ lnq) {
#pragma unroll
  for (int j = 0; j < kE; ++j) s.lq[j] = i0 + j < n ? to_f(__ldg(lnq + pid[j])) : 0.0f;
  if (!kLenIn) ld4<kPol>(s.len, inc_len, off + i0, i0 < n);
  ld4<kPol>(s.mu, inc_mu, off + i0, i0 < n);
  float run = 0.0f;
#pragma unroll
  for (int j = 0; j < kE; ++j) {
    run += s.len[j] * s.lq[j];
    s.C[j] = run;
  }
  const float incl = group_incl_scan(run, gl);
  const float b = carry + (incl - run);
#pragma unroll
  for (int j = 0; j < kE; ++j) s.C[j] += b;
  return __shfl_sync(kFull, incl, kG - 1, kG);
}

// One ray per group (me.n_pre = me.n_post = 0: the group has none).
template <int kPol, int kPf, int kPre, bool kQuiet, typename TL, typename TQ>
__device__ __forceinline__ void ray_bp_group(const RayMeta& me, uint32_t rid, const QuietPrefix& qp,
                                             const uint32_t* __restrict__ inc_pair,
                                             const TL* __restrict__ inc_len,
                                             const float* __restrict__ inc_mu,
                                             const TQ* __restrict__ lnq, float* __restrict__ inc_pl,
                                             int fix_reset, int gl) {
  const int n_pre = me.n_pre, n_post = me.n_post;
  const int r0 = fix_reset ? 0 : me.r0;
  const int k4 = ray_kdyn(me) & ~3;
  const uint32_t off = me.off;
  // kPf >= 1: the first chunk's pair ids are requested before the static
  // prefix's loads, so the two chains of dependent loads overlap
  uint32_t pid_next[kE];
  float len_next[kE];
  if (kPf) ld4<kPol>(pid_next, inc_pair, off + k4 + kE * gl, k4 + kE * gl < n_pre);
  if (kPf == 2) ld4<kPol>(len_next, inc_len, off + k4 + kE * gl, k4 + kE * gl < n_pre);
  // ---- the static prefix [0, k4): sums of l ln q before and from r0 --------
  float la = 0.0f, lb = 0.0f;
  if (kQuiet) {
    // Its quiet incidences (pairs on voxels without a dynamic incidence in
    // any view) keep their ln q from the third iteration of a call on, so
    // their sums were formed once (k_quiet_prefix); only the prefix's loud
    // incidences are gathered here, kLoudPer per lane at a time (the list
    // is short and its loads depend on one another: what counts is how many
    // are in flight).
    QuietRay qr = {};
    if (n_pre) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(qp.ray) + rid);
      qr = *reinterpret_cast<const QuietRay*>(&u);
    }
    const int nl = (int)qr.na + (int)qr.nb;
    for (int i = gl; i < nl; i += kG * kLoudPer) {
      uint2 en[kLoudPer];
#pragma unroll
      for (int k = 0; k < kLoudPer; ++k) {
        en[k] = make_uint2(0u, 0u);
        if (i + k * kG < nl) en[k] = ld_stream<kPol>(qp.loud + qr.first + i + k * kG);
      }
#pragma unroll
      for (int k = 0; k < kLoudPer; ++k) {
        const float c = i + k * kG < nl ? __uint_as_float(en[k].y) * to_f(__ldg(lnq + en[k].x)) : 0.0f;
        if (i + k * kG < (int)qr.na) la += c;
        else lb += c;
      }
    }
    la = group_sum(la) + qr.qa;
    lb = group_sum(lb) + qr.qb;
    if (fix_reset) {
      lb += la;
      la = 0.0f;
    }
  } else {
    // k4 is a multiple of 4: no vector crosses it
    uint32_t p[kPre][kE];
#pragma unroll
    for (int u = 0; u < kPre; ++u) ld4<kPol>(p[u], inc_pair, off + kE * gl + u * kChunk, kE * gl + u * kChunk < k4);
    for (int i = kE * gl; i < k4; i += kPre * kChunk) {
      float l[kPre][kE], q[kPre][kE];
#pragma unroll
      for (int u = 0; u < kPre; ++u) {
        ld4<kPol>(l[u], inc_len, off + i + u * kChunk, i + u * kChunk < k4);
#pragma unroll
        for (int j = 0; j < kE; ++j) q[u][j] = i + u * kChunk < k4 ? to_f(__ldg(lnq + p[u][j])) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kPre; ++u)
        ld4<kPol>(p[u], inc_pair, off + i + (kPre + u) * kChunk, i + (kPre + u) * kChunk < k4);
#pragma unroll
      for (int u = 0; u < kPre; ++u) {
#pragma unroll
        for (int j = 0; j < kE; ++j) l[u][j] *= q[u][j];
        const int iu = i + u * kChunk;
        if (iu + kE <= r0) {
          la += (l[u][0] + l[u][1]) + (l[u][2] + l[u][3]);
        } else if (iu >= r0) {
          lb += (l[u][0] + l[u][1]) + (l[u][2] + l[u][3]);
        } else {
#pragma unroll
          for (int j = 0; j < kE; ++j) {
            if (iu + j < r0) la += l[u][j];
            else lb += l[u][j];
          }
        }
      }
    }
    la = group_sum(la);
    lb = group_sum(lb);
  }
  // ---- pass 1: Pre total ---------------------------------------------------
  // kPf 1: the next chunk's pair ids are requested before this chunk's ln q
  // gathers; kPf 2: its lengths as well.
  float pre = lb;  // A_{k4-1} - A_{r0-1}; la: A_{r0-1}
  float ts = 0.0f, tc = 0.0f, carry = 0.0f;
  const int trips = __reduce_max_sync(kFull, (n_pre - k4 + kChunk - 1) / kChunk);
  const bool behind = __any_sync(kFull, r0 > k4);
  Slice s;
  float e[kE], q[kE];
  for (int t = 0; t < trips; ++t) {
    const int i0 = k4 + t * kChunk + kE * gl;
    uint32_t pid[kE];
    if (kPf) {
#pragma unroll
      for (int j = 0; j < kE; ++j) pid[j] = pid_next[j];
      if (kPf == 2) {
#pragma unroll
        for (int j = 0; j < kE; ++j) s.len[j] = len_next[j];
      }
      ld4<kPol>(pid_next, inc_pair, off + i0 + kChunk, i0 + kChunk < n_pre);
      if (kPf == 2) ld4<kPol>(len_next, inc_len, off + i0 + kChunk, i0 + kChunk < n_pre);
    } else {
      ld4<kPol>(pid, inc_pair, off + i0, i0 < n_pre);
    }
    carry += load_slice<kPol, kPf == 2>(s, pid, off, i0, n_pre, carry, gl, inc_len, inc_mu, lnq);
    if (t == 0 && behind) {
      // r0 behind k4: A_{r0-1} lies in the first vector
      const int m = r0 - 1 - k4;
      const float c = __shfl_sync(kFull, m == 0 ? s.C[0] : (m == 1 ? s.C[1] : s.C[2]), 0, kG);
      if (r0 > k4) {
        la += c;
        pre = -c;
      }
    }
    float w = 0.0f;
#pragma unroll
    for (int j = 0; j < kE; ++j) {
      e[j] = __expf(s.C[j] + pre);
      q[j] = __expf(s.lq[j]);
      w += e[j] * s.mu[j] * (1.0f - q[j]);
    }
    // compensated: the error of the lane's sum stays at a few ulps however
    // long the ray is
    const float y = w - tc;
    const float u = ts + y;
    tc = (u - ts) - y;
    ts = u;
  }
  // The lanes' shares, summed once per ray, and the infinity term: visibility
  // at the end of Pre (gvdbkernels.cu:1196-1208).  Rays longer than kLongRay
  // sum and carry T in FP64 (Dd), the others in FP32 (Df).
  const bool is_long = n_pre > kLongRay;
  const bool any_long = __any_sync(kFull, is_long);
  const float tinf = (me.flags & 1u) ? __expf(carry + pre) : 0.0f;
  float Df = group_sum(ts - tc) + tinf;
  double Dd = 0.0;
  if (any_long) Dd = group_sum((double)ts - (double)tc) + (double)tinf;
  // ---- pass 2: dynamic messages --------------------------------------------
  // F is zero before k_dyn, so the running F starts at zero at k4; the
  // long-range difference T - F is carried, one subtraction per chunk
  const float ratio = __expf(la);
  float cF = 0.0f;
  carry = 0.0f;
  const int trips2 = trips <= 1 ? trips : __reduce_max_sync(kFull, (n_post - k4 + kChunk - 1) / kChunk);
  for (int t = 0; t < trips2; ++t) {
    const int i0 = k4 + t * kChunk + kE * gl;
    if (trips > 1) {
      uint32_t pid[kE];
      ld4<kPol>(pid, inc_pair, off + i0, i0 < n_post);
      carry += load_slice<kPol, false>(s, pid, off, i0, n_post, carry, gl, inc_len, inc_mu, lnq);
#pragma unroll
      for (int j = 0; j < kE; ++j) {
        e[j] = __expf(s.C[j] + pre);
        q[j] = __expf(s.lq[j]);
      }
    }
    float eloc[kE], run = 0.0f;
#pragma unroll
    for (int j = 0; j < kE; ++j) {
      e[j] *= ratio * s.mu[j];  // V mu
      eloc[j] = run;
      run += e[j] * (1.0f - q[j]);
    }
    const float incl = group_incl_scan(run, gl);
    const float ex = incl - run;
    const float D = is_long ? (float)Dd : Df;
    float out[kE];
#pragma unroll
    for (int j = 0; j < kE; ++j) {
      const float fin = ex + eloc[j];
      const float F = cF + fin;
      const float R = (D - fin) - e[j] * (1.0f - q[j]);
      const float mu1 = F + e[j];
      const float mu0 = F + __fdividef(R, q[j]);
      const float p = clampf(__fdividef(mu1, mu1 + mu0 + 1e-7f), kFEps, 1.0f - kFEps);
      out[j] = i0 + j < n_post ? p * s.len[j] : 0.0f;
    }
    if (i0 < n_post)
      *reinterpret_cast<float4*>(inc_pl + off + i0) = make_float4(out[0], out[1], out[2], out[3]);
    const float ct = __shfl_sync(kFull, incl, kG - 1, kG);
    Df -= ct;
    if (any_long) Dd -= (double)ct;
    cF += ct;
  }
}

// Persistent launch: each warp takes its next kRaysPerWarp rays from a work
// counter.  kReg false: one queue, rays longest first (sorted once per
// incidence build, their RayMeta records copied into queue order), so the
// long rays start early and the short ones fill the tail, and a warp's rays
// have nearly equal lengths.  kReg true (SM-affine): the view's pixels are
// cut into regions of consecutive pixels holding equal shares of its
// incidences, one region per SM (block b serves regions b mod G, + G, ...,
// G = min(grid, regions); a persistent grid is placed on the SMs in block
// order, so a region's blocks share an SM); a warp takes the home rays of
// its regions, then drains the view's leftover queue of short rays.  The
// warps of one SM trace neighbouring rays at the same time -- rays that
// cross the same voxels, so their ln q gathers hit the SM's L1.  Which group
// handles a ray does not change its result.  Variants differ only in
// register budget (kMinBlocks resident blocks per SM), load policy and
// schedule: their arithmetic is identical, so the autotuner's choice never
// changes a result.
template <int kMinBlocks, int kPol, int kPf, bool kReg, bool kQuiet, typename TL, typename TQ>
__global__ void __launch_bounds__(kRayWarps * 32, kMinBlocks)
    k_ray_bp(const RayMeta* __restrict__ queue, uint32_t n_rays, const uint32_t* __restrict__ rstart,
             uint32_t nreg, uint32_t rper, const uint32_t* __restrict__ lprefix,
             const uint32_t* __restrict__ lbase, uint32_t nlv, uint32_t* __restrict__ lcounter,
             uint32_t* __restrict__ counter, const uint32_t* __restrict__ inc_pair,
             const TL* __restrict__ inc_len, const float* __restrict__ inc_mu, const TQ* __restrict__ lnq,
             float* __restrict__ inc_pl, const uint32_t* __restrict__ ids, QuietPrefix qp, int fix_reset) {
  const int lane = threadIdx.x & 31;
  const int gl = lane % kG;
  const uint32_t grp = lane / kG;
  // the warp's next tickets of counter c
  auto take = [&](uint32_t* c) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(c, (uint32_t)kRaysPerWarp);
    return __shfl_sync(kFull, t, 0);
  };
  // the queue in use: kReg false, the whole queue (counter); kReg true, the
  // home rays of region r (counter[r]: positions rstart[q (rper + 1) + rr] ..
  // rstart[q (rper + 1) + rr + 1], view q = r / rper, rr = r % rper; block b
  // serves regions b mod G, + G, ..., G = min(grid, regions): every region
  // has a home block), then the views' leftovers (lcounter: ticket t is view
  // q's (t - lprefix[q])-th leftover for the last q with lprefix[q] <= t)
  const uint32_t G = kReg ? min(gridDim.x, nreg) : 1u;
  uint32_t r = kReg ? blockIdx.x % G : 0u;
  uint32_t first = 0, n = n_rays;
  uint32_t* c = counter;
  bool left = !kReg;
  auto open = [&]() {
    if (r < nreg) {
      const uint32_t q = r / rper;
      const uint32_t* rs = rstart + (size_t)q * (rper + 1) + (r - q * rper);
      first = rs[0];
      n = rs[1] - first;
      c = counter + r;
    } else {
      left = true;
      n = lprefix[nlv];
      c = lcounter;
    }
  };
  if (kReg) open();
  // the record of the group's ray among the warp's tickets t..
  auto record = [&](uint32_t t, RayMeta& me, uint32_t& rid) {
    t += grp;
    me = RayMeta{};
    if (t >= n) return;
    uint32_t pos = first + t;
    if (kReg && left) {
      uint32_t lo = 0, hi = nlv;
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (lprefix[mid] <= t) lo = mid;
        else hi = mid;
      }
      pos = lbase[lo] + (t - lprefix[lo]);
    }
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(queue) + pos);
    me = *reinterpret_cast<const RayMeta*>(&u);
    if (kQuiet) rid = __ldg(ids + pos);
  };
  uint32_t idx = take(c);
  for (;;) {
    if (idx >= n) {
      if (left) return;
      r += G;
      open();
      idx = take(c);
      continue;
    }
    RayMeta me;
    uint32_t rid = 0u;
    record(idx, me, rid);
    // the next tickets are taken before the current rays run, so the atomic's
    // latency hides behind their work
    idx = take(c);
    ray_bp_group<kPol, kPf, kPrefixChunks<kMinBlocks>, kQuiet, TL, TQ>(me, rid, qp, inc_pair, inc_len, inc_mu, lnq,
                                                                       inc_pl, fix_reset, gl);
  }
}

// The static prefix of each queued ray of one view (rays r0..r0+n of the
// pixel arrays; a warp per ray): the loud incidences in [0, k4) -- those
// whose pair is among the view's first n_loud, the pairs on voxels with a
// dynamic incidence in any view -- counted to loff[r] (emit false) or listed
// from loud[loff[r]] on (emit true: pair id and length, in ray order; ray[r]
// gets the list's start and its entries before and from r0 on).
template <bool kEmit>
__global__ void k_loud_prefix(const RayMeta* __restrict__ meta, uint32_t r_first, uint32_t n,
                              const uint32_t* __restrict__ inc_pair, const float* __restrict__ inc_len,
                              uint32_t pair_base, uint32_t n_loud, uint32_t* __restrict__ loff,
                              uint2* __restrict__ loud, QuietRay* __restrict__ ray) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const uint32_t r = r_first + w;
  const RayMeta me = meta[r];
  uint32_t cnt = 0, na = 0;
  const uint32_t first = kEmit ? loff[r] : 0u;
  if (ray_in_bp(me)) {
    const int k4 = ray_kdyn(me) & ~3;
    for (int b = 0; b < k4; b += 32) {
      const int j = b + lane;
      const uint32_t p = j < k4 ? inc_pair[me.off + j] : 0u;
      const bool is_loud = j < k4 && p - pair_base < n_loud;
      const unsigned m = __ballot_sync(kFull, is_loud);
      if (kEmit) {
        if (is_loud)
          loud[first + cnt + (uint32_t)__popc(m & ((1u << lane) - 1u))] =
              make_uint2(p, __float_as_uint(inc_len[me.off + j]));
        na += (uint32_t)__popc(__ballot_sync(kFull, is_loud && j < (int)me.r0));
      }
      cnt += (uint32_t)__popc(m);
    }
  }
  if (lane) return;
  if (kEmit) {
    ray[r].first = first;
    ray[r].na = (uint16_t)na;
    ray[r].nb = (uint16_t)(cnt - na);
  } else {
    loff[r] = cnt;
  }
}

// The quiet sums of the static prefix of each queued ray of one view (a
// warp per ray): sum of l ln q over the quiet incidences j < min(r0, k4)
// and min(r0, k4) <= j < k4, written to ray[r] -- valid while the quiet pairs' ln q stay
// fixed, from the third iteration of a call on.  Lane-strided partial
// sums and a butterfly warp sum: a fixed order.
template <typename TQ>
__global__ void k_quiet_prefix(const RayMeta* __restrict__ meta, uint32_t r_first, uint32_t n,
                               const uint32_t* __restrict__ inc_pair, const float* __restrict__ inc_len,
                               const TQ* __restrict__ lnq, uint32_t pair_base, uint32_t n_loud,
                               QuietRay* __restrict__ ray) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= n) return;
  const uint32_t r = r_first + w;
  const RayMeta me = meta[r];
  if (!ray_in_bp(me)) return;
  const int k4 = ray_kdyn(me) & ~3;
  const int ra = min((int)me.r0, k4);
  float qa = 0.0f, qk = 0.0f;
  for (int j = lane; j < k4; j += 32) {
    const uint32_t p = inc_pair[me.off + j];
    if (p - pair_base >= n_loud) {
      const float c = inc_len[me.off + j] * to_f(__ldg(lnq + p));
      if (j < ra) qa += c;
      else qk += c;
    }
  }
  qa = warp_sum(qa);
  qk = warp_sum(qk);
  if (lane == 0) *reinterpret_cast<float2*>(&ray[r].qa) = make_float2(qa, qk);
}

// ray queue of one build: active rays sorted by decreasing length
// The views of a batch: view v has pixels pix[v] .. pix[v + 1] (from the
// batch's first) and act[v + 1] - act[v] rays in BP.
__device__ __forceinline__ uint32_t batch_view(const uint32_t* first, uint32_t n, uint32_t i) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (first[mid] <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}
// the last view that begins at or before i is the one that holds it: of views
// without rays, which share their successor's first, it is the successor
__device__ __forceinline__ uint32_t ray_at(const QueueBatch& b, uint32_t v, uint32_t a) {
  return b.pix[v] + (a - b.act[v]);
}

// sort keys (by view, longest first, rays outside BP last), pixel numbers
// and, for the rays in BP, n_pre
__global__ void k_ray_keys(const __grid_constant__ QueueBatch b, const RayMeta* __restrict__ meta,
                           uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* __restrict__ work) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x, n = b.pix[b.views];
  if (r > n) return;
  if (r == n) {
    work[n] = 0u;
    return;
  }
  const RayMeta me = meta[r];
  const bool in = ray_in_bp(me);
  keys[r] = batch_view(b.pix, b.views, r) << 17 | (in ? 0xFFFFu - me.n_pre : 0x10000u);
  vals[r] = r;
  work[r] = in ? me.n_pre : 0u;
}

// The queues of a batch of views from their sorted rays.
//
// The queue of all rays: each view's rays longest first.  The SM-affine region
// lists (see region_lists, which states them on the host): each ray's region
// from the work before its pixel, a stable sort by region, which leaves a
// region's rays longest first, the work before a ray inside its region, which
// says whether it is a home ray, and one scan that places each view's home
// rays (by region) and behind them its leftovers (longest first).  A dozen
// passes over a few hundred thousand rays at launch latency, which is why
// views go through them together (5 views of 160x120 one by one: 0.5 ms).  With
// the ray records copied down, the lists made by host threads and copied up, an
// appended 640x480 frame took 1.5 ms longer and a build of twelve 4 ms.
__global__ void k_region_keys(const __grid_constant__ QueueBatch b, const RayMeta* __restrict__ meta,
                              const uint32_t* __restrict__ sorted, const uint32_t* __restrict__ before, uint32_t R,
                              uint32_t* __restrict__ region, uint32_t* __restrict__ rank,
                              RayMeta* __restrict__ queue, uint32_t* __restrict__ ids, uint32_t id_base) {
  const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= b.act[b.views]) return;
  const uint32_t v = batch_view(b.act, b.views, a), pix = sorted[ray_at(b, v, a)];
  const uint32_t w0 = before[b.pix[v]];
  const uint64_t work = max(before[b.pix[v + 1]] - w0, 1u);
  region[a] = v * R + (uint32_t)min((uint64_t)(R - 1), (uint64_t)(before[pix] - w0) * R / work);
  rank[a] = a;
  if (queue) {
    queue[a] = meta[pix];
    ids[a] = id_base + pix;
  }
}

// by region: bounds[x], the first ray of a region >= x (x <= views R), and
// the rays' work, from the sort keys of their ranks
__global__ void k_region_bounds(const __grid_constant__ QueueBatch b, const uint32_t* __restrict__ region,
                                const uint32_t* __restrict__ rank, const uint32_t* __restrict__ keys, uint32_t R,
                                uint32_t* __restrict__ bounds, uint32_t* __restrict__ work) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x, n = b.act[b.views];
  if (k > n) return;
  const uint32_t hi = k == n ? b.views * R : region[k];
  for (uint32_t x = k == 0 ? 0u : region[k - 1] + 1u; x <= hi; ++x) bounds[x] = k;
  uint32_t w = 0u;
  if (k < n) {
    const uint32_t a = rank[k], v = batch_view(b.act, b.views, a);
    w = 0xFFFFu - (keys[ray_at(b, v, a)] & 0x1FFFFu);
  }
  work[k] = w;
}

// Flags of a view, at twice its first ray: its rays by region that are home
// rays, then its rays by length that are leftovers.
__global__ void k_region_home(const __grid_constant__ QueueBatch b, const uint32_t* __restrict__ region,
                              const uint32_t* __restrict__ rank, const uint32_t* __restrict__ before,
                              const uint32_t* __restrict__ bounds, uint32_t share, uint32_t* __restrict__ flag) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x, n = b.act[b.views];
  if (k > n) return;
  if (k == n) {
    flag[2 * (size_t)n] = 0u;
    return;
  }
  const uint32_t v = batch_view(b.act, b.views, k);
  const uint32_t x = region[k], lo = before[bounds[x]], hi = before[bounds[x + 1]];
  const bool home = (uint64_t)(before[k] - lo) * 100u < (uint64_t)(hi - lo) * share;
  flag[(size_t)b.act[v] + k] = home;
  flag[(size_t)b.act[v + 1] + rank[k]] = !home;
}

// the lists, and each view's row of region starts (R and the end of its home
// rays), first leftover and {0, leftovers}
__global__ void k_region_emit(const __grid_constant__ QueueBatch b, const RayMeta* __restrict__ meta,
                              const uint32_t* __restrict__ sorted, const uint32_t* __restrict__ rank,
                              const uint32_t* __restrict__ place, const uint32_t* __restrict__ bounds, uint32_t R,
                              uint32_t at, uint32_t id_base, RayMeta* __restrict__ queue, uint32_t* __restrict__ ids,
                              uint32_t* __restrict__ rstart, uint32_t* __restrict__ lbase,
                              uint32_t* __restrict__ lsingle) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x, n = b.act[b.views];
  if (e < b.views * (R + 1)) {
    const uint32_t v = e / (R + 1), r = e - v * (R + 1);
    // a bound at the view's end: the first of its leftovers' flags
    const uint32_t k = r < R ? bounds[v * R + r] : b.act[v + 1];
    const uint32_t p = place[(size_t)b.act[v] + k];
    rstart[e] = at + p;
    if (r == R) {
      lbase[v] = at + p;
      lsingle[2 * v] = 0u;
      lsingle[2 * v + 1] = b.act[v + 1] - p;
    }
  }
  if (e >= 2 * n || place[e + 1] == place[e]) return;
  const uint32_t v = batch_view(b.act, b.views, e >> 1);
  const uint32_t i = e - 2 * b.act[v], m = b.act[v + 1] - b.act[v];
  const uint32_t a = i < m ? rank[b.act[v] + i] : b.act[v] + (i - m);
  const uint32_t pix = sorted[ray_at(b, v, a)];
  queue[at + place[e]] = meta[pix];
  ids[at + place[e]] = id_base + pix;
}

// prefix of the views' leftover counts (lsingle[2 c + 1]), V + 1 entries; one warp
__global__ void k_leftover_prefix(const uint32_t* __restrict__ lsingle, uint32_t V, uint32_t* __restrict__ prefix) {
  uint32_t run = 0;
  for (uint32_t c0 = 0; c0 <= V; c0 += 32) {
    const uint32_t c = c0 + threadIdx.x;
    const uint32_t v = c < V ? lsingle[2 * c + 1] : 0u;
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(kFull, incl, o);
      if ((int)threadIdx.x >= o) incl += u;
    }
    if (c <= V) prefix[c] = run + incl - v;
    run += __shfl_sync(kFull, incl, 31);
  }
}

// Pair update: a load-balanced segmented reduction over the pair-grouped
// permutation of the messages, fused with the per-pair update.  One block
// takes a tile of kTile consecutive positions: it gathers the tile's messages
// into shared memory (coalesced permutation reads, kTile independent gathers
// in flight) together with the segment bounds of the pairs the tile
// touches; each thread then sums whole pairs sequentially from shared memory
// (a fixed order) and updates them.  A block owns the pairs that start in its
// tile, so no tile waits for another and no second kernel adds carries (4.5 us
// per view and iteration, 14 % of an iteration on 160x120 views).  It gathers
// kAhead positions of the next tile too, which ends nearly every pair that
// crosses over; a longer one is summed on by the whole block (lane-strided,
// then a fixed tree).
constexpr int kTileThreads = 256;
constexpr int kTile = 4 * kTileThreads;
constexpr uint32_t kAhead = 32;

// a dynamic run's update with its old message mo and the voxel's old total
// Lo already loaded (the gate c > kCumLenGate already checked)
__device__ __forceinline__ void apply_run_loaded(const uint4 r, float mo, float Lo, float acc_dyn,
                                                 float* __restrict__ m, float* __restrict__ L,
                                                 float* __restrict__ dm, int jacobi) {
  const uint32_t p = r.x, v = r.y;
  const float c = __uint_as_float(r.z);
  float a = clampf((__uint_as_float(r.w) + acc_dyn) / c, kFEps, 1.0f - kFEps);
  float mn = logf(a) - logf(1.0f - a);
  m[p] = mn;
  if (jacobi) {
    dm[p] = mn - mo;
    return;
  }
  L[v] = Lo + (mn - mo);
}

// factor->voxel update of one pair (gvdbkernels.cu:457-479).  The belief
// 1 - clamp(1 / (1 + e^L)) is not written here: k_belief_refresh derives it
// from L once the iterations of a call are done.
__device__ __forceinline__ void apply_pair(uint32_t p, float acc, const uint32_t* __restrict__ pair_vox,
                                           float* __restrict__ m, const float* __restrict__ cum,
                                           float* __restrict__ L, float* __restrict__ dm, int jacobi) {
  const float c = cum[p];
  const float mo = m[p];
  const uint32_t v = pair_vox[p];
  if (!(c > kCumLenGate)) return;  // gvdbkernels.cu:408: the pair never updates
  float a = clampf(acc / c, kFEps, 1.0f - kFEps);
  float mn = logf(a) - logf(1.0f - a);
  m[p] = mn;
  if (jacobi) {
    dm[p] = mn - mo;
    return;
  }
  L[v] = L[v] + (mn - mo);
}

// the same for a dynamic run, whose pair id, voxel, cumulative length and
// static-message sum are stored together (one 16-byte load; the voxel's L
// gather does not wait on a pair-id lookup)
__device__ __forceinline__ void apply_run(const uint4 r, float acc_dyn, float* __restrict__ m,
                                          float* __restrict__ L, float* __restrict__ dm, int jacobi) {
  const uint32_t p = r.x, v = r.y;
  const float c = __uint_as_float(r.z);
  if (!(c > kCumLenGate)) return;  // gvdbkernels.cu:408: the pair never updates
  apply_run_loaded(r, m[p], jacobi ? 0.0f : L[v], acc_dyn, m, L, dm, jacobi);
}

// kTwo false: one prefetched pair per thread, 32 registers (8 blocks per
// SM); true: two, 48 registers (5 blocks per SM).  Same arithmetic.
template <bool kTwo>
__global__ void __launch_bounds__(kTileThreads, kTwo ? 5 : 8)
    k_pair_reduce(const uint32_t* __restrict__ perm, const float* __restrict__ pl,
                  const uint32_t* __restrict__ seg, const uint32_t* __restrict__ tile_first,
                  uint32_t k0, uint32_t k1, uint32_t p_end, const uint4* __restrict__ drun, float* __restrict__ m, float* __restrict__ L,
                  float* __restrict__ dm, int jacobi) {
  __shared__ float sv[kTile + kAhead];
  __shared__ uint32_t sseg[kTile + 2];
  __shared__ float open_sum, part[kTileThreads / 32];
  const int t = threadIdx.x;
  const uint32_t base = k0 + blockIdx.x * kTile;
  const uint32_t n = min((uint32_t)kTile, k1 - base);
  const uint32_t end = base + n;
  const uint32_t ahead = min(kAhead, k1 - end);
  const uint32_t pf = tile_first[blockIdx.x];
  // a tile touches at most n pairs: their starts and the next pair's start
  const uint32_t nseg = min(n + 1, p_end - pf) + 1;
  // the run records of this thread's first two pairs (q = t, t + 256; a
  // tile of 1024 positions holds about 340 pairs), and those pairs' messages
  // and voxel totals, are requested before the message gathers so that no
  // dependent load waits after the barrier.  The tile's pairs end at the
  // next tile's first pair.
  const uint32_t last = blockIdx.x + 1 < gridDim.x ? tile_first[blockIdx.x + 1] : p_end - 1;
  uint4 r0 = make_uint4(0u, 0u, 0u, 0u), r1 = make_uint4(0u, 0u, 0u, 0u);
  float mo0 = 0.0f, Lo0 = 0.0f, mo1 = 0.0f, Lo1 = 0.0f;
  const bool pre = t < n && pf + t < p_end;
  const bool pre1 = kTwo && t + kTileThreads < n && pf + t + kTileThreads <= min(last, p_end - 1);
  if (pre) r0 = drun[pf + t];
  if (pre1) r1 = drun[pf + t + kTileThreads];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t i = j * kTileThreads + t;
    if (i < n) sv[i] = pl[perm[base + i]];
  }
  if (t < ahead) sv[n + t] = pl[perm[end + t]];
  for (uint32_t q = t; q < nseg; q += kTileThreads) sseg[q] = seg[pf + q];
  const bool gate0 = pre && __uint_as_float(r0.z) > kCumLenGate;
  if (gate0) {
    mo0 = m[r0.x];
    if (!jacobi) Lo0 = L[r0.y];
  }
  const bool gate1 = pre1 && __uint_as_float(r1.z) > kCumLenGate;
  if (gate1) {
    mo1 = m[r1.x];
    if (!jacobi) Lo1 = L[r1.y];
  }
  __syncthreads();
  for (uint32_t q = t; q < n && pf + q < p_end && sseg[q] < end; q += kTileThreads) {
    const uint32_t s0 = sseg[q], s1 = sseg[q + 1];
    if (s0 < base) continue;  // an earlier tile's
    const uint32_t a = s0 - base, b = min(s1, end + ahead) - base;
    float acc = 0.0f;
    for (uint32_t i = a; i < b; ++i) acc += sv[i];
    if (s1 > end + ahead) {  // the last one
      open_sum = acc;
      continue;
    }
    if (q == t) {
      if (gate0) apply_run_loaded(r0, mo0, Lo0, acc, m, L, dm, jacobi);
    } else if (q == t + kTileThreads && pre1) {
      if (gate1) apply_run_loaded(r1, mo1, Lo1, acc, m, L, dm, jacobi);
    } else {
      apply_run(drun[pf + q], acc, m, L, dm, jacobi);
    }
  }
  // a pair that goes on for longer, if it starts in the tile
  const uint32_t ql = last - pf;
  if (sseg[ql] < base || sseg[ql] >= end || sseg[ql + 1] <= end + ahead) return;
  const uint32_t s1 = sseg[ql + 1];
  float x = 0.0f;
  for (uint32_t i = end + ahead + t; i < s1; i += kTileThreads) x += pl[perm[i]];
  x = warp_sum(x);
  if ((t & 31) == 0) part[t >> 5] = x;
  __syncthreads();  // open_sum and the warps' parts
  if (t == 0) {
    for (int w = 1; w < kTileThreads / 32; ++w) x += part[w];
    apply_run(drun[last], open_sum + x, m, L, dm, jacobi);
  }
}

// first pair of every tile of a position range (pairs are sorted, so it is
// the pair whose segment holds the tile's first position)
__global__ void k_tile_first(const uint32_t* __restrict__ seg, uint32_t p0, uint32_t p1, uint32_t k0,
                             uint32_t ntiles, uint32_t* __restrict__ out) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  uint32_t pos = k0 + t * kTile;
  uint32_t lo = p0, hi = p1;  // last p with seg[p] <= pos
  while (hi - lo > 1) {
    uint32_t mid = lo + ((hi - lo) >> 1);
    if (seg[mid] <= pos) lo = mid;
    else hi = mid;
  }
  out[t] = lo;
}

// per dynamic run: {pair id, voxel, cumulative length, static-message sum}
__global__ void k_drun(const uint32_t* __restrict__ dpair, uint32_t n, const uint32_t* __restrict__ pair_vox,
                       const float* __restrict__ cum, const float* __restrict__ stat,
                       uint4* __restrict__ drun) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t p = dpair[j];
  drun[j] = make_uint4(p, pair_vox[p], __float_as_uint(cum[p]), __float_as_uint(stat[p]));
}

// pairs whose incidences are all static: a = (sum of F_EPS * l) / cum is a
// build constant, so their update changes the state only right after their
// messages were zeroed or remapped
__global__ void k_static_pairs(uint32_t p0, uint32_t p1, const uint32_t* __restrict__ ndyn,
                               const float* __restrict__ stat, const uint32_t* __restrict__ pair_vox,
                               float* __restrict__ m, const float* __restrict__ cum,
                               float* __restrict__ L, float* __restrict__ dm, int jacobi) {
  uint32_t p = p0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= p1 || ndyn[p]) return;
  apply_pair(p, stat[p], pair_vox, m, cum, L, dm, jacobi);
}

// Jacobi: total log-odds of each voxel moves by the sum of its cameras'
// message changes (pairs of a voxel grouped by a voxel-sorted CSR)
__global__ void k_voxel_apply(const uint32_t* __restrict__ vseg, const uint32_t* __restrict__ vpairs,
                              const uint32_t* __restrict__ vvox, uint32_t nvox,
                              const float* __restrict__ dm, float* __restrict__ L) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvox) return;
  float s = 0.0f;
  bool any = false;
  for (uint32_t k = vseg[i]; k < vseg[i + 1]; ++k) {
    float d = dm[vpairs[k]];
    if (d == d) {  // pairs below the length gate carry NaN and are skipped
      s += d;
      any = true;
    }
  }
  if (!any) return;
  uint32_t v = vvox[i];
  L[v] = L[v] + s;
}

// beliefs of the voxels the iterations update (those with a pair past the
// length gate in some camera), from their total log-odds: the per-voxel
// belief of gvdbkernels.cu:474-477, written once per call instead of at
// every message update
__global__ void k_belief_refresh(const float* __restrict__ L, const uint8_t* __restrict__ active, int64_t n,
                                 float* __restrict__ belief) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (active[i]) belief[i] = 1.0f - clampf(1.0f / (1.0f + expf(L[i])), kFEps, 1.0f - kFEps);
}

__global__ void k_max_abs_diff(const float* __restrict__ a, const float* __restrict__ b, int64_t n,
                               uint32_t* __restrict__ out) {
  float mx = 0.0f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    mx = fmaxf(mx, fabsf(a[i] - b[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(mx));
}

// total log-odds of each voxel rebuilt from its messages (voxel CSR):
// L = L (already the prior) + sum m over the pairs that pass the length gate
__global__ void k_voxel_rebuild(const uint32_t* __restrict__ vseg, const uint32_t* __restrict__ vpairs,
                                const uint32_t* __restrict__ vvox, uint32_t nvox,
                                const float* __restrict__ m, const float* __restrict__ cum,
                                float* __restrict__ L, float* __restrict__ belief) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvox) return;
  float s = 0.0f;
  bool any = false;
  for (uint32_t k = vseg[i]; k < vseg[i + 1]; ++k) {
    const uint32_t p = vpairs[k];
    if (cum[p] > kCumLenGate) {
      s += m[p];
      any = true;
    }
  }
  if (!any) return;
  uint32_t v = vvox[i];
  float Lv = L[v] + s;
  L[v] = Lv;
  belief[v] = 1.0f - clampf(1.0f / (1.0f + expf(Lv)), kFEps, 1.0f - kFEps);
}

// Warm-start initial messages of every voxel's pairs from a predicted total
// log-odds: pairs without dynamic incidences get their exact constant
// message; the rest of (L_pred - logit(prior)) is shared among the dynamic
// pairs in proportion to their cumulative length.  Pairs below the length
// gate keep 0 (they never update).
__global__ void k_warm_split(const uint32_t* __restrict__ vseg, const uint32_t* __restrict__ vpairs,
                             const uint32_t* __restrict__ vvox, uint32_t nvox,
                             const float* __restrict__ L_pred, float lp, const float* __restrict__ base,
                             const float* __restrict__ cum, const float* __restrict__ stat,
                             const uint32_t* __restrict__ ndyn, float* __restrict__ m) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvox) return;
  float fixed = 0.0f, dyn_len = 0.0f;
  for (uint32_t k = vseg[i]; k < vseg[i + 1]; ++k) {
    const uint32_t p = vpairs[k];
    const float c = cum[p];
    if (!(c > kCumLenGate)) continue;
    if (ndyn[p]) {
      dyn_len += c;
    } else {
      float a = clampf(stat[p] / c, kFEps, 1.0f - kFEps);
      fixed += logf(a) - logf(1.0f - a);
    }
  }
  const float rest = L_pred[vvox[i]] - (base ? base[vvox[i]] : lp) - fixed;
  for (uint32_t k = vseg[i]; k < vseg[i + 1]; ++k) {
    const uint32_t p = vpairs[k];
    const float c = cum[p];
    float mv = 0.0f;
    if (c > kCumLenGate) {
      if (ndyn[p]) {
        mv = rest * (c / dyn_len);
      } else {
        float a = clampf(stat[p] / c, kFEps, 1.0f - kFEps);
        mv = logf(a) - logf(1.0f - a);
      }
    }
    m[p] = mv;
  }
}

// Warm-start features of every voxel slot, [slot*512 + local][4]:
// 0 current belief, 1 log(1 + pass-through length), 2 log(1 + potential
// mass sum mu*l), 3 log(1 + length inside the potential windows); lengths
// in voxels, summed over the voxel's cameras in pair order.
__global__ void k_feat_belief(const float* __restrict__ belief, int64_t n, float* __restrict__ feat) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  *reinterpret_cast<float4*>(feat + 4 * i) = make_float4(belief[i], 0.0f, 0.0f, 0.0f);
}

__global__ void k_voxel_features(const uint32_t* __restrict__ vseg, const uint32_t* __restrict__ vpairs,
                                 const uint32_t* __restrict__ vvox, uint32_t nvox,
                                 const float* __restrict__ cum, const float* __restrict__ stat,
                                 const float* __restrict__ hit, float* __restrict__ feat) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvox) return;
  float pass = 0.0f, mass = 0.0f, win = 0.0f;
  for (uint32_t k = vseg[i]; k < vseg[i + 1]; ++k) {
    const uint32_t p = vpairs[k];
    const float sl = stat[p] * (1.0f / kFEps);
    pass += sl;
    mass += hit[p];
    win += fmaxf(cum[p] - sl, 0.0f);
  }
  float* f = feat + 4 * (int64_t)vvox[i];
  f[1] = log1pf(pass);
  f[2] = log1pf(mass);
  f[3] = log1pf(win);
}

// moving a camera: take its messages out of the total log-odds
__global__ void k_remove_messages(const uint32_t* __restrict__ pair_vox, float* __restrict__ m,
                                  uint32_t p0, uint32_t p1, float* __restrict__ L,
                                  float* __restrict__ belief) {
  uint32_t p = p0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= p1) return;
  float mo = m[p];
  if (mo == 0.0f) return;
  uint32_t v = pair_vox[p];
  float Lv = L[v] - mo;
  L[v] = Lv;
  belief[v] = 1.0f - clampf(1.0f / (1.0f + expf(Lv)), kFEps, 1.0f - kFEps);
  m[p] = 0.0f;
}

// a retired camera's messages added to the base log-odds (one pair per
// voxel within a camera: no two threads share a voxel)
__global__ void k_fold_messages(const uint32_t* __restrict__ pv, const float* __restrict__ m, uint32_t n,
                                float* __restrict__ base) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n && m[p] != 0.0f) base[pv[p]] += m[p];
}

__global__ void k_remap_scatter(const uint32_t* __restrict__ pv, const float* __restrict__ m,
                                uint32_t n, float* __restrict__ dense) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) dense[pv[p]] = m[p];
}

__global__ void k_remap_gather(const uint32_t* __restrict__ pv, float* __restrict__ m, uint32_t n,
                               const float* __restrict__ dense) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) m[p] = dense[pv[p]];
}

__global__ void k_fill_u32(uint32_t* p, int64_t n, uint32_t v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

__global__ void k_fill(float* p, int64_t n, float v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// sort keys of the pairs' voxels: voxels without a dynamic incidence behind
// the others (top: a bit above every voxel id)
__global__ void k_voxel_keys(const uint32_t* __restrict__ pair_vox, uint32_t n, const uint8_t* __restrict__ loud,
                             uint32_t top, uint32_t* __restrict__ key) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) key[p] = pair_vox[p] | (loud[pair_vox[p]] ? 0u : top);
}

__global__ void k_vflag(const uint32_t* __restrict__ sk, uint32_t n, uint32_t* __restrict__ flag) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) flag[k] = (k == 0 || sk[k] != sk[k - 1]) ? 1u : 0u;
}

__global__ void k_vassign(const uint32_t* __restrict__ sk, const uint32_t* __restrict__ flag,
                          const uint32_t* __restrict__ scan, uint32_t n, uint32_t top,
                          uint32_t* __restrict__ vvox, uint32_t* __restrict__ vseg, uint32_t* __restrict__ n_loud) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !flag[k]) return;
  vvox[scan[k]] = sk[k] & ~top;
  vseg[scan[k]] = k;
  // the loud voxels end where the first other one begins
  if (top && (sk[k] & top) && (k == 0 || !(sk[k - 1] & top))) *n_loud = scan[k];
}

__global__ void k_scatter_const(const uint32_t* __restrict__ idx, uint32_t n, float v,
                                float* __restrict__ dense) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) dense[idx[p]] = v;
}

// pairs past the length gate (the ones that ever update): counted, and
// their voxels flagged
__global__ void k_touch_pairs(const uint32_t* __restrict__ pair_vox, const float* __restrict__ cum,
                              uint32_t np, uint8_t* __restrict__ flag,
                              unsigned long long* __restrict__ n_active) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = p < np && cum[p] > kCumLenGate;
  if (act) flag[pair_vox[p]] = 1;
  const unsigned b = __ballot_sync(kFull, act);
  if (n_active && (threadIdx.x & 31) == 0 && b) atomicAdd(n_active, (unsigned long long)__popc(b));
}

__global__ void k_count_flags(const uint8_t* __restrict__ flag, int64_t n, unsigned long long* __restrict__ out) {
  unsigned c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += flag[i] != 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, (unsigned long long)c);
}

inline unsigned blocks(int64_t n, int t) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

}  // namespace

cudaError_t launch_pair_prepare(const BpArrays& a, uint32_t p0, uint32_t p1, int jacobi,
                                cudaStream_t s) {
  if (p1 <= p0) return cudaSuccess;
  k_pair_prepare<<<blocks(p1 - p0, kPrepThreads * kPrepPer), kPrepThreads, 0, s>>>(
      a.pair_vox, a.pair_m, a.L, a.pair_lnq, a.half_streams ? a.pair_lnq16 : nullptr,
      jacobi ? a.pair_dm : nullptr, p0, p1);
  return cudaGetLastError();
}


cudaError_t launch_pair_prepare_loud(const BpArrays& a, const uint32_t* prefix, const uint32_t* base, int nv,
                                     uint32_t n, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_pair_prepare_loud<<<blocks(n, kPrepThreads * kPrepPer), kPrepThreads, 0, s>>>(
      a.pair_vox, a.pair_m, a.L, a.pair_lnq, a.half_streams ? a.pair_lnq16 : nullptr, a.pair_dm, prefix, base, nv);
  return cudaGetLastError();
}

// ray-kernel variants: (id, resident-block target, load policy, chunk
// prefetch, schedule: 0 longest first, 1 SM regions)
#define MRF_RAY_VARIANTS(X) \
  X(0, 8, 0, 0, 0) X(1, 8, 0, 1, 0) X(2, 7, 0, 2, 0) X(3, 8, 0, 0, 1) X(4, 8, 0, 1, 1) X(5, 7, 0, 2, 1) \
  X(6, 10, 0, 1, 1) X(7, 8, 1, 1, 1)
constexpr int kRayVariants = 8;

int ray_bp_variants() { return kRayVariants; }

namespace {
using RayKernel32 = decltype(&k_ray_bp<8, 0, 0, false, false, float, float>);
using RayKernel16 = decltype(&k_ray_bp<8, 0, 0, false, false, __half, __half>);

#define X(id, mb, pol, pf, sc) \
  {k_ray_bp<mb, pol, pf, (sc > 0), false, float, float>, k_ray_bp<mb, pol, pf, (sc > 0), true, float, float>},
const RayKernel32 kRay32[kRayVariants][2] = {MRF_RAY_VARIANTS(X)};
#undef X
#define X(id, mb, pol, pf, sc) \
  {k_ray_bp<mb, pol, pf, (sc > 0), false, __half, __half>, k_ray_bp<mb, pol, pf, (sc > 0), true, __half, __half>},
const RayKernel16 kRay16[kRayVariants][2] = {MRF_RAY_VARIANTS(X)};
#undef X
#define X(id, mb, pol, pf, sc) (sc > 0),
const bool kRayRegions[kRayVariants] = {MRF_RAY_VARIANTS(X)};
#undef X

template <typename K>
int resident_of(K kernel) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel,
                                                    kRayWarps * 32, 0) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  return per_sm;
}
}  // namespace

bool ray_bp_regions(int variant) { return variant >= 0 && variant < kRayVariants && kRayRegions[variant]; }

int ray_bp_resident_blocks(int variant, int half_streams, int quiet) {
  static int resident[2][2][kRayVariants] = {{{0}}};
  if (variant < 0 || variant >= kRayVariants) return 1;
  int& r = resident[half_streams ? 1 : 0][quiet ? 1 : 0][variant];
  if (!r)
    r = half_streams ? resident_of(kRay16[variant][quiet ? 1 : 0]) : resident_of(kRay32[variant][quiet ? 1 : 0]);
  return r;
}

cudaError_t launch_ray_bp(const BpArrays& a, const RayWork& w, int fix_reset, int num_sms, int variant,
                          bool quiet, cudaStream_t s) {
  if (!w.n_rays) return cudaSuccess;
  QuietPrefix qp{};
  if (quiet) {
    qp.ray = a.quiet_ray;
    qp.loud = a.loud;
  }
  if (variant < 0 || variant >= kRayVariants) return cudaErrorInvalidValue;
  constexpr int kRaysPerBlock = kRayWarps * kRaysPerWarp;
  int64_t b = std::min<int64_t>((int64_t)num_sms * ray_bp_resident_blocks(variant, a.half_streams, quiet),
                                (w.n_rays + kRaysPerBlock - 1) / kRaysPerBlock);
  const unsigned grid = (unsigned)std::max<int64_t>(b, 1);
  const bool reg = kRayRegions[variant];
  const RayMeta* queue = reg ? w.region : w.queue;
  uint32_t* counter = reg ? w.rcounter : w.counter;
  const uint32_t* ids = reg ? w.region_ids : w.queue_ids;
  if (a.half_streams)
    kRay16[variant][quiet]<<<grid, kRayWarps * 32, 0, s>>>(
        queue, w.n_rays, w.rstart, w.nreg, w.rper, w.lprefix, w.lbase, w.nlv, w.lcounter, counter, a.inc_pair,
        a.inc_len16, a.inc_mu, a.pair_lnq16, a.inc_pl, ids, qp, fix_reset);
  else
    kRay32[variant][quiet]<<<grid, kRayWarps * 32, 0, s>>>(
        queue, w.n_rays, w.rstart, w.nreg, w.rper, w.lprefix, w.lbase, w.nlv, w.lcounter, counter, a.inc_pair,
        a.inc_len, a.inc_mu, a.pair_lnq, a.inc_pl, ids, qp, fix_reset);
  return cudaGetLastError();
}

cudaError_t launch_ray_keys(const QueueBatch& b, const RayMeta* meta, uint32_t* keys, uint32_t* vals, uint32_t* work,
                            cudaStream_t s) {
  k_ray_keys<<<blocks((uint64_t)b.pix[b.views] + 1, 256), 256, 0, s>>>(b, meta, keys, vals, work);
  return cudaGetLastError();
}

cudaError_t launch_region_keys(const QueueBatch& b, const RayMeta* meta, const uint32_t* sorted,
                               const uint32_t* before, uint32_t R, uint32_t* region, uint32_t* rank, RayMeta* queue,
                               uint32_t* ids, uint32_t id_base, cudaStream_t s) {
  if (!b.act[b.views]) return cudaSuccess;
  k_region_keys<<<blocks(b.act[b.views], 256), 256, 0, s>>>(b, meta, sorted, before, R, region, rank, queue, ids,
                                                           id_base);
  return cudaGetLastError();
}

cudaError_t launch_region_bounds(const QueueBatch& b, const uint32_t* region, const uint32_t* rank,
                                 const uint32_t* keys, uint32_t R, uint32_t* bounds, uint32_t* work, cudaStream_t s) {
  k_region_bounds<<<blocks((uint64_t)b.act[b.views] + 1, 256), 256, 0, s>>>(b, region, rank, keys, R, bounds, work);
  return cudaGetLastError();
}

cudaError_t launch_region_home(const QueueBatch& b, const uint32_t* region, const uint32_t* rank,
                               const uint32_t* before, const uint32_t* bounds, uint32_t share, uint32_t* flag,
                               cudaStream_t s) {
  k_region_home<<<blocks((uint64_t)b.act[b.views] + 1, 256), 256, 0, s>>>(b, region, rank, before, bounds, share, flag);
  return cudaGetLastError();
}

cudaError_t launch_region_emit(const QueueBatch& b, const RayMeta* meta, const uint32_t* sorted, const uint32_t* rank,
                               const uint32_t* place, const uint32_t* bounds, uint32_t R, uint32_t at,
                               uint32_t id_base, RayMeta* queue, uint32_t* ids, uint32_t* rstart, uint32_t* lbase,
                               uint32_t* lsingle, cudaStream_t s) {
  const uint64_t rays = 2 * (uint64_t)b.act[b.views], rows = (uint64_t)b.views * (R + 1);
  k_region_emit<<<blocks(rays > rows ? rays : rows, 256), 256, 0, s>>>(b, meta, sorted, rank, place, bounds, R, at,
                                                                      id_base, queue, ids, rstart, lbase, lsingle);
  return cudaGetLastError();
}

cudaError_t launch_leftover_prefix(const uint32_t* lsingle, uint32_t V, uint32_t* prefix, cudaStream_t s) {
  k_leftover_prefix<<<1, 32, 0, s>>>(lsingle, V, prefix);
  return cudaGetLastError();
}

cudaError_t launch_loud_prefix(const RayMeta* meta, uint32_t r_first, uint32_t n, const uint32_t* inc_pair,
                               const float* inc_len, uint32_t pair_base, uint32_t n_loud, uint32_t* loff,
                               uint2* loud, QuietRay* ray, bool emit, cudaStream_t s) {
  if (!n) return cudaSuccess;
  const unsigned g = blocks((uint64_t)n * 32, 256);
  if (emit)
    k_loud_prefix<true><<<g, 256, 0, s>>>(meta, r_first, n, inc_pair, inc_len, pair_base, n_loud, loff, loud, ray);
  else
    k_loud_prefix<false><<<g, 256, 0, s>>>(meta, r_first, n, inc_pair, inc_len, pair_base, n_loud, loff, loud,
                                           ray);
  return cudaGetLastError();
}

cudaError_t launch_quiet_prefix(const BpArrays& a, uint32_t r_first, uint32_t n, uint32_t pair_base,
                                uint32_t n_loud, QuietRay* ray, cudaStream_t s) {
  if (!n) return cudaSuccess;
  const unsigned g = blocks((uint64_t)n * 32, 256);
  if (a.half_streams)
    k_quiet_prefix<__half><<<g, 256, 0, s>>>(a.meta, r_first, n, a.inc_pair, a.inc_len, a.pair_lnq16, pair_base,
                                             n_loud, ray);
  else
    k_quiet_prefix<float><<<g, 256, 0, s>>>(a.meta, r_first, n, a.inc_pair, a.inc_len, a.pair_lnq, pair_base,
                                            n_loud, ray);
  return cudaGetLastError();
}

cudaError_t launch_pair_update(const BpArrays& a, uint32_t k0, uint32_t k1, uint32_t j0, uint32_t j1,
                               const uint32_t* tile_first, int jacobi, cudaStream_t s) {
  (void)j0;
  if (k1 <= k0) return cudaSuccess;
  uint32_t ntiles = (k1 - k0 + kTile - 1) / kTile;
  if (a.pair_variant)
    k_pair_reduce<true><<<ntiles, kTileThreads, 0, s>>>(a.dperm, a.inc_pl, a.dseg, tile_first, k0, k1, j1,
                                                        a.drun, a.pair_m, a.L, a.pair_dm, jacobi);
  else
    k_pair_reduce<false><<<ntiles, kTileThreads, 0, s>>>(a.dperm, a.inc_pl, a.dseg, tile_first, k0, k1, j1,
                                                         a.drun, a.pair_m, a.L, a.pair_dm, jacobi);
  return cudaGetLastError();
}

cudaError_t launch_drun(const uint32_t* dpair, uint32_t n, const uint32_t* pair_vox, const float* cum,
                        const float* stat, uint4* drun, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_drun<<<blocks(n, 256), 256, 0, s>>>(dpair, n, pair_vox, cum, stat, drun);
  return cudaGetLastError();
}

cudaError_t launch_static_pairs(const BpArrays& a, uint32_t p0, uint32_t p1, int jacobi,
                                cudaStream_t s) {
  if (p1 <= p0) return cudaSuccess;
  k_static_pairs<<<blocks(p1 - p0, 256), 256, 0, s>>>(p0, p1, a.pair_ndyn, a.pair_stat, a.pair_vox,
                                                      a.pair_m, a.pair_cum, a.L, a.pair_dm, jacobi);
  return cudaGetLastError();
}

cudaError_t launch_tile_first(const uint32_t* seg, uint32_t p0, uint32_t p1, uint32_t k0, uint32_t k1,
                              uint32_t* out, cudaStream_t s) {
  if (k1 <= k0) return cudaSuccess;
  uint32_t ntiles = (k1 - k0 + kTile - 1) / kTile;
  k_tile_first<<<blocks(ntiles, 256), 256, 0, s>>>(seg, p0, p1, k0, ntiles, out);
  return cudaGetLastError();
}

uint32_t pair_update_tiles(uint32_t n) { return (n + kTile - 1) / kTile; }

cudaError_t launch_voxel_apply(const uint32_t* vseg, const uint32_t* vpairs, const uint32_t* vvox,
                               uint32_t nvox, const float* pair_dm, float* L, cudaStream_t s) {
  if (!nvox) return cudaSuccess;
  k_voxel_apply<<<blocks(nvox, 256), 256, 0, s>>>(vseg, vpairs, vvox, nvox, pair_dm, L);
  return cudaGetLastError();
}

cudaError_t launch_active_voxels(const uint32_t* pair_vox, const float* cum, uint32_t np, uint8_t* flag,
                                 int64_t nvox, cudaStream_t s) {
  if (nvox <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(flag, 0, (size_t)nvox, s);
  if (e != cudaSuccess) return e;
  if (np) k_touch_pairs<<<blocks(np, 256), 256, 0, s>>>(pair_vox, cum, np, flag, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_mark_active(const uint32_t* pair_vox, const float* cum, uint32_t np, uint8_t* flag,
                               cudaStream_t s) {
  if (!np) return cudaSuccess;
  k_touch_pairs<<<blocks(np, 256), 256, 0, s>>>(pair_vox, cum, np, flag, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_belief_refresh(const float* L, const uint8_t* active, int64_t nvox, float* belief,
                                  cudaStream_t s) {
  if (nvox <= 0) return cudaSuccess;
  k_belief_refresh<<<(unsigned)std::min<int64_t>(blocks(nvox, 256), 8192), 256, 0, s>>>(L, active, nvox, belief);
  return cudaGetLastError();
}

cudaError_t launch_max_abs_diff(const float* a, const float* b, int64_t n, uint32_t* out,
                                cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(out, 0, 4, s);
  if (e != cudaSuccess || n <= 0) return e;
  int64_t nb = std::min<int64_t>((n + 255) / 256, 4096);
  k_max_abs_diff<<<(unsigned)nb, 256, 0, s>>>(a, b, n, out);
  return cudaGetLastError();
}

cudaError_t launch_warm_split(const uint32_t* vseg, const uint32_t* vpairs, const uint32_t* vvox,
                              uint32_t nvox, const float* L_pred, float lp, const float* base, const float* cum,
                              const float* stat, const uint32_t* ndyn, float* m, cudaStream_t s) {
  if (!nvox) return cudaSuccess;
  k_warm_split<<<blocks(nvox, 256), 256, 0, s>>>(vseg, vpairs, vvox, nvox, L_pred, lp, base, cum, stat, ndyn, m);
  return cudaGetLastError();
}

cudaError_t launch_voxel_features(const uint32_t* vseg, const uint32_t* vpairs, const uint32_t* vvox,
                                  uint32_t nvox, const float* cum, const float* stat, const float* hit,
                                  const float* belief, int64_t n_slots_vox, float* feat, cudaStream_t s) {
  if (n_slots_vox <= 0) return cudaSuccess;
  k_feat_belief<<<blocks(n_slots_vox, 256), 256, 0, s>>>(belief, n_slots_vox, feat);
  if (nvox) k_voxel_features<<<blocks(nvox, 256), 256, 0, s>>>(vseg, vpairs, vvox, nvox, cum, stat, hit, feat);
  return cudaGetLastError();
}

cudaError_t launch_voxel_rebuild(const uint32_t* vseg, const uint32_t* vpairs, const uint32_t* vvox,
                                 uint32_t nvox, const float* m, const float* cum, float* L, float* belief,
                                 cudaStream_t s) {
  if (!nvox) return cudaSuccess;
  k_voxel_rebuild<<<blocks(nvox, 256), 256, 0, s>>>(vseg, vpairs, vvox, nvox, m, cum, L, belief);
  return cudaGetLastError();
}

cudaError_t launch_remove_messages(const BpArrays& a, uint32_t p0, uint32_t p1, cudaStream_t s) {
  if (p1 <= p0) return cudaSuccess;
  k_remove_messages<<<blocks(p1 - p0, 256), 256, 0, s>>>(a.pair_vox, a.pair_m, p0, p1, a.L, a.belief);
  return cudaGetLastError();
}

cudaError_t launch_fold_messages(const uint32_t* pair_vox, const float* pair_m, uint32_t n, float* base,
                                 cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_fold_messages<<<blocks(n, 256), 256, 0, s>>>(pair_vox, pair_m, n, base);
  return cudaGetLastError();
}

cudaError_t launch_remap_scatter(const uint32_t* pair_vox, const float* pair_m, uint32_t n,
                                 float* dense, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_remap_scatter<<<blocks(n, 256), 256, 0, s>>>(pair_vox, pair_m, n, dense);
  return cudaGetLastError();
}

cudaError_t launch_remap_gather(const uint32_t* pair_vox, float* pair_m, uint32_t n,
                                const float* dense, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_remap_gather<<<blocks(n, 256), 256, 0, s>>>(pair_vox, pair_m, n, dense);
  return cudaGetLastError();
}

__global__ void k_to_half(const float* __restrict__ in, int64_t n, __half* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __float2half_rn(in[i]);
}

cudaError_t launch_to_half(const float* in, int64_t n, __half* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_to_half<<<(unsigned)std::min<int64_t>(blocks(n, 256), 16384), 256, 0, s>>>(in, n, out);
  return cudaGetLastError();
}

cudaError_t launch_fill_u32(uint32_t* p, int64_t n, uint32_t v, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_fill_u32<<<blocks(n, 256), 256, 0, s>>>(p, n, v);
  return cudaGetLastError();
}

cudaError_t launch_fill_f32(float* p, int64_t n, float v, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_fill<<<blocks(n, 256), 256, 0, s>>>(p, n, v);
  return cudaGetLastError();
}

cudaError_t launch_vflag(const uint32_t* sk, uint32_t n, uint32_t* flag, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_vflag<<<blocks(n, 256), 256, 0, s>>>(sk, n, flag);
  return cudaGetLastError();
}

cudaError_t launch_voxel_keys(const uint32_t* pair_vox, uint32_t n, const uint8_t* loud, uint32_t top,
                              uint32_t* key, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_voxel_keys<<<blocks(n, 256), 256, 0, s>>>(pair_vox, n, loud, top, key);
  return cudaGetLastError();
}

cudaError_t launch_vassign(const uint32_t* sk, const uint32_t* flag, const uint32_t* scan, uint32_t n, uint32_t top,
                           uint32_t* vvox, uint32_t* vseg, uint32_t* n_loud, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_vassign<<<blocks(n, 256), 256, 0, s>>>(sk, flag, scan, n, top, vvox, vseg, n_loud);
  return cudaGetLastError();
}

cudaError_t launch_touch_counts(const uint32_t* pair_vox, const float* cum, uint32_t np, uint8_t* flag,
                                int64_t nvox, unsigned long long* out2, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(out2, 0, 16, s);
  if (e == cudaSuccess && nvox > 0) e = cudaMemsetAsync(flag, 0, (size_t)nvox, s);
  if (e != cudaSuccess) return e;
  if (np) k_touch_pairs<<<blocks(np, 256), 256, 0, s>>>(pair_vox, cum, np, flag, out2);
  if (nvox > 0)
    k_count_flags<<<(unsigned)std::min<int64_t>(blocks(nvox, 256), 4096), 256, 0, s>>>(flag, nvox, out2 + 1);
  return cudaGetLastError();
}

cudaError_t launch_scatter_const(const uint32_t* idx, uint32_t n, float v, float* dense,
                                 cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_scatter_const<<<blocks(n, 256), 256, 0, s>>>(idx, n, v, dense);
  return cudaGetLastError();
}

}  // namespace mrf
