// mrf_like_pixel.cuh -- per-pixel log-likelihood of a depth return under the
// belief field (src/cuda/gvdbkernels.cu:183-293, 1246-1274).  Visibility
// V = exp(-sum alpha l) with alpha = -ln(1 - p); each voxel adds
// (V_prev - V) * P(z | first return in the voxel); the tail adds
// V_end * P(z | no return).  Every active brick to the volume exit counts.
//
// P is LIKE_EPS at every voxel outside the return's window, so their sum is
// LIKE_EPS times the visibility lost there: V at the near limit, minus V at
// the end, minus what the window took.  Outside the window a voxel then
// costs its exponent only -- ln(1 - p) by its series for the small p of free
// space -- and two exponentials inside it.  Inactive bricks are left in one
// go.  A ray whose visibility is below 1e-30 while the sum is above 1e-18
// ends: the rest cannot change the FP32 result.
#pragma once
#include "mrf_geometry.cuh"
#include "mrf_internal.h"

namespace mrf {

// ln(1 - p): the Taylor series to p^5 below 1/64 (next term p^6/6: relative
// 1.6e-10), CUDA's log1pf above
__device__ __forceinline__ float log_free(float p) {
  if (!(fabsf(p) <= 0.015625f)) return log1pf(-p);
  return -p * (1.0f + p * (0.5f + p * (1.0f / 3.0f + p * (0.25f + p * 0.2f))));
}

// e^x - 1: the Taylor series to x^6 / 720 up to 0.04 (next term relative
// 8e-13), CUDA's expm1f beyond
__device__ __forceinline__ float expm1_free(float x) {
  if (!(fabsf(x) <= 0.04f)) return expm1f(x);
  return x * (1.0f + x * (0.5f + x * (1.0f / 6.0f + x * (1.0f / 24.0f + x * (1.0f / 120.0f + x * (1.0f / 720.0f))))));
}

__device__ __forceinline__ float likelihood_pixel(const Geom& g, const Pose& P,
                                                  const float* __restrict__ belief, int pix, float d) {
  const int x = pix % g.cols, y = pix / g.cols;
  const Sensor c = sensor_at(g, x, y);
  Ray ray;
  ray_setup(g, P, x, y, ray);
  // A: exponent of the visibility; Vz: visibility at the near limit; inside
  // the window: sum of w and of w P
  float A = 0.0f, Vz = 1.0f, win_w = 0.0f, win = 0.0f, prev_s = 0.0f, s_last = 0.0f;
  bool first_run = true, run_open = false, near = true;
  const float s_win = window_start(c, d, 3.0f, 0.9999f);  // the window begins behind it
  Dda r;
  if (dda_init(r, g, ray)) {
    while (r.alive && r.guard > 0) {
      // a brick hands s + bias(s) to the next as its previous s
      // (gvdbkernels.cu:209, 292)
      if (run_open) {
        prev_s = s_last + c.bias(s_last);
        run_open = false;
        if (A < -69.0f && !near) {
          const float V = expf(A);
          if (kLikeEps * (Vz - V - win_w) + win > 1e-18f) break;
        }
      }
      const int slot = g.brick_slot[r.lin];
      if (slot < 0) {
        int steps;
        dda_cross(r, g, ray, steps);
        continue;
      }
      if (first_run) {
        prev_s = fm(r.tprev, ray.mult);
        first_run = false;
      }
      run_open = true;
      const float* __restrict__ bel = belief + (int64_t)slot * kBrickVox;
      // the brick's voxels, the lanes of a warp together
      bool left;
      do {
        const float p = bel[dda_local(r)];
        float l, tin, te;
        left = dda_step(r, g, l, tin, te);
        const float dA = log_free(p) * l;
        const float s = fm(te, ray.mult);
        if (near && !(s < kZMin)) {
          Vz = expf(A);
          near = false;
        }
        if (s >= s_win && !near && fabsf(fs(fa(s, c.bias(s)), d)) <= fm(3.0f, c.sigma(s))) {
          const float w = expf(A) * -expm1f(dA);
          win_w += w;
          win += w * ((1.0f - kLikeEps) * 0.5f * (potential(c, s, d) + potential(c, prev_s, d)));
        }
        A += dA;
        prev_s = s;
      } while (!left && r.guard > 0);
      s_last = prev_s;
    }
  }
  const float V = expf(A);
  if (near) Vz = V;
  const float sum = kLikeEps * (Vz - V - win_w) + win + V * (d >= kZMax ? 1.0f - kLikeEps : kLikeEps);
  return logf(sum);
}

// exclusive prefix and total over the kSplit lanes of a ray (mask: those lanes).
// The prefix is shifted out of the inclusive scan, not formed as scan minus
// value: a voxel of occupancy 1 makes a lane's value -inf, and behind a wall
// (-100) the subtraction leaves 4e-6 in the exponent of the lane's own brick.
__device__ __forceinline__ float split_prefix(float v, unsigned mask, int sub, float& total) {
  float incl = v;
#pragma unroll
  for (int o = 1; o < kSplit; o <<= 1) {
    const float u = __shfl_up_sync(mask, incl, o, kSplit);
    if (sub >= o) incl += u;
  }
  total = __shfl_sync(mask, incl, kSplit - 1, kSplit);
  const float before = __shfl_up_sync(mask, incl, 1, kSplit);
  return sub ? before : 0.0f;
}
__device__ __forceinline__ float split_sum(float v, unsigned mask) {
#pragma unroll
  for (int o = 1; o < kSplit; o <<= 1) v += __shfl_xor_sync(mask, v, o, kSplit);
  return v;
}

// The same by kSplit lanes (sub: this one), which take the ray's active bricks
// in turn.  A brick's part is formed from its own start (exponent a, window
// sums relative to the visibility there) and scaled by the visibility that
// the lanes before it leave.
__device__ __forceinline__ float likelihood_pixel_split(const Geom& g, const Pose& P,
                                                        const float* __restrict__ belief, int pix, float d,
                                                        unsigned mask, int sub) {
  const int x = pix % g.cols, y = pix / g.cols;
  const Sensor c = sensor_at(g, x, y);
  Ray ray;
  ray_setup(g, P, x, y, ray);
  float A = 0.0f, Vz = 0.0f, win_w = 0.0f, win = 0.0f;
  bool near = true;  // no voxel behind the near limit so far
  const float s_win = window_start(c, d, 3.0f, 0.9999f);
  Dda r;
  bool going = dda_init(r, g, ray);
  int slot = going ? dda_next_active(r, g, ray) : -1;
  float prev_s = slot >= 0 ? fm(r.tprev, ray.mult) : 0.0f;
  // past n active bricks, to the next one
  auto skip = [&](int n) {
    for (int k = 0; k < n && slot >= 0; ++k) {
      int steps;
      const float s = fm(dda_cross(r, g, ray, steps), ray.mult);
      prev_s = s + c.bias(s);
      slot = dda_next_active(r, g, ray);
    }
  };
  skip(sub);
  while (__any_sync(mask, slot >= 0)) {
    float a = 0.0f, w_rel = 0.0f, p_rel = 0.0f, a_near = 0.0f;
    bool crossed = false;  // a voxel of the brick lies behind the near limit
    if (slot >= 0) {
      const float* __restrict__ bel = belief + (int64_t)slot * kBrickVox;
      bool left;
      do {
        const float p = bel[dda_local(r)];
        float l, tin, te;
        left = dda_step(r, g, l, tin, te);
        const float dA = log_free(p) * l;
        const float s = fm(te, ray.mult);
        if (!crossed && !(s < kZMin)) {
          crossed = true;
          a_near = a;
        }
        if (s >= s_win && crossed && fabsf(fs(fa(s, c.bias(s)), d)) <= fm(3.0f, c.sigma(s))) {
          const float w = expf(a) * -expm1f(dA);
          w_rel += w;
          p_rel += w * ((1.0f - kLikeEps) * 0.5f * (potential(c, s, d) + potential(c, prev_s, d)));
        }
        a += dA;
        prev_s = s;
      } while (!left && r.guard > 0);
      prev_s += c.bias(prev_s);
      slot = dda_next_active(r, g, ray);
      skip(kSplit - 1);
    }
    float sum;
    const float A0 = A + split_prefix(a, mask, sub, sum);
    const float V0 = expf(A0);
    win_w += V0 * w_rel;
    win += V0 * p_rel;
    // the first brick, in order, with a voxel behind the near limit
    const unsigned far = __ballot_sync(mask, crossed) & mask;
    if (near && far) {
      Vz = __shfl_sync(mask, expf(A0 + a_near), __ffs(far) - 1);
      near = false;
    }
    A += sum;
    if (A < -69.0f && !near) {
      const float V = expf(A);
      if (kLikeEps * (Vz - V - split_sum(win_w, mask)) + split_sum(win, mask) > 1e-18f) break;
    }
  }
  const float V = expf(A);
  if (near) Vz = V;
  const float sum = kLikeEps * (Vz - V - split_sum(win_w, mask)) + split_sum(win, mask) +
                    V * (d >= kZMax ? 1.0f - kLikeEps : kLikeEps);
  return logf(sum);
}

// FP64 sum over the block, returned on thread 0 (blockDim.x == kThreadsLike)
template <int kThreadsLike>
__device__ __forceinline__ double like_block_sum(double v) {
  __shared__ double sh[kThreadsLike / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kThreadsLike / 32; ++i) t += sh[i];
  }
  return t;
}

}  // namespace mrf
