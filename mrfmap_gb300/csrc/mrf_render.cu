// mrf_render.cu -- evaluation renders over the belief field, on the same
// traversal as the likelihood (every active brick to the volume exit):
//   mode 0  expected depth            gvdbkernels.cu:295-354, 1332-1363
//   mode 1  accuracy (peak of the first-return density within 1 sigma)
//                                      gvdbkernels.cu:183-293, 1066-1104
//   mode 2  simple accuracy (first voxel above a threshold)
//                                      gvdbkernels.cu:135-181, 1106-1134
//   mode 3  occupancy at the first voxel past the measurement
//                                      gvdbkernels.cu:183-293, 1136-1162
// Labels of modes 1-3 are histogrammed (-1, 0, 1, 2) for the frame scores of
// src/cuda/gvdbhelper.cu:16-62 (integer counts: order-independent).
#include "mrf_geometry.cuh"
#include "mrf_internal.h"
#include "mrf_like_pixel.cuh"

namespace mrf {

namespace {

constexpr int kRenderThreads = 128;

template <int kMode>
__device__ float render_pixel(const Geom& g, const Pose& P, const float* __restrict__ belief, int pix,
                              float d, float thresh) {
  const int x = pix % g.cols, y = pix / g.cols;
  const Sensor c = sensor_at(g, x, y);
  Ray ray;
  ray_setup(g, P, x, y, ray);
  float A = 0.0f, Vprev = 1.0f, sum = 0.0f, peak = 0.0f, s_last = 0.0f;
  int peak_ok = 0, occ = -1;
  bool run_open = false;
  Dda r;
  if (dda_init(r, g, ray)) {
    const Corner corner(r);
    while (r.alive && r.guard > 0) {
      // simple accuracy: a brick that ends past the return is a miss
      if (kMode == 2 && run_open && s_last >= d) return 0.0f;
      // expected depth: nothing visible is left, the rest cannot change the
      // FP32 sum
      if (kMode == 0 && Vprev < 1e-30f && sum > 1e-18f) break;
      // the label is known
      if (kMode == 3 && occ != -1) break;
      run_open = false;
      const int slot = g.brick_slot[r.lin];
      if (slot < 0) {
        int steps;
        dda_cross(r, g, ray, steps);
        continue;
      }
      run_open = true;
      const float* __restrict__ bel = belief + (int64_t)slot * kBrickVox;
      // the brick's voxels, the lanes of a warp together
      bool left;
      do {
        const float p = bel[dda_local(r)];
        const float vx = corner.x(r), vy = corner.y(r), vz = corner.z(r);
        float l, tin, te;
        left = dda_step(r, g, l, tin, te);
        const float s = fm(te, ray.mult);
        s_last = s;
        if (kMode == 2) {
          if (p >= thresh) return fabsf(s - d) <= g.res ? 1.0f : 2.0f;
        }
        if (kMode == 3) {
          if (fs(fa(s, c.bias(s)), d) > 0.0f && occ == -1) occ = p >= thresh ? 1 : 0;
        }
        if (kMode == 0 && p != 0.0f) {
          const float dA = log_free(p) * l;
          const float dv = Vprev * -expm1_free(dA);
          A += dA;
          Vprev = expf(A);
          // z-depth of the voxel's corner (the GVDB atlas-to-world position)
          const float zc = fabsf(P.m[2] * (vx - ray.o[0]) + P.m[6] * (vy - ray.o[1]) + P.m[10] * (vz - ray.o[2])) *
                           g.res;
          sum += dv * zc;
        }
        if (kMode == 1) {
          const float dA = log1pf(-p) * l;
          A += dA;
          const float V = expf(A);
          const float dv = Vprev * -expm1f(dA);
          const float w = dv / l;
          if (w > peak) {
            peak = w;
            peak_ok = fabsf(fs(fa(s, c.bias(s)), d)) <= c.sigma(s);
          }
          Vprev = V;
        }
      } while (!left && r.guard > 0);
    }
  }
  if (kMode == 0) return sum / (1.0f - Vprev + kFEps);
  if (kMode == 1) {
    if (peak > 0.0f && Vprev >= 0.9f) return fa(s_last, c.bias(s_last)) <= d ? -1.0f : 0.0f;
    if (peak > 0.0f) return (float)peak_ok;
    return -1.0f;
  }
  if (kMode == 2) return (run_open && s_last >= d) ? 0.0f : -1.0f;
  return (float)occ;
}

// Expected depth by kSplit lanes per pixel, as likelihood_pixel_split: a
// brick's depth sum relative to the visibility at its start.
__device__ __forceinline__ float depth_pixel_split(const Geom& g, const Pose& P, const float* __restrict__ belief,
                                                   int pix, unsigned mask, int sub) {
  Ray ray;
  ray_setup(g, P, pix % g.cols, pix / g.cols, ray);
  float A = 0.0f, sum = 0.0f;
  Dda r;
  const bool in = dda_init(r, g, ray);
  if (!in) r = Dda{};
  const Corner corner(r);
  int slot = in ? dda_next_active(r, g, ray) : -1;
  auto skip = [&](int n) {
    for (int k = 0; k < n && slot >= 0; ++k) {
      int steps;
      dda_cross(r, g, ray, steps);
      slot = dda_next_active(r, g, ray);
    }
  };
  skip(sub);
  while (__any_sync(mask, slot >= 0)) {
    float a = 0.0f, rel = 0.0f;
    if (slot >= 0) {
      const float* __restrict__ bel = belief + (int64_t)slot * kBrickVox;
      bool left;
      do {
        const float p = bel[dda_local(r)];
        const float vx = corner.x(r), vy = corner.y(r), vz = corner.z(r);
        float l, tin, te;
        left = dda_step(r, g, l, tin, te);
        if (p != 0.0f) {
          const float dA = log_free(p) * l;
          rel += expf(a) * -expm1_free(dA) *
                 (fabsf(P.m[2] * (vx - ray.o[0]) + P.m[6] * (vy - ray.o[1]) + P.m[10] * (vz - ray.o[2])) * g.res);
          a += dA;
        }
      } while (!left && r.guard > 0);
      slot = dda_next_active(r, g, ray);
      skip(kSplit - 1);
    }
    float total;
    sum += expf(A + split_prefix(a, mask, sub, total)) * rel;
    A += total;
    if (A < -69.0f && split_sum(sum, mask) > 1e-18f) break;
  }
  return split_sum(sum, mask) / (1.0f - expf(A) + kFEps);
}

__global__ void __launch_bounds__(kRenderThreads)
    k_depth_split(Geom g, Pose P, const float* __restrict__ belief, float* __restrict__ out) {
  const int lane = threadIdx.x & 31, sub = lane % kSplit;
  const int pix =
      tile_pixel<4, 2>(g.rows, g.cols, (blockIdx.x * (int64_t)kRenderThreads + threadIdx.x) >> 5, lane / kSplit);
  if (pix < 0) return;
  const float v = depth_pixel_split(g, P, belief, pix, ((1u << kSplit) - 1u) << (lane - sub), sub);
  if (sub == 0) out[pix] = v;
}

template <int kMode>
__global__ void __launch_bounds__(kRenderThreads)
    k_render(Geom g, Pose P, const float* __restrict__ depth, const float* __restrict__ belief,
             float thresh, float* __restrict__ out, unsigned long long* __restrict__ counts) {
  __shared__ unsigned int hist[4];
  if (threadIdx.x < 4) hist[threadIdx.x] = 0;
  __syncthreads();
  const int pix =
      tile_pixel<kViewTileX, kViewTileY>(g.rows, g.cols, (blockIdx.x * (int64_t)kRenderThreads + threadIdx.x) >> 5,
                                         threadIdx.x & 31);
  if (pix >= 0) {
    float d = depth[pix];
    float v;
    if (kMode != 0 && !(d > 0.0f)) v = -1.0f;
    else v = render_pixel<kMode>(g, P, belief, pix, d, thresh);
    out[pix] = v;
    if (kMode != 0) {
      int k = (int)v + 1;
      if (k >= 0 && k < 4) atomicAdd(&hist[k], 1u);
    }
  }
  __syncthreads();
  if (kMode != 0 && threadIdx.x < 4 && hist[threadIdx.x])
    atomicAdd(&counts[threadIdx.x], (unsigned long long)hist[threadIdx.x]);
}

// Per-voxel record of one pixel's ray (src/cuda/gvdbkernels.cu:573-672,
// 1365-1384): ten floats per active voxel along the ray to the volume exit
// -- [0] exit distance s, [1] belief, [2..3] voxel id (u64: slot*512 +
// local), [4] w = (V_prev - V) / l, [5] visibility V, [6..7] brick slot
// (u64), [8] brick-local x, y, z as bytes -- and the record count in the
// last float.  One thread: this is a debugging probe.
__global__ void k_pixel_diag(Geom g, Pose P, const float* __restrict__ belief, int x, int y,
                             float* __restrict__ out, int64_t n_floats) {
  if (blockIdx.x || threadIdx.x) return;
  constexpr int kStride = 10;
  const int64_t cap = (n_floats - 1) / kStride;
  Ray ray;
  ray_setup(g, P, x, y, ray);
  int64_t count = 0;
  float A = 0.0f, Vprev = 1.0f;
  Dda r;
  if (dda_init(r, g, ray)) {
    bool enter = true;
    int slot = -1;
    while (r.alive && r.guard > 0) {
      if (enter) {
        slot = g.brick_slot[r.lin];
        if (slot < 0) {
          int steps;
          dda_cross(r, g, ray, steps);
          continue;
        }
      }
      if (count >= cap) break;
      const int loc = (int)dda_local(r);
      const uint32_t xyz = r.loc;
      float l, tin, te;
      enter = dda_step(r, g, l, tin, te);
      const float p = belief[(int64_t)slot * kBrickVox + loc];
      A += log1pf(-p) * l;
      const float V = expf(A);
      float* rec = out + count * kStride;
      rec[0] = fm(te, ray.mult);
      rec[1] = p;
      reinterpret_cast<unsigned long long*>(out)[count * (kStride / 2) + 1] =
          (unsigned long long)slot * kBrickVox + loc;
      rec[4] = (Vprev - V) / l;
      rec[5] = V;
      reinterpret_cast<unsigned long long*>(out)[count * (kStride / 2) + 3] = (unsigned long long)slot;
      unsigned char* b = reinterpret_cast<unsigned char*>(rec + 8);
      b[0] = (unsigned char)(xyz >> 8 & 7);
      b[1] = (unsigned char)(xyz >> 4 & 7);
      b[2] = (unsigned char)(xyz & 7);
      Vprev = V;
      ++count;
    }
  }
  out[n_floats - 1] = (float)count;
}

}  // namespace

cudaError_t launch_pixel_diag(const Geom& g, const Pose& P, const float* belief, int x, int y, float* out,
                              int64_t n_floats, cudaStream_t s) {
  k_pixel_diag<<<1, 1, 0, s>>>(g, P, belief, x, y, out, n_floats);
  return cudaGetLastError();
}

cudaError_t launch_render(int mode, const Geom& g, const Pose& P, const float* depth,
                          const float* belief, float thresh, float* out, unsigned long long* counts,
                          int num_sms, cudaStream_t s) {
  if (mode == 0 && split_rays(g.rows, g.cols, num_sms)) {
    const int64_t warps = (int64_t)((g.cols + 3) / 4) * ((g.rows + 1) / 2);
    k_depth_split<<<(unsigned)((warps + kRenderThreads / 32 - 1) / (kRenderThreads / 32)), kRenderThreads, 0, s>>>(
        g, P, belief, out);
    return cudaGetLastError();
  }
  constexpr int kTiles = kRenderThreads / 32;
  const int nb = (int)((image_tiles(g.rows, g.cols) + kTiles - 1) / kTiles);
  switch (mode) {
    case 0: k_render<0><<<nb, kRenderThreads, 0, s>>>(g, P, depth, belief, thresh, out, counts); break;
    case 1: k_render<1><<<nb, kRenderThreads, 0, s>>>(g, P, depth, belief, thresh, out, counts); break;
    case 2: k_render<2><<<nb, kRenderThreads, 0, s>>>(g, P, depth, belief, thresh, out, counts); break;
    case 3: k_render<3><<<nb, kRenderThreads, 0, s>>>(g, P, depth, belief, thresh, out, counts); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace mrf
