// mrf_like.cu -- per-view log-likelihood of a depth image under the belief
// field (src/cuda/gvdbkernels.cu:183-293, 1246-1274), with the frame sum
// (src/cuda/gvdbhelper.cu:10-14) fused as a deterministic two-level
// reduction: FP64 block partials, then one ordered pass over the partials.
#include "mrf_internal.h"
#include "mrf_like_pixel.cuh"

namespace mrf {

namespace {

constexpr int kLikeThreads = 128;

// A warp per tile of pixels (per-pixel body in mrf_like_pixel.cuh).
__global__ void __launch_bounds__(kLikeThreads)
    k_likelihood(Geom g, Pose P, const float* __restrict__ depth, const float* __restrict__ belief,
                 float* __restrict__ out_img, double* __restrict__ partials) {
  const int pix = tile_pixel<kViewTileX, kViewTileY>(
      g.rows, g.cols, (blockIdx.x * (int64_t)kLikeThreads + threadIdx.x) >> 5, threadIdx.x & 31);
  float val = 0.0f;
  if (pix >= 0) {
    float d = depth[pix];
    if (d > 0.0f) val = likelihood_pixel(g, P, belief, pix, d);
    if (out_img) out_img[pix] = val;
  }
  double t = like_block_sum<kLikeThreads>((double)val);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}

// the same with kSplit lanes per pixel: a warp's tile is 4 x 2
__global__ void __launch_bounds__(kLikeThreads)
    k_likelihood_split(Geom g, Pose P, const float* __restrict__ depth, const float* __restrict__ belief,
                       float* __restrict__ out_img, double* __restrict__ partials) {
  const int lane = threadIdx.x & 31, sub = lane % kSplit;
  const int pix = tile_pixel<4, 2>(g.rows, g.cols, (blockIdx.x * (int64_t)kLikeThreads + threadIdx.x) >> 5, lane / kSplit);
  float val = 0.0f;
  if (pix >= 0) {
    const float d = depth[pix];
    const unsigned mask = ((1u << kSplit) - 1u) << (lane - sub);
    if (d > 0.0f) val = likelihood_pixel_split(g, P, belief, pix, d, mask, sub);
    if (out_img && sub == 0) out_img[pix] = val;
  }
  double t = like_block_sum<kLikeThreads>(sub == 0 ? (double)val : 0.0);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}
static_assert(kSplit * 4 * 2 == 32, "a warp per tile");

__global__ void k_reduce_partials(const double* __restrict__ partials, int n, float* out) {
  __shared__ double sh[256];
  double v = 0.0;
  // fixed assignment of partials to threads and a fixed tree: reproducible
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += partials[i];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = (float)sh[0];
}

}  // namespace

int likelihood_blocks(const Geom& g, int num_sms) {
  constexpr int kTiles = kLikeThreads / 32;
  const int64_t tiles = split_rays(g.rows, g.cols, num_sms) ? (int64_t)((g.cols + 3) / 4) * ((g.rows + 1) / 2)
                                                            : image_tiles(g.rows, g.cols);
  return (int)((tiles + kTiles - 1) / kTiles);
}

cudaError_t launch_likelihood(const Geom& g, const Pose& P, const float* depth, const float* belief,
                              float* out_img, double* partials, int num_sms, cudaStream_t s) {
  const int nblocks = likelihood_blocks(g, num_sms);
  if (split_rays(g.rows, g.cols, num_sms))
    k_likelihood_split<<<nblocks, kLikeThreads, 0, s>>>(g, P, depth, belief, out_img, partials);
  else
    k_likelihood<<<nblocks, kLikeThreads, 0, s>>>(g, P, depth, belief, out_img, partials);
  return cudaGetLastError();
}

cudaError_t launch_reduce_partials(const double* partials, int n, float* out_sum, cudaStream_t s) {
  k_reduce_partials<<<1, 256, 0, s>>>(partials, n, out_sum);
  return cudaGetLastError();
}

}  // namespace mrf
