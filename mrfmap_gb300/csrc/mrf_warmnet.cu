// mrf_warmnet.cu -- the learned warm start's network and its training
// kernels.  Three 3x3x3 convolutions over one 8^3 brick at a time
// (4 -> 16 -> 16 -> 1 channels, ReLU after the first two, zeros beyond the
// brick faces) predict a voxel's converged log-odds from four per-voxel
// features.  Every convolution -- forward, the input gradient (the same
// convolution with flipped, transposed weights) and the weight gradient --
// runs on the tensor cores as BF16 x BF16 -> FP32 (mma.sync m16n8k16) over
// operands staged in shared memory; FP32 master weights, Adam.
//
// A brick stays on one SM: the forward kernel takes its features through all
// three layers in shared memory and registers, the backward kernel its output
// gradient through both input gradients and all weight gradients.  Only the
// activations that training needs go to memory.  Blocks are persistent; a
// block's weight gradients stay in registers over its bricks and are summed
// over the blocks, in block order, at the end: a training step is
// deterministic.  Every value that is rounded to BF16 comes from the same
// products in the same order in both kernels and whatever the block count.
//
// Brick layout everywhere: voxel (x*8 + y)*8 + z, channels innermost.  In
// shared memory 16 channels are two planes of 8 (16 bytes a voxel), so that the
// eight rows of an ldmatrix tile, eight voxels in z, are 128 consecutive
// bytes.
#include <cuda_bf16.h>

#include <algorithm>

#include "mrf_internal.h"

namespace mrf {
namespace net {

constexpr int kHaloVox = 1000;  // (8 + 2)^3
constexpr int kC0 = 4, kC1 = 16, kC2 = 16, kC3 = 1;
// parameter vector (fp32): W1[27][4][16] b1[16] W2[27][16][16] b2[16] W3[27][16][1] b3[1]
constexpr int oW1 = 0;
constexpr int oB1 = oW1 + 27 * kC0 * kC1;
constexpr int oW2 = oB1 + kC1;
constexpr int oB2 = oW2 + 27 * kC1 * kC2;
constexpr int oW3 = oB2 + kC2;
constexpr int oB3 = oW3 + 27 * kC2 * kC3;
constexpr int kNParams = oB3 + kC3;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void add4(float (&s)[4], const float (&x)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) s[r] += x[r];
}

// four 8x8 BF16 matrices; lane l gives row l % 8 of matrix l / 8
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}
__device__ __forceinline__ uint32_t pack2f(float lo, float hi) {
  return pack2(__float2bfloat16_rn(lo), __float2bfloat16_rn(hi));
}
__device__ __forceinline__ float lo_f(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi_f(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

// A voxel's four features, as one load where the array starts on 16 bytes
// (vec); any float array is taken, a view into a tensor may start anywhere.
__device__ __forceinline__ bool vec_ok(const float* feat) { return (reinterpret_cast<uintptr_t>(feat) & 15u) == 0; }
__device__ __forceinline__ float4 load_feat(const float* __restrict__ feat, int64_t v, bool vec) {
  if (vec) return reinterpret_cast<const float4*>(feat)[v];
  const float* f = feat + 4 * v;
  return make_float4(f[0], f[1], f[2], f[3]);
}

// halo position of voxel v's window origin; tap offsets inside the window
__device__ __forceinline__ int halo_base(int v) { return ((v >> 6) * 10 + ((v >> 3) & 7)) * 10 + (v & 7); }
__host__ __device__ constexpr int tap_off(int tap) { return ((tap / 9) * 10 + (tap / 3) % 3) * 10 + tap % 3; }
constexpr int kCentre = tap_off(13);  // of the voxel itself
__device__ __forceinline__ int halo_of(int v) { return halo_base(v) + kCentre; }

// the B fragment of K-step ks for the warp's lane: rows ks * 16 + 2t, +1 and
// + 8, + 9 of columns j * 8 + g (n-tile j), w(k, n) the matrix
template <typename F>
__device__ __forceinline__ uint2 b_frag(int ks, int j, int lane, F w) {
  const int g = lane >> 2, t = lane & 3, k = ks * 16 + 2 * t, n = j * 8 + g;
  return make_uint2(pack2f(w(k, n), w(k + 1, n)), pack2f(w(k + 8, n), w(k + 9, n)));
}
// both n-tiles of 16 columns, for every step, into dst[ks * 32 + lane]
template <typename F>
__device__ __forceinline__ void stage_frags(uint4* dst, int steps, int threads, F w) {
  for (int i = threadIdx.x; i < steps * 32; i += threads) {
    const uint2 a = b_frag(i >> 5, 0, i & 31, w), b = b_frag(i >> 5, 1, i & 31, w);
    dst[i] = make_uint4(a.x, a.y, b.x, b.y);
  }
}

// One 16-channel convolution of the warp's kTiles tiles of 16 voxels (from
// tile0 on) over all taps: rows from two halo planes at src, fragments wf.
template <int kTiles>
__device__ __forceinline__ void conv16(float (&acc)[kTiles][2][4], const uint4* src, const uint4* wf, int tile0,
                                       int lane) {
  uint32_t at[kTiles];
#pragma unroll
  for (int i = 0; i < kTiles; ++i) {
    const int v = (tile0 + i) * 16 + (lane & 15);
    at[i] = saddr(src + (lane >> 4) * kHaloVox + halo_base(v));
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0f;
  }
#pragma unroll 9
  for (int tap = 0; tap < 27; ++tap) {
    const uint4 b = wf[tap * 32 + lane];
#pragma unroll
    for (int i = 0; i < kTiles; ++i) {
      uint32_t a[4];
      ldm4(a, at[i] + 16u * (uint32_t)tap_off(tap));
      mma_bf16(acc[i][0], a, b.x, b.y);
      mma_bf16(acc[i][1], a, b.z, b.w);
    }
  }
}

// ---- forward ----------------------------------------------------------------
// 8 warps, four tiles of 16 voxels each.  Prediction (kTrain false): the second
// layer's accumulators are, packed, the A fragments of the third layer taken
// as one product with all 27 taps as columns, P[voxel][tap]; a voxel's output
// is the sum of 27 of its neighbours' entries (128 mma a brick instead of 864
// with one column in use).  Training: the activations go to memory, and the
// third layer runs tap by tap like the others, because its output's gradient
// is rounded to BF16 next; the loss's gradient and per-brick sum come with it.
//
// 18432 bricks: 2.15 ms as three kernels (80 TFLOP/s of the network's
// operations; intermediate activations through memory, fragments in single
// 4-byte loads, weights staged again for every brick), 0.50 so (343 TFLOP/s):
// two blocks of 113 KB an SM, bound by mma.sync and the barriers between the
// layers.
constexpr int kFwdThreads = 256;
constexpr int kPStride = 516;  // P by tap: the lanes' 8 voxels x 4 columns in different banks

struct FwdShared {
  uint4 w2[27 * 32];
  uint4 w1[7 * 32];
  uint4 a1[2 * kHaloVox];
  uint2 f[kHaloVox];
  union {
    float p[27 * kPStride];
    struct {
      uint4 a2[2 * kHaloVox];
      uint2 w3[27 * 32];
      float red[kFwdThreads / 32];
    } t;
  };
};

template <bool kTrain>
__global__ void __launch_bounds__(kFwdThreads, 2)
    k_forward(const float* __restrict__ W, const float* __restrict__ feat, int nb, float* __restrict__ out,
              __nv_bfloat16* __restrict__ g_a1, __nv_bfloat16* __restrict__ g_a2,
              const float* __restrict__ target, const float* __restrict__ weight, float inv_norm,
              float* __restrict__ lpart) {
  extern __shared__ __align__(16) unsigned char raw[];
  FwdShared& sh = *reinterpret_cast<FwdShared*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  stage_frags(sh.w1, 7, kFwdThreads, [&](int k, int n) { return k < 27 * kC0 ? W[oW1 + k * kC1 + n] : 0.0f; });
  stage_frags(sh.w2, 27, kFwdThreads, [&](int k, int n) { return W[oW2 + k * kC2 + n]; });
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < 2 * kHaloVox; i += kFwdThreads) {
    sh.a1[i] = zero4;
    if (kTrain) sh.t.a2[i] = zero4;
    if (i < kHaloVox) sh.f[i] = make_uint2(0u, 0u);
  }
  if (kTrain)
    for (int i = tid; i < 27 * 32; i += kFwdThreads)
      sh.t.w3[i] = b_frag(i >> 5, 0, i & 31, [&](int k, int n) { return n == 0 ? W[oW3 + k] : 0.0f; });
  // third layer's fragments with the taps as columns; biases of the lane's columns
  uint2 w3[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    w3[j] = b_frag(0, j, lane, [&](int k, int n) { return !kTrain && n < 27 ? W[oW3 + n * kC2 + k] : 0.0f; });
  float b1[2][2], b2[2][2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      b1[j][e] = W[oB1 + j * 8 + 2 * t + e];
      b2[j][e] = W[oB2 + j * 8 + 2 * t + e];
    }
  const float b3 = W[oB3];
  const bool vec = vec_ok(feat);
  float4 f0 = make_float4(0, 0, 0, 0), f1 = f0;
  if (blockIdx.x < nb) {
    f0 = load_feat(feat, (int64_t)blockIdx.x * 512 + tid, vec);
    f1 = load_feat(feat, (int64_t)blockIdx.x * 512 + tid + 256, vec);
  }
  __syncthreads();  // the halos are zero
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    sh.f[halo_of(tid)] = make_uint2(pack2f(f0.x, f0.y), pack2f(f0.z, f0.w));
    sh.f[halo_of(tid + 256)] = make_uint2(pack2f(f1.x, f1.y), pack2f(f1.z, f1.w));
    __syncthreads();
    if (b + gridDim.x < nb) {  // the next brick's features, while this one runs
      f0 = load_feat(feat, (b + gridDim.x) * 512 + tid, vec);
      f1 = load_feat(feat, (b + gridDim.x) * 512 + tid + 256, vec);
    }
    float acc[4][2][4];
    // layer 1: k = tap * 4 + channel; a lane's words: taps 4 ks + t / 2 and + 2
    {
      const uint32_t* word[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = (warp * 4 + i) * 16 + g;
        word[i][0] = reinterpret_cast<const uint32_t*>(sh.f + halo_base(v)) + (t & 1);
        word[i][1] = reinterpret_cast<const uint32_t*>(sh.f + halo_base(v + 8)) + (t & 1);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0f;
      }
#pragma unroll
      for (int ks = 0; ks < 7; ++ks) {
        const uint4 bw = sh.w1[ks * 32 + lane];
        const int oa = 2 * (t < 2 ? tap_off(4 * ks) : tap_off(4 * ks + 1));
        const bool last = ks == 6 && t >= 2;  // tap 27: none
        const int ob = 2 * (t < 2 ? tap_off(4 * ks + 2) : (ks == 6 ? 0 : tap_off(4 * ks + 3)));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t a[4] = {word[i][0][oa], word[i][1][oa], last ? 0u : word[i][0][ob], last ? 0u : word[i][1][ob]};
          mma_bf16(acc[i][0], a, bw.x, bw.y);
          mma_bf16(acc[i][1], a, bw.z, bw.w);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int v = (warp * 4 + i) * 16 + g + 8 * h;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t y = pack2f(fmaxf(acc[i][j][2 * h] + b1[j][0], 0.0f), fmaxf(acc[i][j][2 * h + 1] + b1[j][1], 0.0f));
          reinterpret_cast<uint32_t*>(sh.a1 + j * kHaloVox + halo_of(v))[t] = y;
          if (kTrain) reinterpret_cast<uint32_t*>(g_a1)[(b * 512 + v) * 8 + j * 4 + t] = y;
        }
      }
    __syncthreads();
    conv16<4>(acc, sh.a1, sh.w2, warp * 4, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t a[4];  // (row g, n-tile 0), (g + 8, 0), (g, 1), (g + 8, 1)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          a[2 * j + h] = pack2f(fmaxf(acc[i][j][2 * h] + b2[j][0], 0.0f), fmaxf(acc[i][j][2 * h + 1] + b2[j][1], 0.0f));
      const int v = (warp * 4 + i) * 16 + g;
      if (kTrain) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            reinterpret_cast<uint32_t*>(sh.t.a2 + j * kHaloVox + halo_of(v + 8 * h))[t] = a[2 * j + h];
            reinterpret_cast<uint32_t*>(g_a2)[(b * 512 + v + 8 * h) * 8 + j * 4 + t] = a[2 * j + h];
          }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float p[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          mma_bf16(p, a, w3[j].x, w3[j].y);
          const int n = j * 8 + 2 * t;
          if (n < 27) {
            sh.p[n * kPStride + v] = p[0];
            sh.p[n * kPStride + v + 8] = p[2];
          }
          if (n + 1 < 27) {
            sh.p[(n + 1) * kPStride + v] = p[1];
            sh.p[(n + 1) * kPStride + v + 8] = p[3];
          }
        }
      }
    }
    __syncthreads();
    if (!kTrain) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int v = tid + 256 * h;
        const int x = v >> 6, y = (v >> 3) & 7, z = v & 7;
        float sum = 0.0f;
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          if (x + dx < 1 || x + dx > 8) continue;
#pragma unroll
          for (int dy = 0; dy < 3; ++dy) {
            if (y + dy < 1 || y + dy > 8) continue;
            const float* p = sh.p + (dx * 9 + dy * 3) * kPStride + v + (dx - 1) * 64 + (dy - 1) * 8;
            if (z > 0) sum += p[-1];
            sum += p[kPStride];
            if (z < 7) sum += p[2 * kPStride + 1];
          }
        }
        out[b * 512 + v] = sum + b3;
      }
    } else {
      float y[4][4];
      uint32_t at[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        at[i] = saddr(sh.t.a2 + (lane >> 4) * kHaloVox + halo_base((warp * 4 + i) * 16 + (lane & 15)));
#pragma unroll
        for (int r = 0; r < 4; ++r) y[i][r] = 0.0f;
      }
#pragma unroll 9
      for (int tap = 0; tap < 27; ++tap) {
        const uint2 bw = sh.t.w3[tap * 32 + lane];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t a[4];
          ldm4(a, at[i] + 16u * (uint32_t)tap_off(tap));
          mma_bf16(y[i], a, bw.x, bw.y);
        }
      }
      // masked squared error on log-odds: dy = 2 w (y - t) / norm
      float s = 0.0f;
      if (t == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int64_t v = b * 512 + (warp * 4 + i) * 16 + g + 8 * h;
            const float e = (y[i][2 * h] + b3) - target[v], wv = weight[v];
            out[v] = 2.0f * wv * e * inv_norm;
            s += wv * e * e;
          }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
      if (lane == 0) sh.t.red[warp] = s;
      __syncthreads();
      if (tid == 0) {
        float tot = 0.0f;
        for (int k = 0; k < kFwdThreads / 32; ++k) tot += sh.t.red[k];
        lpart[b] = tot;
      }
    }
  }
}

// ---- backward ---------------------------------------------------------------
// 16 warps, two tiles of 16 voxels each.  From the output gradient dy and the
// stored activations of a brick: dZ2 = (dy * W3) masked by a2 > 0 and
// dZ1 = (dZ2 * W2) masked by a1 > 0 (the convolutions with flipped taps), and
// the weight gradients, sums over voxels of window values times gradients:
//   layer 2, layer 1: rows (tap, channel), columns the 16 gradients
//   layer 3: rows the 16 channels of a2, columns the 27 taps, the gradient
//            read at the tap's opposite offset (128 mma a brick instead of 864
//            with one column in use)
// Operands are the planes that the convolutions read, through transposing
// ldmatrix.  A training step on 512 bricks took 455 us as 17 kernels: weight
// gradients of every brick through memory and a thread per weight over all
// bricks 170, the loss's sum in one thread 44, operand staging most of the
// rest.  Now 97: 33 forward, 52 here, 10 to sum the blocks.
constexpr int kBwdThreads = 512;
constexpr int kSide = 2 * 27 * kC0 * kC1 + kC1 + kC2 + 4 * 27 * kC2 + 1;  // a block's partials but W2's
constexpr int kSideStride = (kSide + 63) / 64 * 64;
constexpr int sW1 = 0, sB1 = 2 * 27 * kC0 * kC1, sB2 = sB1 + kC1, sW3 = sB2 + kC2, sB3 = sW3 + 4 * 27 * kC2;

struct BwdShared {
  uint4 w2[27 * 32];
  uint4 w3[4 * 32];
  uint4 a1[2 * kHaloVox];
  uint4 dz2[2 * kHaloVox];
  uint4 a2[2 * 512];
  uint4 dz1[2 * 512];
  uint2 f[kHaloVox];
  uint32_t dy[kHaloVox];  // (dy, 0): the input gradient's convolution has two channels a tap
  float red[kBwdThreads / 32][2][kC1];
  float red3[kBwdThreads / 32];
};

__global__ void __launch_bounds__(kBwdThreads, 1)
    k_backward(const float* __restrict__ W, const float* __restrict__ feat, const __nv_bfloat16* __restrict__ g_a1,
               const __nv_bfloat16* __restrict__ g_a2, const float* __restrict__ g_dy, int nb,
               float* __restrict__ part2, float* __restrict__ side) {
  extern __shared__ __align__(16) unsigned char raw[];
  BwdShared& sh = *reinterpret_cast<BwdShared*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  stage_frags(sh.w2, 27, kBwdThreads,
              [&](int k, int n) { return W[oW2 + ((26 - k / kC2) * kC1 + n) * kC2 + k % kC2]; });
  stage_frags(sh.w3, 4, kBwdThreads,
              [&](int k, int n) { return k < 54 && k % 2 == 0 ? W[oW3 + (26 - k / 2) * kC2 + n] : 0.0f; });
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < 2 * kHaloVox; i += kBwdThreads) {
    sh.a1[i] = zero4;
    sh.dz2[i] = zero4;
    if (i < kHaloVox) {
      sh.f[i] = make_uint2(0u, 0u);
      sh.dy[i] = 0u;
    }
  }
  // weight gradients of the warp: layer 2's taps warp and warp + 16; layer 1's
  // row tile warp % 7 over half warp / 7 of the voxels (14 warps); layer 3's
  // taps 8 (warp % 4) .. + 7 over quarter warp / 4.  The tensor cores add a
  // product to the accumulator by truncation: a brick's 8 to 32 steps lose
  // 1e-6, a whole block's thousands 2e-4 (18432 bricks, 122 a block).  So a
  // brick's accumulators start at zero and are added to these, rounded.
  float g2[2][2][4] = {}, g1[2][4] = {}, g3[4] = {};
  float db1[2][2] = {}, db2[2][2] = {}, db3 = 0.0f;
  const bool vec = vec_ok(feat);
  for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
    __syncthreads();  // the previous brick's readers
    {
      const int v = tid, h = halo_of(v);
      const uint4* p1 = reinterpret_cast<const uint4*>(g_a1) + (b * 512 + v) * 2;
      const uint4* p2 = reinterpret_cast<const uint4*>(g_a2) + (b * 512 + v) * 2;
      const float4 f = load_feat(feat, b * 512 + v, vec);
      const __nv_bfloat16 dy = __float2bfloat16_rn(g_dy[b * 512 + v]);
      sh.a1[h] = p1[0];
      sh.a1[kHaloVox + h] = p1[1];
      sh.a2[v] = p2[0];
      sh.a2[512 + v] = p2[1];
      sh.f[h] = make_uint2(pack2f(f.x, f.y), pack2f(f.z, f.w));
      sh.dy[h] = __bfloat16_as_ushort(dy);
      db3 += __bfloat162float(dy);
    }
    __syncthreads();
    float acc[2][2][4];
    // the masked gradient of one tile's voxel and column pair, and its bias sum
    auto masked = [&](const float* y, uint32_t act, float (&db)[2]) {
      const float y0 = lo_f(act) > 0.0f ? y[0] : 0.0f, y1 = hi_f(act) > 0.0f ? y[1] : 0.0f;
      const uint32_t r = pack2f(y0, y1);
      db[0] += lo_f(r);
      db[1] += hi_f(r);
      return r;
    };
    // dZ2: k = tap * 2 (+ 1: zero); a lane's words: taps 8 ks + t and + 4
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int v = (warp * 2 + i) * 16 + g;
      const uint32_t* w0 = sh.dy + halo_base(v);
      const uint32_t* w1 = sh.dy + halo_base(v + 8);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0f;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint4 bw = sh.w3[ks * 32 + lane];
        const int ta = 8 * ks + t, tb = ta + 4;
        const int oa = ta < 27 ? tap_off(ta) : 0, ob = tb < 27 ? tap_off(tb) : 0;
        uint32_t a[4] = {ta < 27 ? w0[oa] : 0u, ta < 27 ? w1[oa] : 0u, tb < 27 ? w0[ob] : 0u, tb < 27 ? w1[ob] : 0u};
        mma_bf16(acc[i][0], a, bw.x, bw.y);
        mma_bf16(acc[i][1], a, bw.z, bw.w);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int u = v + 8 * h;
          const uint32_t act = reinterpret_cast<const uint32_t*>(sh.a2 + j * 512 + u)[t];
          reinterpret_cast<uint32_t*>(sh.dz2 + j * kHaloVox + halo_of(u))[t] = masked(acc[i][j] + 2 * h, act, db2[j]);
        }
    }
    __syncthreads();
    // dZ1
    conv16<2>(acc, sh.dz2, sh.w2, warp * 2, lane);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int u = (warp * 2 + i) * 16 + g + 8 * h;
          const uint32_t act = reinterpret_cast<const uint32_t*>(sh.a1 + j * kHaloVox + halo_of(u))[t];
          reinterpret_cast<uint32_t*>(sh.dz1 + j * 512 + u)[t] = masked(acc[i][j] + 2 * h, act, db1[j]);
        }
    // layer 2's weights.  A (rows channels, columns voxels): voxels 0-7 then
    // 8-15 of plane 0 and 1; B (rows voxels, columns gradients) likewise
    {
      const int va = (lane & 7) + 8 * (lane >> 4), pa = (lane >> 3) & 1;
      const int vb = (lane & 7) + 8 * ((lane >> 3) & 1), pb = lane >> 4;
      const int n_taps = warp + 16 < 27 ? 2 : 1;
      const uint32_t o0 = 16u * (uint32_t)tap_off(warp), o1 = 16u * (uint32_t)tap_off(n_taps > 1 ? warp + 16 : warp);
      float d2[2][2][4] = {};
      for (int ks = 0; ks < 32; ++ks) {
        uint32_t a[4], bw[4];
        ldm4t(bw, saddr(sh.dz2 + pb * kHaloVox + halo_of(ks * 16 + vb)));
        const uint32_t at = saddr(sh.a1 + pa * kHaloVox + halo_base(ks * 16 + va));
        ldm4t(a, at + o0);
        mma_bf16(d2[0][0], a, bw[0], bw[1]);
        mma_bf16(d2[0][1], a, bw[2], bw[3]);
        if (n_taps > 1) {
          ldm4t(a, at + o1);
          mma_bf16(d2[1][0], a, bw[0], bw[1]);
          mma_bf16(d2[1][1], a, bw[2], bw[3]);
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) add4(g2[k][j], d2[k][j]);
      // layer 3's: the columns' taps at the opposite offset of dy
      float d3[4] = {};
      const int tap = (warp & 3) * 8 + g;
      const uint32_t* dyo = sh.dy + 2 * kCentre - (tap < 27 ? tap_off(tap) : 0);
      for (int ks = (warp >> 2) * 8; ks < (warp >> 2) * 8 + 8; ++ks) {
        uint32_t a[4];
        ldm4t(a, saddr(sh.a2 + pa * 512 + ks * 16 + va));
        const uint32_t* q = dyo + halo_base(ks * 16 + 2 * t);  // rows 2t, 2t + 1; the next y for + 8, + 9
        const uint32_t b0 = tap < 27 ? q[0] | (q[1] << 16) : 0u, b1 = tap < 27 ? q[10] | (q[11] << 16) : 0u;
        mma_bf16(d3, a, b0, b1);
      }
      add4(g3, d3);
    }
    __syncthreads();
    // layer 1's weights
    if (warp < 14) {
      const int mt = warp % 7, half = warp / 7;
      const int vb = (lane & 7) + 8 * ((lane >> 3) & 1), pb = lane >> 4;
      const __nv_bfloat16* x[2];
      bool ok[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = mt * 16 + g + 8 * h, tap = k / kC0;
        ok[h] = tap < 27;
        x[h] = reinterpret_cast<const __nv_bfloat16*>(sh.f + (ok[h] ? tap_off(tap) : 0)) + k % kC0;
      }
      float d1[2][4] = {};
      for (int ks = half * 16; ks < half * 16 + 16; ++ks) {
        uint32_t bw[4], a[4];
        ldm4t(bw, saddr(sh.dz1 + pb * 512 + ks * 16 + vb));
        const int q = kC0 * halo_base(ks * 16 + 2 * t);  // + 1: the next z, + 8: the next y
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          a[h] = ok[h] ? pack2(x[h][q], x[h][q + kC0]) : 0u;
          a[h + 2] = ok[h] ? pack2(x[h][q + 10 * kC0], x[h][q + 11 * kC0]) : 0u;
        }
        mma_bf16(d1[0], a, bw[0], bw[1]);
        mma_bf16(d1[1], a, bw[2], bw[3]);
      }
      add4(g1[0], d1[0]);
      add4(g1[1], d1[1]);
    }
  }
  // the block's sums
  float* p2 = part2 + (int64_t)blockIdx.x * (27 * kC1 * kC2);
  float* ps = side + (int64_t)blockIdx.x * kSideStride;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int tap = warp + 16 * k;
    if (tap >= 27) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) p2[(tap * kC1 + g + 8 * (r >> 1)) * kC2 + j * 8 + 2 * t + (r & 1)] = g2[k][j][r];
  }
  if (warp < 14) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int k = (warp % 7) * 16 + g + 8 * (r >> 1);
        if (k < 27 * kC0) ps[sW1 + ((warp / 7) * 27 * kC0 + k) * kC1 + j * 8 + 2 * t + (r & 1)] = g1[j][r];
      }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int tap = (warp & 3) * 8 + 2 * t + (r & 1), c = g + 8 * (r >> 1);
    if (tap < 27) ps[sW3 + ((warp >> 2) * 27 + tap) * kC2 + c] = g3[r];
  }
  // bias sums: over the lanes of a column, then the warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) db3 += __shfl_xor_sync(0xFFFFFFFFu, db3, o);
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int o = 16; o >= 4; o >>= 1) {
        db1[j][e] += __shfl_xor_sync(0xFFFFFFFFu, db1[j][e], o);
        db2[j][e] += __shfl_xor_sync(0xFFFFFFFFu, db2[j][e], o);
      }
  if (g == 0) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sh.red[warp][0][j * 8 + 2 * t + e] = db1[j][e];
        sh.red[warp][1][j * 8 + 2 * t + e] = db2[j][e];
      }
  }
  if (lane == 0) sh.red3[warp] = db3;
  __syncthreads();
  if (tid < 2 * kC1) {
    float s = 0.0f;
    for (int w = 0; w < kBwdThreads / 32; ++w) s += sh.red[w][tid / kC1][tid % kC1];
    ps[(tid < kC1 ? sB1 : sB2) + tid % kC1] = s;
  }
  if (tid == 64) {
    float s = 0.0f;
    for (int w = 0; w < kBwdThreads / 32; ++w) s += sh.red3[w];
    ps[sB3] = s;
  }
}

// gradients summed over the blocks (in block order within each of eight
// slices, then the slices), 32 parameters a block; the last block sums the
// loss in FP64
constexpr int kReduceThreads = 256;
__global__ void __launch_bounds__(kReduceThreads)
    k_reduce(const float* __restrict__ part2, const float* __restrict__ side, int blocks,
             const float* __restrict__ lpart, int64_t nb, float inv_norm, float* __restrict__ grad,
             float* __restrict__ loss) {
  __shared__ float red[8][33];
  __shared__ double dred[kReduceThreads];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  if (blockIdx.x == gridDim.x - 1) {
    double s = 0.0;
    for (int64_t b = threadIdx.x; b < nb; b += kReduceThreads) s += lpart[b];
    dred[threadIdx.x] = s;
    __syncthreads();
    for (int o = kReduceThreads / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) dred[threadIdx.x] += dred[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss = (float)(dred[0] * inv_norm);
    return;
  }
  const int i = blockIdx.x * 32 + lane;
  // the parameter's place among a block's partials, the block stride, and the
  // parts it came in
  const float* p = side;
  int64_t stride = kSideStride, step = 0;
  int parts = 1;
  if (i < oB1) {
    p += sW1 + i;
    parts = 2;
    step = 27 * kC0 * kC1;
  } else if (i < oW2) {
    p += sB1 + (i - oB1);
  } else if (i < oB2) {
    p = part2 + (i - oW2);
    stride = 27 * kC1 * kC2;
  } else if (i < oW3) {
    p += sB2 + (i - oB2);
  } else if (i < oB3) {
    p += sW3 + (i - oW3);
    parts = 4;
    step = 27 * kC2;
  } else {
    p += sB3;
  }
  float s = 0.0f;
  if (i < kNParams)
    for (int k = 0; k < parts; ++k) {
      // eight loads in flight: one at a time, the 152 blocks' rows took 20 us
      int b = slice;
      for (; b + 56 < blocks; b += 64) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = p[(b + 8 * u) * stride + k * step];
#pragma unroll
        for (int u = 0; u < 8; ++u) s += x[u];
      }
      for (; b < blocks; b += 8) s += p[b * stride + k * step];
    }
  red[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && i < kNParams) {
    for (int k = 1; k < 8; ++k) s += red[k][lane];
    grad[i] = s;
  }
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, int n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.0f - b1) * gi;
  const float v = b2 * m2[i] + (1.0f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = v;
  p[i] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}

// The workspace: activations, the output gradient, the blocks' partial sums
// (layer 2's in part; the others in side, two activations' room per brick, of
// which a block of at least one brick needs kSideStride floats) and the loss
// per brick.  It may start at any float: the base is rounded up to the 16
// bytes that the activations' loads want, into the room at the end.
struct Work {
  __nv_bfloat16 *a1, *a2;
  float *side, *dy, *part, *lpart;
};
static_assert(kSideStride * 4 <= 2 * 512 * kC1 * 2, "a block's partials fit a brick's room");

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

inline size_t work_bytes(int64_t nb, Work* w, char* base) {
  base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(base) + 15) & ~(uintptr_t)15);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  const size_t vox = (size_t)nb * 512;
  char* a1 = take(vox * kC1 * 2);
  char* a2 = take(vox * kC2 * 2);
  char* side = take(vox * kC2 * 2);
  take(vox * kC1 * 2);
  char* dy = take(vox * 4);
  char* part = take((size_t)nb * 27 * kC1 * kC2 * 4);
  char* lpart = take((size_t)nb * 4);
  take(vox * 4);
  take((size_t)nb * kC1 * 4);
  if (w) {
    w->a1 = reinterpret_cast<__nv_bfloat16*>(a1);
    w->a2 = reinterpret_cast<__nv_bfloat16*>(a2);
    w->side = reinterpret_cast<float*>(side);
    w->dy = reinterpret_cast<float*>(dy);
    w->part = reinterpret_cast<float*>(part);
    w->lpart = reinterpret_cast<float*>(lpart);
  }
  return off;
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  return n < 1 ? 1 : n;
}

// more than 48 KiB of shared memory is asked for per device
template <typename K>
cudaError_t allow_shared(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t forward(const float* P, const float* feat, int64_t nb, float* out, cudaStream_t s) {
  cudaError_t e = allow_shared(k_forward<false>, sizeof(FwdShared));
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)std::min<int64_t>(nb, 2 * sm_count());
  k_forward<false><<<grid, kFwdThreads, sizeof(FwdShared), s>>>(P, feat, (int)nb, out, nullptr, nullptr, nullptr,
                                                                nullptr, 0.0f, nullptr);
  return cudaGetLastError();
}

cudaError_t gradients(const float* P, const float* feat, const float* target, const float* wt, int64_t nb,
                      float inv_norm, float* grad, float* loss, const Work& w, cudaStream_t s) {
  cudaError_t e = allow_shared(k_forward<true>, sizeof(FwdShared));
  if (e == cudaSuccess) e = allow_shared(k_backward, sizeof(BwdShared));
  if (e != cudaSuccess) return e;
  const int sms = sm_count();
  const unsigned fgrid = (unsigned)std::min<int64_t>(nb, 2 * sms), bgrid = (unsigned)std::min<int64_t>(nb, sms);
  k_forward<true><<<fgrid, kFwdThreads, sizeof(FwdShared), s>>>(P, feat, (int)nb, w.dy, w.a1, w.a2, target, wt,
                                                                inv_norm, w.lpart);
  k_backward<<<bgrid, kBwdThreads, sizeof(BwdShared), s>>>(P, feat, w.a1, w.a2, w.dy, (int)nb, w.part, w.side);
  k_reduce<<<(kNParams + 31) / 32 + 1, kReduceThreads, 0, s>>>(w.part, w.side, (int)bgrid, w.lpart, nb, inv_norm, grad,
                                                               loss);
  return cudaGetLastError();
}

}  // namespace net
}  // namespace mrf

using namespace mrf;

extern "C" {

int64_t mrf_net_num_params(void) { return net::kNParams; }

int64_t mrf_net_workspace_bytes(int64_t n_bricks) {
  if (n_bricks < 0) return -1;
  return (int64_t)net::work_bytes(n_bricks, nullptr, nullptr);
}

static mrf_status net_status(cudaError_t e) {
  if (e == cudaSuccess) return MRF_OK;
  mrf_internal_set_error(std::string("CUDA: ") + cudaGetErrorString(e));
  return MRF_ERR_CUDA;
}

static bool net_args_ok(const void* a, const void* b, const void* ws, int64_t nb) {
  if (!a || !b || !ws || nb < 1 || nb > 0x7FFFFFFF) {
    mrf_internal_set_error("invalid network arguments");
    return false;
  }
  return true;
}

mrf_status mrf_net_forward(const float* params, const float* feat, int64_t n_bricks, float* out,
                           void* workspace, void* stream) {
  if (!net_args_ok(params, feat, workspace, n_bricks) || !out) return MRF_ERR_INVALID;
  return net_status(net::forward(params, feat, n_bricks, out, static_cast<cudaStream_t>(stream)));
}

mrf_status mrf_net_gradients(const float* params, const float* feat, const float* target,
                             const float* weight, int64_t n_bricks, float norm, float* grads,
                             float* loss, void* workspace, void* stream) {
  if (!net_args_ok(params, feat, workspace, n_bricks) || !target || !weight || !grads || !loss ||
      !(norm > 0.0f))
    return MRF_ERR_INVALID;
  net::Work w;
  net::work_bytes(n_bricks, &w, static_cast<char*>(workspace));
  return net_status(net::gradients(params, feat, target, weight, n_bricks, 1.0f / norm, grads, loss, w,
                                   static_cast<cudaStream_t>(stream)));
}

mrf_status mrf_net_adam(float* params, const float* grads, float* m1, float* m2, int64_t n, float lr,
                        float beta1, float beta2, float eps, int step, void* stream) {
  if (!params || !grads || !m1 || !m2 || n < 1 || n > 0x7FFFFFFF || step < 1) {
    mrf_internal_set_error("invalid Adam arguments");
    return MRF_ERR_INVALID;
  }
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  net::k_adam<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params, grads, m1, m2, (int)n, lr, beta1, beta2, eps, c1, c2);
  return net_status(cudaGetLastError());
}

}  // extern "C"
