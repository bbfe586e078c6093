// mrf_build.cu -- per-keyframe work that runs once per brick-set change:
// depth clean-up, brick activation, the 3D-DDA traversal that emits each
// ray's incidence list, and the (camera, voxel) pair / CSR construction.
//
// Reference behaviour restated here (paths inside the MRFMap project):
//   depth clean-up            src/GVDBImage.cpp:32-40
//   endpoint back-projection  src/GVDBImage.cpp:48-56, src/GVDBCamera.cpp:70-100
//   activation radius 1       src/GVDBMRFMap.cpp:117-135
//   per-brick stop rules      src/cuda/gvdbkernels.cu:568, 816, 1035
//   infinity-term gate        src/cuda/gvdbkernels.cu:1196-1208
//   Pre-pass visibility reset src/cuda/gvdbkernels.cu:708-715
#include <algorithm>
#include <cub/cub.cuh>

#include "mrf_geometry.cuh"
#include "mrf_internal.h"

namespace mrf {

namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(int64_t n, int t = kThreads) {
  int64_t b = (n + t - 1) / t;
  return (unsigned)(b < 1 ? 1 : b);
}

__global__ void k_clean_depth(const float* __restrict__ in, float* __restrict__ out, int rows,
                              int cols) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * cols) return;
  out[i] = clean_depth_value(in[i], i, rows, cols);
}

__device__ __forceinline__ int floordiv8(int v) { return v >= 0 ? v / 8 : -((-v + 7) / 8); }

__device__ __forceinline__ void mark_point(const Geom& g, float px, float py, float pz,
                                           uint8_t* flags) {
  int lo[3], hi[3];
  float pv[3] = {px, py, pz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    int vi = (int)floorf(pv[a]);
    lo[a] = max(floordiv8(vi - 1), g.blo[a] / kBrick);
    hi[a] = min(floordiv8(vi + 1), g.bhi[a] / kBrick - 1);
  }
  for (int bx = lo[0]; bx <= hi[0]; ++bx)
    for (int by = lo[1]; by <= hi[1]; ++by)
      for (int bz = lo[2]; bz <= hi[2]; ++bz)
        flags[((int64_t)bx * g.NB[1] + by) * g.NB[2] + bz] = 1;
}

__global__ void k_activate(Geom g, Pose P, const float* __restrict__ depth, int policy,
                           uint8_t* __restrict__ flags) {
  const int pix = tile_pixel(g.rows, g.cols, (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, threadIdx.x & 31);
  if (pix < 0) return;
  float d = depth[pix];
  if (!(d > 0.0f)) return;
  int x = pix % g.cols, y = pix / g.cols;
  // back-projection with fx on both axes and integer pixel coordinates
  float f = fd(d, g.fx);
  float X = fm(f, fs((float)x, g.cx));
  float Y = fm(f, fs((float)y, g.cy));
  float pv[3];
  bool inside = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float pw = fa(fa(fa(fm(P.m[a * 4 + 0], X), fm(P.m[a * 4 + 1], Y)), fm(P.m[a * 4 + 2], d)),
                  P.m[a * 4 + 3]);
    pv[a] = fa(fm(pw, g.inv_res), g.off[a]);
    if (!(pv[a] >= g.glo[a] && pv[a] < g.hi[a])) inside = false;
  }
  if (inside) mark_point(g, pv[0], pv[1], pv[2], flags);
  if (policy == 1) {
    // every brick the ray crosses up to the brick run where the Pre pass
    // stops (the trace's test: at the exit s of a run's last voxel,
    // s + bias(s) > d + 3 sigma(s)).  The trace then meets only bricks its
    // own view activated before its stop, so bricks other views activate
    // later never change this view's lists.
    const Sensor c = sensor_at(g, x, y);
    Ray ray;
    ray_setup(g, P, x, y, ray);
    Dda r;
    if (dda_init(r, g, ray)) {
      float s_last = 0.0f;
      for (bool first = true; r.alive && r.guard > 0; first = false) {
        if (!first && fa(s_last, c.bias(s_last)) > fa(d, fm(3.0f, c.sigma(s_last)))) break;
        flags[r.lin] = 1;
        int steps;
        s_last = fm(dda_cross(r, g, ray, steps), ray.mult);
      }
    }
  }
}

__global__ void k_activate_points(Geom g, const float* __restrict__ pts, int64_t n,
                                  uint8_t* __restrict__ flags) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  if (!(px >= 0.0f && py >= 0.0f && pz >= 0.0f && px < (float)g.E[0] && py < (float)g.E[1] &&
        pz < (float)g.E[2]))
    return;
  mark_point(g, px, py, pz, flags);
}

__global__ void k_new_indicator(const uint8_t* __restrict__ flags, const int* __restrict__ slot,
                                int* __restrict__ ind, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ind[i] = (flags[i] && slot[i] < 0) ? 1 : 0;
}

__global__ void k_assign_slots(Geom g, const int* __restrict__ ind, const int* __restrict__ scan,
                               int nb_base, int* __restrict__ slot, int* __restrict__ coord,
                               int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !ind[i]) return;
  int s = nb_base + scan[i];
  slot[i] = s;
  int bz = (int)(i % g.NB[2]);
  int by = (int)((i / g.NB[2]) % g.NB[1]);
  int bx = (int)(i / ((int64_t)g.NB[2] * g.NB[1]));
  coord[3 * s + 0] = bx;
  coord[3 * s + 1] = by;
  coord[3 * s + 2] = bz;
}

__global__ void k_fill_new_voxels(float* L, float* belief, int64_t v0, int64_t v1, float lp) {
  int64_t i = v0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v1) return;
  L[i] = lp;
  belief[i] = 0.0f;
}

// set_channel_kernel (gvdbkernels.cu:1040-1064): write occupancies of points
// (voxel units) into the belief field
__global__ void k_set_points(Geom g, const float* __restrict__ pts, const float* __restrict__ occ,
                             int64_t n, float* __restrict__ belief) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  if (!(px >= 0.0f && py >= 0.0f && pz >= 0.0f && px < (float)g.E[0] && py < (float)g.E[1] &&
        pz < (float)g.E[2]))
    return;
  int vx = (int)floorf(px), vy = (int)floorf(py), vz = (int)floorf(pz);
  int s = g.brick_slot[brick_lin(g, vx, vy, vz)];
  if (s < 0) return;
  belief[(int64_t)s * kBrickVox + voxel_local(vx, vy, vz)] = occ[i];
}

// the view of a block of a batch
__device__ __forceinline__ int batch_view(const TraceBatch& b) {
  int k = 0;
  while (k + 1 < b.n && blockIdx.x >= b.first[k + 1]) ++k;
  return k;
}
constexpr int kTraceThreads = 128;

// Incidences of each pixel's Pre pass, padded to a multiple of 4 (the emit
// pass's offsets): the voxels the ray crosses in active bricks up to the
// brick run whose end is past the return, counted brick by brick.
__global__ void __launch_bounds__(kTraceThreads)
    k_trace_count(const __grid_constant__ TraceBatch batch, int* __restrict__ err) {
  const TraceView& w = batch.v[batch_view(batch)];
  const Geom& g = w.g;
  const int64_t block = blockIdx.x - batch.first[batch_view(batch)];
  const int pix = tile_pixel(g.rows, g.cols, (block * kTraceThreads + threadIdx.x) >> 5, threadIdx.x & 31);
  int count = 0;
  const float d = pix < 0 ? 0.0f : w.depth[pix];
  if (d > 0.0f) {
    const int x = pix % g.cols, y = pix / g.cols;
    const Sensor c = sensor_at(g, x, y);
    Ray ray;
    ray_setup(g, w.P, x, y, ray);
    Dda r;
    if (dda_init(r, g, ray)) {
      while (r.alive && r.guard > 0) {
        const int slot = g.brick_slot[r.lin];
        int steps;
        const float s = fm(dda_cross(r, g, ray, steps), ray.mult);
        if (slot < 0) continue;
        if (count + steps > kMaxRayLen) {
          atomicOr(err, 1);
          count = kMaxRayLen;
          break;
        }
        count += steps;
        if (fa(s, c.bias(s)) > fa(d, fm(3.0f, c.sigma(s)))) break;
      }
    }
  }
  const uint32_t padded = (uint32_t)((count + 3) & ~3);
  if (pix >= 0) w.counts[pix] = padded;
  if (pix == 0) w.counts[g.rows * g.cols] = 0u;
  const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, padded);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(w.total, (unsigned long long)sum);
}

// One thread per pixel walks the DDA through the active bricks.  Runs of
// voxels in one brick end with the reference's per-brick stop tests.  A
// thread's last incidences wait in shared memory (its own column) and go out
// eight at a time, as two 16-byte stores per list: single incidences, or
// groups of four in registers, leave half-written sectors behind that L2
// reads and writes twice.  A ray's lists start on a multiple of four; the last
// group is completed with padding.  A list that does not fill the room its
// count gave it raises the error flag.
constexpr int kEmitStride = 12;  // words of a thread's eight in each list: 16-byte loads, four ways to a bank

__device__ __forceinline__ RayMeta emit_ray(const TraceView& w, int pix,
                                            uint32_t (&pending)[3][kTraceThreads * kEmitStride],
                                            uint8_t* __restrict__ loud, int* __restrict__ err) {
  const Geom& g = w.g;
  uint32_t* __restrict__ inc_vox = w.vox;
  float* __restrict__ inc_len = w.len;
  float* __restrict__ inc_mu = w.mu;
  const float d = w.depth[pix];
  int count = 0, n_pre = -1, n_post = -1, r0 = -1, run_start = 0, kmu = -1;
  bool gate = false;
  const uint32_t base = w.pix_off[pix] - w.pix_off[0];
  const int room = (int)(w.pix_off[pix + 1] - w.pix_off[0] - base);
  // the group of eight incidence k belongs to, counted in the arena so that
  // whole groups are whole sectors; the ray's first may be a half
  const uint32_t mine = threadIdx.x * kEmitStride;
  const uint32_t phase = (w.inc_base + base) & 7u;
  auto push = [&](uint32_t k, uint32_t v, float len, float mu) {
    const uint32_t a = mine + ((phase + k) & 7u);
    pending[0][a] = v;
    pending[1][a] = __float_as_uint(len);
    pending[2][a] = __float_as_uint(mu);
  };
  // half h of the group goes to incidences first .. first + 3
  auto store = [&](uint32_t first, uint32_t h) {
    const uint32_t a = mine + 4 * h;
    *reinterpret_cast<uint4*>(inc_vox + first) = *reinterpret_cast<const uint4*>(pending[0] + a);
    *reinterpret_cast<uint4*>(inc_len + first) = *reinterpret_cast<const uint4*>(pending[1] + a);
    *reinterpret_cast<uint4*>(inc_mu + first) = *reinterpret_cast<const uint4*>(pending[2] + a);
  };
  auto flush = [&](uint32_t k) {
    // k completes its group of eight: both halves, unless the ray began in
    // the second one
    const uint32_t end = base + k + 1;
    if (k + 1 >= 8) store(end - 8, 0);
    store(end - 4, 1);
  };
  if (d > 0.0f) {
    const int x = pix % g.cols, y = pix / g.cols;
    const Sensor c = sensor_at(g, x, y);
    Ray ray;
    ray_setup(g, w.P, x, y, ray);
    Dda r;
    if (dda_init(r, g, ray)) {
      bool run_open = false;
      float s_last = 0.0f;
      // no potential before it: 13.3 sigma' with room for rounding
      const float s_first = window_start(c, d, 40.0f, 0.999f);
      // the run that ends here: the stop tests
      auto stop = [&]() {
        const float lhs = fa(s_last, c.bias(s_last));
        const float rhs = fa(d, fm(3.0f, c.sigma(s_last)));
        if (n_post < 0 && lhs >= rhs) n_post = count;
        if (lhs > rhs) n_pre = count;
        return lhs > rhs;
      };
      while (r.alive && r.guard > 0) {
        if (run_open && stop()) break;
        run_open = false;
        const int slot = g.brick_slot[r.lin];
        if (slot < 0) {
          int steps;
          dda_cross(r, g, ray, steps);
          continue;
        }
        run_start = count;
        run_open = true;
        // the brick's voxels: neighbouring rays enter and leave it nearly
        // together, so the lanes that are done wait a step or two here
        // rather than entering their next brick on their own
        bool left;
        do {
          if (count >= room) {
            atomicOr(err, 2);
            r.alive = false;
            break;
          }
          const uint32_t v = (uint32_t)slot * kBrickVox + dda_local(r);
          float l, tin, te;
          left = dda_step(r, g, l, tin, te);
          s_last = fm(te, ray.mult);
          float mu = 0.0f;
          if (s_last >= s_first && !potential_is_zero(c, s_last, d)) {
            mu = potential(c, s_last, d);
            if (r0 < 0) r0 = run_start;
            if (kmu < 0) kmu = count;
          }
          push((uint32_t)count, v, l, mu);
          if (((phase + count) & 7) == 7) flush((uint32_t)count);
          // dynamic: in the Post range, from the first non-zero potential on
          if (kmu >= 0 && n_post < 0) loud[v] = 1;
          ++count;
        } while (!left && r.guard > 0);
      }
      if (n_pre < 0 && run_open) stop();
      if (n_pre < 0) {
        n_pre = count;
        if (count > 0) gate = d > fa(s_last, c.bias(s_last));
      }
    }
  }
  if (n_pre < 0) n_pre = count;
  if (n_post < 0) n_post = count;
  // the last group, completed with padding (invalid voxel, zeros; 16-byte
  // vector loads in the BP kernels)
  const int padded = (n_pre + 3) & ~3;
  for (int k = count; k < padded; ++k) push((uint32_t)k, kNoVoxel, 0.0f, 0.0f);
  const uint32_t left = padded ? (phase + (uint32_t)padded) & 7u : 0u;  // in the last, unfinished group of eight
  if (count < padded && left == 0) flush((uint32_t)padded - 1u);
  if (left == 4) store(base + (uint32_t)padded - 4u, 0);
  if (padded != room) atomicOr(err, 2);
  const int kdyn = (kmu >= 0 && kmu < n_post) ? kmu : n_post;
  RayMeta m;
  m.off = w.inc_base + base;
  m.n_pre = (uint16_t)n_pre;
  m.n_post = (uint16_t)n_post;
  m.r0 = (uint16_t)(r0 >= 0 ? r0 : n_pre);
  m.rinf = (uint16_t)(r0 >= 0 ? r0 : run_start);
  m.flags = (gate ? 1u : 0u) | ((uint32_t)kdyn << 16);
  w.meta[pix] = m;
  return m;
}

__global__ void __launch_bounds__(kTraceThreads, 6)
    k_trace_emit(const __grid_constant__ TraceBatch batch, uint8_t* __restrict__ loud, int* __restrict__ err) {
  __shared__ __align__(16) uint32_t pending[3][kTraceThreads * kEmitStride];
  const int vi = batch_view(batch);
  const TraceView& w = batch.v[vi];
  const Geom& g = w.g;
  const int64_t block = blockIdx.x - batch.first[vi];
  const int pix = tile_pixel(g.rows, g.cols, (block * kTraceThreads + threadIdx.x) >> 5, threadIdx.x & 31);
  RayMeta m = {};
  if (pix >= 0) m = emit_ray(w, pix, pending, loud, err);
  // the view's totals: a warp's in 32 bits (rays are shorter than 2^16)
  const bool bp = ray_in_bp(m);
  const uint32_t c[kRayCounters] = {m.n_pre,
                                    m.n_pre > 0 ? 1u : 0u,
                                    m.n_post,
                                    (uint32_t)(m.n_post - ray_kdyn(m)),
                                    bp ? 1u : 0u,
                                    bp ? m.n_pre : 0u,
                                    bp ? (uint32_t)(m.n_pre - (ray_kdyn(m) & ~3)) : 0u};
#pragma unroll
  for (int k = 0; k < kRayCounters; ++k) {
    const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, c[k]);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(w.counters + k, (unsigned long long)sum);
  }
}

// Pairs.  A pair is a (camera, voxel) with at least one incidence.  The pairs
// of a view are numbered brick-major by first visit: pairs on loud voxels
// (voxels with a dynamic incidence in some view) first, then the others; in
// each part the bricks in the order of their first incidence (pixel order,
// then along the ray) and a brick's pairs by their own first incidence.  Rays
// of neighbouring pixels cross the same bricks and voxels in the same order,
// so the pair ids met along a ray come in runs of nearby ids (the ray
// kernel's ln q gathers share sectors), while a brick's pairs stay together
// (the per-pair kernels' L accesses stay within the brick).
//
// The numbering needs no sort of the incidences: a table over the voxels
// holds each voxel's first incidence, the (few) bricks are sorted by theirs,
// a block orders the up to 512 voxels of a brick in shared memory, and the
// table then maps voxels to pairs.  Only the dynamic incidences, the ones the
// pair update visits, are grouped by pair (a stable radix sort of a sixth of
// the incidences).  View of 104 M incidences at 1 cm: 13.5 ms with sorts of
// all incidences by voxel and of all pairs by first visits.

// first[v]: lowest index of an incidence on voxel v.  Most visits come after
// the first one: a look at the table, stale in the SM's own cache at worst,
// saves the atomic (0.56 ms for a view of 104 M incidences; a look in L2 takes
// 0.92, near incidences through shared memory as below 0.56).
__global__ void k_first_visit(const uint32_t* __restrict__ vox, uint32_t n4, uint32_t* first) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n4) return;
  const uint4 u = reinterpret_cast<const uint4*>(vox)[t];
  const uint32_t v[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (v[j] != kNoVoxel && first[v[j]] > 4 * t + j) atomicMin(first + v[j], 4 * t + j);
}

// per brick: its first incidence (kNoVoxel: none), its loud voxels with an
// incidence and its other voxels with one.  A warp per brick.
__global__ void k_brick_count(uint32_t nb, const uint32_t* __restrict__ first, const uint8_t* __restrict__ loud,
                              uint32_t* __restrict__ bfirst, uint32_t* __restrict__ bloud,
                              uint32_t* __restrict__ bquiet) {
  const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (b >= nb) return;
  uint32_t nl = 0, nq = 0, lo = kNoVoxel;
  const size_t at = (size_t)b * (kBrickVox / 4);
#pragma unroll
  for (int k = 0; k < kBrickVox / 128; ++k) {
    const uint4 f = reinterpret_cast<const uint4*>(first)[at + k * 32 + lane];
    const uchar4 l = reinterpret_cast<const uchar4*>(loud)[at + k * 32 + lane];
    auto add = [&](uint32_t fv, uint8_t lv) {
      nl += fv != kNoVoxel && lv;
      nq += fv != kNoVoxel && !lv;
      lo = min(lo, fv);
    };
    add(f.x, l.x);
    add(f.y, l.y);
    add(f.z, l.z);
    add(f.w, l.w);
  }
  nl = __reduce_add_sync(0xFFFFFFFFu, nl);
  nq = __reduce_add_sync(0xFFFFFFFFu, nq);
  lo = __reduce_min_sync(0xFFFFFFFFu, lo);
  if (lane == 0) {
    bfirst[b] = lo;
    bloud[b] = nl;
    bquiet[b] = nq;
  }
}

// the counts in brick order: cnt[i] loud, cnt[nb + i] others, of brick order[i]
__global__ void k_order_counts(const uint32_t* __restrict__ order, uint32_t nb, const uint32_t* __restrict__ bloud,
                               const uint32_t* __restrict__ bquiet, uint32_t* __restrict__ cnt) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  cnt[i] = bloud[order[i]];
  cnt[nb + i] = bquiet[order[i]];
}

// Ascending bitonic sort of 512 keys of a warp, 16 per lane (element e = 16
// lane + r): steps within a lane are register compares, the 15 others one
// shuffle per key.
__device__ __forceinline__ void warp_sort512(uint32_t (&x)[16], int lane) {
#pragma unroll
  for (int k = 2; k <= kBrickVox; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 16) {
        const bool keep_min = ((lane & (j / 16)) == 0) == ((lane & (k / 16)) == 0);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x[r], j / 16);
          x[r] = keep_min ? min(x[r], y) : max(x[r], y);
        }
      } else {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          if (r & j) continue;
          const bool up = k < 16 ? (r & k) == 0 : (lane & (k / 16)) == 0;
          const uint32_t lo = min(x[r], x[r | j]), hi = max(x[r], x[r | j]);
          x[r] = up ? lo : hi;
          x[r | j] = up ? hi : lo;
        }
      }
    }
  }
}

// numbers of the i-th brick's pairs: its loud voxels from start[i] on, the
// others from start[nb + i] on (start: the exclusive scan of cnt), each part
// by first incidence.  Writes the pairs' voxels and turns the table's entries
// into the voxels' pair numbers.  A warp per brick sorts the first incidences;
// no two voxels share one, so vox gives each its voxel back.  (A block per
// brick sorting 64-bit keys in shared memory: 0.61 ms for a 1 cm view of 13 M
// pairs.)
__global__ void __launch_bounds__(kThreads)
    k_brick_number(const uint32_t* __restrict__ bkey, const uint32_t* __restrict__ order, uint32_t nb,
                   uint32_t* __restrict__ table, const uint8_t* __restrict__ loud, const uint32_t* __restrict__ vox,
                   const uint32_t* __restrict__ start, uint32_t pair_base, uint32_t* __restrict__ pair_vox) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= nb || bkey[i] == kNoVoxel) return;
  const uint4* src = reinterpret_cast<const uint4*>(table) + (size_t)order[i] * (kBrickVox / 4);
  uint32_t x[16];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint4 f = src[k * 32 + lane];
    x[4 * k + 0] = f.x;
    x[4 * k + 1] = f.y;
    x[4 * k + 2] = f.z;
    x[4 * k + 3] = f.w;
  }
  warp_sort512(x, lane);  // voxels without an incidence (kNoVoxel) last
  // loud voxels before each of the lane's, then every voxel's number
  unsigned is_loud = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (x[k] == kNoVoxel) continue;
    x[k] = vox[x[k]];
    if (loud[x[k]]) is_loud |= 1u << k;
  }
  uint32_t nl = __popc(is_loud);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, nl, o);
    if (lane >= o) nl += u;
  }
  nl -= __popc(is_loud);
  const uint32_t l0 = start[i], q0 = start[nb + i];
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (x[k] == kNoVoxel) continue;
    const uint32_t before = nl + __popc(is_loud & ((1u << k) - 1u));
    const uint32_t q = (is_loud >> k) & 1u ? l0 + before : q0 + (16 * lane + k - before);
    pair_vox[pair_base + q] = x[k];
    table[x[k]] = q;
  }
}

// Sums of segment lengths are carried as 64-bit integers in units of 2^-40
// voxel: exact for lengths of at least 2^-16 (the rest is below 2^-41 each),
// rounded once to FP32 at the end, and independent of the order of the
// atomics that form them (the reference adds with float atomics).  2^20 voxels
// of summed length, 3e5 rays through one voxel, stay below 2^61.
constexpr float kLenUnit = 1099511627776.0f;  // 2^40
__device__ __forceinline__ long long len_fixed(float l) { return __float2ll_rn(l * kLenUnit); }
__device__ __forceinline__ float len_float(long long s) { return __ll2float_rn(s) * (1.0f / kLenUnit); }

// every incidence's pair id; the static incidences' lengths summed per pair;
// the dynamic incidences (pair number, incidence index) listed in ray order
// at doff[r].
//
// All rays start at the camera: its voxel gets a length from every ray of the
// view, the ones around it from thousands, and their atomics serialise (1.9
// ms of a 1 cm view, 0.7 without the first 64 incidences of each ray).  A
// block takes kNearRays consecutive rays, which cross the same near voxels,
// and adds up the lengths of a ray's first kNear incidences in a shared hash
// table (four probes; a pair that finds no place goes straight to memory):
// the low 21 bits and the rest apart, in 32-bit sums that kNearRays additions
// of at most 2^41 cannot overflow.  0.67 ms; a small image (160x120) wants few
// rays a block: 0.05 ms with 64, 0.03 with 32.
constexpr int kRayLanes = 8;  // lanes per ray, four incidences each
constexpr int kNearThreads = 128;
constexpr int kNearRays = 32;
constexpr int kNear = 64;
constexpr uint32_t kNearSlots = 1024;
static_assert(kNearSlots == 1u << 10, "the hash keeps ten bits");

__global__ void __launch_bounds__(kNearThreads)
    k_assign_pairs(const RayMeta* __restrict__ meta, uint32_t npix, const uint32_t* __restrict__ vox,
                   const float* __restrict__ len, const uint32_t* __restrict__ table, uint32_t inc_base,
                   uint32_t pair_base, const uint32_t* __restrict__ doff, uint32_t* __restrict__ inc_pair,
                   unsigned long long* __restrict__ static_len, uint32_t* __restrict__ dkey,
                   uint32_t* __restrict__ dval) {
  __shared__ uint32_t skey[kNearSlots], slo[kNearSlots], shi[kNearSlots];
  for (uint32_t k = threadIdx.x; k < kNearSlots; k += kNearThreads) {
    skey[k] = kNoVoxel;
    slo[k] = 0u;
    shi[k] = 0u;
  }
  __syncthreads();
  const uint32_t r1 = min(npix, (blockIdx.x + 1) * kNearRays);
  for (uint32_t r = blockIdx.x * kNearRays + threadIdx.x / kRayLanes; r < r1; r += kNearThreads / kRayLanes) {
    const RayMeta me = meta[r];
    const int n = me.n_pre, np = me.n_post, kd = ray_kdyn(me);
    const uint32_t off = me.off - inc_base;
    const uint32_t d0 = doff[r] - (uint32_t)kd;
    for (int i = 4 * (threadIdx.x % kRayLanes); i < n; i += 4 * kRayLanes) {
      const uint4 u = *reinterpret_cast<const uint4*>(vox + off + i);
      const float4 lv = *reinterpret_cast<const float4*>(len + off + i);
      const uint32_t v[4] = {u.x, u.y, u.z, u.w};
      const float l[4] = {lv.x, lv.y, lv.z, lv.w};
      uint32_t q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = i + j < n ? table[v[j]] : 0u;
      *reinterpret_cast<uint4*>(inc_pair + off + i) =
          make_uint4(pair_base + q[0], pair_base + q[1], pair_base + q[2], pair_base + q[3]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i + j < kd) {
          const unsigned long long x = (unsigned long long)len_fixed(l[j]);
          bool added = false;
          if (i < kNear) {
            uint32_t h = (q[j] * 2654435761u) >> 22;
            for (int probe = 0; probe < 4 && !added; ++probe) {
              const uint32_t old = skey[h] == q[j] ? q[j] : atomicCAS(skey + h, kNoVoxel, q[j]);
              added = old == q[j] || old == kNoVoxel;
              if (!added) h = (h + 1) & (kNearSlots - 1);
            }
            if (added) {
              atomicAdd(slo + h, (uint32_t)x & 0x1FFFFFu);
              atomicAdd(shi + h, (uint32_t)(x >> 21));
            }
          }
          if (!added) atomicAdd(static_len + q[j], x);
        } else if (i + j < np) {
          dkey[d0 + i + j] = q[j];
          dval[d0 + i + j] = me.off + i + j;
        }
      }
    }
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < kNearSlots; k += kNearThreads)
    if (skey[k] != kNoVoxel)
      atomicAdd(static_len + skey[k], (unsigned long long)slo[k] + ((unsigned long long)shi[k] << 21));
}

// dynamic incidences of each ray
__global__ void k_dyn_counts(const RayMeta* __restrict__ meta, uint32_t npix, uint32_t* __restrict__ cnt) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < npix) cnt[r] = (uint32_t)(meta[r].n_post - ray_kdyn(meta[r]));
}

// *count += number of pairs on loud voxels
__global__ void k_count_loud(const uint32_t* __restrict__ pair_vox, uint32_t np,
                             const uint8_t* __restrict__ loud, uint32_t* __restrict__ count) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool l = p < np && loud[pair_vox[p]];
  const unsigned b = __ballot_sync(0xFFFFFFFFu, l);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(count, (uint32_t)__popc(b));
}

// Per pair: cumulative length, the sum of its static messages F_EPS * l, the
// number of dynamic incidences and the potential mass sum mu * l (a
// warm-start feature).  First every pair from its static lengths, then the
// pairs with dynamic incidences from their runs.
__global__ void k_static_stats(const unsigned long long* __restrict__ static_len, uint32_t np,
                               float* __restrict__ cum, float* __restrict__ stat, uint32_t* __restrict__ ndyn,
                               float* __restrict__ hit) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float s = len_float((long long)static_len[p]);
  cum[p] = s;
  stat[p] = kFEps * s;
  ndyn[p] = 0u;
  hit[p] = 0.0f;
}

// heads of the runs of one pair in the pair-sorted dynamic incidences
__global__ void k_run_heads(const uint32_t* __restrict__ sk, uint32_t n, uint32_t* __restrict__ flag) {
  uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) flag[k] = (k == 0 || sk[k] != sk[k - 1]) ? 1u : 0u;
}

// per run: its pair and first dynamic position
__global__ void k_runs(const uint32_t* __restrict__ sk, const uint32_t* __restrict__ flag,
                       const uint32_t* __restrict__ scan, uint32_t n, uint32_t pair_base, uint32_t dperm_base,
                       uint32_t* __restrict__ dpair, uint32_t* __restrict__ dseg) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !flag[k]) return;
  dpair[scan[k]] = pair_base + sk[k];
  dseg[scan[k]] = dperm_base + k;
}

// The potential mass is carried as an unevaluated FP32 pair (s, e) updated by
// an error-free two-sum (Knuth's TwoSum: e collects every rounding error of
// s), i.e. to about twice FP32's precision, and rounded once through FP64.
// GB300 issues FP64 at 1/64 of the FP32 rate: plain FP64 accumulation would
// make this kernel FP64-bound.  A thread sums a run, whose gathers are what it
// waits for: eight incidences' are in flight together (the build of five
// 160x120 views 2.46 -> 2.35 ms, of twelve 640x480 10.76 -> 10.45 against one
// at a time; short runs at 1 cm 33.3 either way; loads left out past the run's
// end instead of repeated 2.41 and 10.68).  Runs longer than kLongRun (voxels next to a camera) are appended
// to a list and summed by a whole block each.
constexpr uint32_t kLongRun = 512;
constexpr int kStatThreads = 256;

struct F2 {
  float s, e;
  __device__ __forceinline__ void add(float x) {
    const float t = __fadd_rn(s, x);
    const float bp = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp));
    e = __fadd_rn(e, err);
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)e; }
};

struct RunStats {
  static constexpr int kAhead = 8;
  const uint32_t* dpair;
  const uint32_t* dseg;
  const uint32_t* dperm;
  const float* len;
  const float* mu;
  const unsigned long long* static_len;
  uint32_t pair_base;
  float *cum, *hit;
  uint32_t* ndyn;

  __device__ __forceinline__ void add(uint32_t k, long long& d, F2& h) const {
    const uint32_t i = dperm[k];
    const float l = len[i];
    d += len_fixed(l);
    h.add(__fmul_rn(mu[i], l));
  }
  // kAhead incidences from k on (k1: the run's end), added in their order,
  // their gathers in flight together
  __device__ __forceinline__ void add_some(uint32_t k, uint32_t k1, long long& d, F2& h) const {
    uint32_t i[kAhead];
    float l[kAhead], u[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) i[q] = dperm[min(k + q, k1 - 1)];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      l[q] = len[i[q]];
      u[q] = mu[i[q]];
    }
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      if (k + q < k1) {
        d += len_fixed(l[q]);
        h.add(__fmul_rn(u[q], l[q]));
      }
    }
  }
  __device__ __forceinline__ void store(uint32_t j, uint32_t n, long long d, double h) const {
    const uint32_t p = dpair[j];
    cum[p] = len_float((long long)static_len[p - pair_base] + d);
    ndyn[p] = n;
    hit[p] = (float)h;
  }
};

__global__ void k_run_stats(RunStats a, uint32_t j0, uint32_t nrun, uint32_t* __restrict__ long_list) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrun) return;
  const uint32_t j = j0 + r;
  const uint32_t k0 = a.dseg[j], k1 = a.dseg[j + 1];
  if (k1 - k0 > kLongRun) {
    long_list[1 + atomicAdd(long_list, 1u)] = j;
    return;
  }
  long long d = 0;
  F2 h{0.0f, 0.0f};
  for (uint32_t k = k0; k < k1; k += RunStats::kAhead) a.add_some(k, k1, d, h);
  a.store(j, k1 - k0, d, h.value());
}

// one block per listed long run; block sums in a fixed tree order
__global__ void __launch_bounds__(kStatThreads)
    k_run_stats_long(RunStats a, const uint32_t* __restrict__ long_list) {
  __shared__ long long sd[kStatThreads];
  __shared__ double sh[kStatThreads];
  const uint32_t n = long_list[0];
  for (uint32_t q = blockIdx.x; q < n; q += gridDim.x) {
    const uint32_t j = long_list[1 + q];
    const uint32_t k0 = a.dseg[j], k1 = a.dseg[j + 1];
    long long d = 0;
    F2 h{0.0f, 0.0f};
    for (uint32_t k = k0 + threadIdx.x; k < k1; k += kStatThreads) a.add(k, d, h);
    sd[threadIdx.x] = d;
    sh[threadIdx.x] = h.value();
    __syncthreads();
    for (int o = kStatThreads / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) {
        sd[threadIdx.x] += sd[threadIdx.x + o];
        sh[threadIdx.x] += sh[threadIdx.x + o];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) a.store(j, k1 - k0, sd[0], sh[0]);
    __syncthreads();
  }
}

__global__ void k_iota(uint32_t* out, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}

}  // namespace

cudaError_t launch_clean_depth(const float* in, float* out, int rows, int cols, cudaStream_t s) {
  k_clean_depth<<<grid_for((int64_t)rows * cols), kThreads, 0, s>>>(in, out, rows, cols);
  return cudaGetLastError();
}

cudaError_t launch_activate(const Geom& g, const Pose& P, const float* depth, int policy,
                            uint8_t* flags, cudaStream_t s) {
  k_activate<<<grid_for(pixel_tiles(g.rows, g.cols) * 32, 128), 128, 0, s>>>(g, P, depth, policy, flags);
  return cudaGetLastError();
}

cudaError_t launch_activate_points(const Geom& g, const float* pts, int64_t n, uint8_t* flags,
                                   cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_activate_points<<<grid_for(n), kThreads, 0, s>>>(g, pts, n, flags);
  return cudaGetLastError();
}

cudaError_t launch_new_indicator(const uint8_t* flags, const int* slot, int* ind, int64_t n,
                                 cudaStream_t s) {
  k_new_indicator<<<grid_for(n), kThreads, 0, s>>>(flags, slot, ind, n);
  return cudaGetLastError();
}

cudaError_t launch_assign_slots2(const Geom& g, const int* ind, const int* scan, int nb_base,
                                 int* brick_slot, int* brick_coord, int64_t n, cudaStream_t s) {
  k_assign_slots<<<grid_for(n), kThreads, 0, s>>>(g, ind, scan, nb_base, brick_slot, brick_coord, n);
  return cudaGetLastError();
}

cudaError_t launch_fill_new_voxels(float* L, float* belief, int64_t v0, int64_t v1, float lp,
                                   cudaStream_t s) {
  if (v1 <= v0) return cudaSuccess;
  k_fill_new_voxels<<<grid_for(v1 - v0), kThreads, 0, s>>>(L, belief, v0, v1, lp);
  return cudaGetLastError();
}

cudaError_t launch_set_points(const Geom& g, const float* pts, const float* occ, int64_t n,
                              float* belief, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_set_points<<<grid_for(n), kThreads, 0, s>>>(g, pts, occ, n, belief);
  return cudaGetLastError();
}

// batches of up to kTraceBatch views, the blocks of one view after another's
template <typename F>
cudaError_t trace_batches(const TraceView* views, int n, F launch) {
  for (int k0 = 0; k0 < n; k0 += kTraceBatch) {
    TraceBatch b;
    b.n = std::min(kTraceBatch, n - k0);
    uint32_t blocks = 0;
    for (int k = 0; k < b.n; ++k) {
      b.v[k] = views[k0 + k];
      b.first[k] = blocks;
      blocks += grid_for(pixel_tiles(b.v[k].g.rows, b.v[k].g.cols) * 32, kTraceThreads);
    }
    b.first[b.n] = blocks;
    launch(b, blocks);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_trace_count(const TraceView* views, int n, int* err, cudaStream_t s) {
  return trace_batches(views, n, [&](const TraceBatch& b, uint32_t blocks) {
    k_trace_count<<<blocks, kTraceThreads, 0, s>>>(b, err);
  });
}

cudaError_t launch_trace_emit(const TraceView* views, int n, uint8_t* loud, int* err, cudaStream_t s) {
  return trace_batches(views, n, [&](const TraceBatch& b, uint32_t blocks) {
    k_trace_emit<<<blocks, kTraceThreads, 0, s>>>(b, loud, err);
  });
}

// The pixels of a view whose rays may cross one of the bricks in slots
// b0..b1 (bricks activated after the view's lists were built): each brick's
// eight corners projected through the view's camera (the inverse of
// ray_setup: a pixel's ray projects onto that pixel), the box of the
// projections widened by a pixel against rounding, marked in mask.  A brick
// with a corner at or behind the camera plane, or whose box covers more
// than a quarter of the image, sets *all instead (every pixel is checked).
__global__ void k_brick_footprint(Geom g, Pose P, const int* __restrict__ coord, uint32_t b0, uint32_t b1,
                                  uint8_t* __restrict__ mask, int* __restrict__ all) {
  const uint32_t b = b0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= b1) return;
  const float o0 = fa(fd(P.m[3], g.res), g.off[0]);
  const float o1 = fa(fd(P.m[7], g.res), g.off[1]);
  const float o2 = fa(fd(P.m[11], g.res), g.off[2]);
  const float kx = g.fx / g.cx, ky = g.fy / g.cy;
  float x_lo = 3.0e38f, x_hi = -3.0e38f, y_lo = 3.0e38f, y_hi = -3.0e38f;
  for (int k = 0; k < 8; ++k) {
    const float v0 = (float)(kBrick * (coord[3 * b + 0] + (k & 1))) - o0;
    const float v1 = (float)(kBrick * (coord[3 * b + 1] + ((k >> 1) & 1))) - o1;
    const float v2 = (float)(kBrick * (coord[3 * b + 2] + ((k >> 2) & 1))) - o2;
    const float xc = P.m[0] * v0 + P.m[4] * v1 + P.m[8] * v2;
    const float yc = P.m[1] * v0 + P.m[5] * v1 + P.m[9] * v2;
    const float zc = P.m[2] * v0 + P.m[6] * v1 + P.m[10] * v2;
    if (!(zc > 1e-3f)) {
      atomicExch(all, 1);
      return;
    }
    const float px = (xc / zc * kx + 1.0f) * 0.5f * (float)g.cols - 0.5f;
    const float py = (yc / zc * ky + 1.0f) * 0.5f * (float)g.rows - 0.5f;
    x_lo = fminf(x_lo, px);
    x_hi = fmaxf(x_hi, px);
    y_lo = fminf(y_lo, py);
    y_hi = fmaxf(y_hi, py);
  }
  const int x0 = max(0, (int)floorf(fmaxf(x_lo, -4.0f)) - 1);
  const int x1 = min(g.cols - 1, (int)ceilf(fminf(x_hi, (float)g.cols + 4.0f)) + 1);
  const int y0 = max(0, (int)floorf(fmaxf(y_lo, -4.0f)) - 1);
  const int y1 = min(g.rows - 1, (int)ceilf(fminf(y_hi, (float)g.rows + 4.0f)) + 1);
  if (x0 > x1 || y0 > y1) return;
  if ((int64_t)(x1 - x0 + 1) * (y1 - y0 + 1) * 4 > (int64_t)g.rows * g.cols) {
    atomicExch(all, 1);
    return;
  }
  for (int y = y0; y <= y1; ++y)
    for (int x = x0; x <= x1; ++x) mask[y * g.cols + x] = 1;
}

cudaError_t launch_brick_footprint(const Geom& g, const Pose& P, const int* coord, uint32_t b0, uint32_t b1,
                                   uint8_t* mask, int* all, cudaStream_t s) {
  if (b1 <= b0) return cudaSuccess;
  k_brick_footprint<<<grid_for(b1 - b0), kThreads, 0, s>>>(g, P, coord, b0, b1, mask, all);
  return cudaGetLastError();
}

cudaError_t launch_first_visit(const uint32_t* vox, uint32_t n, uint32_t* first, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_first_visit<<<grid_for(n / 4), kThreads, 0, s>>>(vox, n / 4, first);
  return cudaGetLastError();
}

cudaError_t launch_brick_count(uint32_t nb, const uint32_t* first, const uint8_t* loud, uint32_t* bfirst,
                               uint32_t* bloud, uint32_t* bquiet, cudaStream_t s) {
  if (!nb) return cudaSuccess;
  k_brick_count<<<grid_for((int64_t)nb * 32), kThreads, 0, s>>>(nb, first, loud, bfirst, bloud, bquiet);
  return cudaGetLastError();
}

cudaError_t launch_order_counts(const uint32_t* order, uint32_t nb, const uint32_t* bloud, const uint32_t* bquiet,
                                uint32_t* cnt, cudaStream_t s) {
  if (!nb) return cudaSuccess;
  k_order_counts<<<grid_for(nb), kThreads, 0, s>>>(order, nb, bloud, bquiet, cnt);
  return cudaGetLastError();
}

cudaError_t launch_brick_number(const uint32_t* bkey, const uint32_t* order, uint32_t nb, uint32_t* table,
                                const uint8_t* loud, const uint32_t* vox, const uint32_t* start,
                                uint32_t pair_base, uint32_t* pair_vox, cudaStream_t s) {
  if (!nb) return cudaSuccess;
  k_brick_number<<<grid_for((int64_t)nb * 32), kThreads, 0, s>>>(bkey, order, nb, table, loud, vox, start, pair_base,
                                                                 pair_vox);
  return cudaGetLastError();
}

cudaError_t launch_dyn_counts(const RayMeta* meta, uint32_t npix, uint32_t* cnt, cudaStream_t s) {
  if (!npix) return cudaSuccess;
  k_dyn_counts<<<grid_for(npix), kThreads, 0, s>>>(meta, npix, cnt);
  return cudaGetLastError();
}

cudaError_t launch_assign_pairs(const RayMeta* meta, uint32_t npix, const uint32_t* vox, const float* len,
                                const uint32_t* table, uint32_t inc_base, uint32_t pair_base, const uint32_t* doff,
                                uint32_t* inc_pair, unsigned long long* static_len, uint32_t* dkey, uint32_t* dval,
                                cudaStream_t s) {
  if (!npix) return cudaSuccess;
  k_assign_pairs<<<grid_for(npix, kNearRays), kNearThreads, 0, s>>>(
      meta, npix, vox, len, table, inc_base, pair_base, doff, inc_pair, static_len, dkey, dval);
  return cudaGetLastError();
}

cudaError_t launch_static_stats(const unsigned long long* static_len, uint32_t np, float* cum, float* stat,
                                uint32_t* ndyn, float* hit, cudaStream_t s) {
  if (!np) return cudaSuccess;
  k_static_stats<<<grid_for(np), kThreads, 0, s>>>(static_len, np, cum, stat, ndyn, hit);
  return cudaGetLastError();
}

cudaError_t launch_run_heads(const uint32_t* sk, uint32_t n, uint32_t* flag, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_run_heads<<<grid_for(n), kThreads, 0, s>>>(sk, n, flag);
  return cudaGetLastError();
}

cudaError_t launch_runs(const uint32_t* sk, const uint32_t* flag, const uint32_t* scan, uint32_t n,
                        uint32_t pair_base, uint32_t dperm_base, uint32_t* dpair, uint32_t* dseg, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_runs<<<grid_for(n), kThreads, 0, s>>>(sk, flag, scan, n, pair_base, dperm_base, dpair, dseg);
  return cudaGetLastError();
}

cudaError_t launch_run_stats(const uint32_t* dpair, const uint32_t* dseg, const uint32_t* dperm, uint32_t j0,
                             uint32_t nrun, const float* len, const float* mu,
                             const unsigned long long* static_len, uint32_t pair_base, float* cum, uint32_t* ndyn,
                             float* hit, uint32_t* long_list, cudaStream_t s) {
  if (!nrun) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(long_list, 0, 4, s);
  if (e != cudaSuccess) return e;
  const RunStats a{dpair, dseg, dperm, len, mu, static_len, pair_base, cum, hit, ndyn};
  k_run_stats<<<grid_for(nrun), kThreads, 0, s>>>(a, j0, nrun, long_list);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_run_stats_long<<<1024, kStatThreads, 0, s>>>(a, long_list);
  return cudaGetLastError();
}

cudaError_t launch_count_loud(const uint32_t* pair_vox, uint32_t np, const uint8_t* loud, uint32_t* count,
                              cudaStream_t s) {
  if (!np) return cudaSuccess;
  k_count_loud<<<grid_for(np), kThreads, 0, s>>>(pair_vox, np, loud, count);
  return cudaGetLastError();
}

cudaError_t launch_iota(uint32_t* out, uint32_t n, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_iota<<<grid_for(n), kThreads, 0, s>>>(out, n);
  return cudaGetLastError();
}

size_t scan_temp_bytes(uint32_t n) {
  size_t b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b, (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n);
  return b;
}

cudaError_t exclusive_scan_u32(void* tmp, size_t tmp_bytes, const uint32_t* in, uint32_t* out,
                               uint32_t n, cudaStream_t s) {
  return cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, in, out, (int)n, s);
}

size_t scan_temp_bytes_i32(int64_t n) {
  size_t b = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, b, (const int*)nullptr, (int*)nullptr, (int)n);
  return b;
}

cudaError_t exclusive_scan_i32(void* tmp, size_t tmp_bytes, const int* in, int* out, int64_t n,
                               cudaStream_t s) {
  return cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, in, out, (int)n, s);
}

size_t sort_temp_bytes(uint32_t n, int bits) {
  size_t b = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, b, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                  (const uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0, bits);
  return b;
}

cudaError_t sort_pairs_u32(void* tmp, size_t tmp_bytes, const uint32_t* kin, uint32_t* kout,
                           const uint32_t* vin, uint32_t* vout, uint32_t n, int bits,
                           cudaStream_t s) {
  return cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kin, kout, vin, vout, (int)n, 0, bits, s);
}

}  // namespace mrf
