// mrf_geometry.cuh -- device geometry shared by the traversal, activation and
// likelihood kernels: pixel rays, the voxel DDA over the brick grid, the
// sensor polynomials and the depth potential.
//
// Every geometric quantity is built from separately rounded fp32 operations
// (__fmul_rn/__fadd_rn/__fdiv_rn, which nvcc never contracts into FMAs), in
// one fixed order, so the incidence lists are reproducible bit for bit on any
// host that evaluates the same IEEE operations.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mrf_internal.h"

namespace mrf {

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

// The traversal kernels give a warp 8 x 4 pixels: 32 pixels of a row span
// several bricks a few metres out, and lanes that enter and leave their bricks
// at different steps wait for one another (15 of 32 active); the tile's rays
// mostly share a brick.  (Likelihood and renders: kViewTileX x kViewTileY.)
template <int kTileX = 8, int kTileY = 4>
__device__ __forceinline__ int tile_pixel(int rows, int cols, int64_t tile, int lane) {
  const int tx = (cols + kTileX - 1) / kTileX;
  const int x = (int)(tile % tx) * kTileX + lane % kTileX;
  const int64_t y = tile / tx * kTileY + lane / kTileX;
  return x < cols && y < rows ? (int)y * cols + x : -1;
}

// depth clean-up of pixel i of a rows x cols image (src/GVDBImage.cpp:32-40):
// a non-finite return becomes "no return" (-1), and 848x480 images lose a
// 24-pixel left/right and a 20-pixel top/bottom border
__device__ __forceinline__ float clean_depth_value(float d, int i, int rows, int cols) {
  float v = isfinite(d) ? d : -1.0f;
  if (rows == 480 && cols == 848) {
    int x = i % cols, y = i / cols;
    if (x < 24 || x >= cols - 24 || y < 20 || y >= rows - 20) v = -1.0f;
  }
  return v;
}

// per-20x20-tile coefficient rows; tiles indexed by the upward (GL) row as in
// gvdbkernels.cu:47 (the reference flips the image on upload)
// a camera of another resolution than the tables' maps its pixel into the
// tables' image (identity for the map's own camera)
__device__ __forceinline__ const float* lut_at(const Geom& g, const float* lut, int x, int y) {
  int ygl = g.rows - 1 - y;
  int xs = (int)(((int64_t)x * g.lut_cols) / g.cols);
  int ys = (int)(((int64_t)ygl * g.lut_rows) / g.rows);
  return lut + ((ys / kLookupPx) * g.n_tiles_u + (xs / kLookupPx)) * g.lookup_n;
}

// sensor polynomials p0 + p1 z (+ p2 z^2) of a pixel's tile, the standard
// deviation's and the bias's (src/cuda/gvdbkernels.cu:46-55); a degree-1 table
// gets p2 = 0, which leaves the value unchanged
struct Sensor {
  float s[3], b[3];
  __device__ __forceinline__ static float poly(const float* c, float z) {
    return fa(fa(fm(fm(z, z), c[2]), fm(z, c[1])), c[0]);
  }
  __device__ __forceinline__ float sigma(float z) const { return poly(s, z); }
  __device__ __forceinline__ float bias(float z) const { return poly(b, z); }
};

__device__ __forceinline__ Sensor sensor_at(const Geom& g, int x, int y) {
  const float* sg = lut_at(g, g.sigma, x, y);
  const float* bs = lut_at(g, g.bias, x, y);
  Sensor c;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    c.s[k] = k < g.lookup_n ? sg[k] : 0.0f;
    c.b[k] = k < g.lookup_n ? bs[k] : 0.0f;
  }
  return c;
}

// A range s below which d - s > k sigma(s) for certain, so that the tests
// against the return's window need no polynomials there: the smaller root of
// s + k sigma(s) = d, taken in a little.  Only where sigma grows with s and
// there is no bias, else 0 (every s is tested).
__device__ __forceinline__ float window_start(const Sensor& c, float d, float k, float shrink) {
  if (!(c.s[0] >= 0.0f && c.s[1] >= 0.0f && c.s[2] >= 0.0f && c.b[0] == 0.0f && c.b[1] == 0.0f && c.b[2] == 0.0f))
    return 0.0f;
  const float e = d - k * c.s[0], b = 1.0f + k * c.s[1];
  if (!(e > 0.0f)) return 0.0f;
  return shrink * (2.0f * e / (b + sqrtf(b * b + 4.0f * k * c.s[2] * e)));
}

// exact-zero test of the fp32 depth potential (gvdbkernels.cu:57-72; the
// reference's __expf flushes below 2^-126).  The test divides; sqrt(2
// kMuCutoff) = 13.19, so beyond 13.3 sigma' the answer is known without.
__device__ __forceinline__ bool potential_is_zero(const Sensor& c, float s, float d) {
  const float sig3 = fm(3.0f, c.sigma(s));
  const float diff = fabsf(fs(d, fa(s, c.bias(s))));
  if (sig3 > 0.0f && diff > fm(13.3f, sig3)) return true;
  const float x = fd(diff, sig3);
  const float h = fm(0.5f, fm(x, x));
  return !(h <= kMuCutoff);
}

// Gaussian depth potential with sigma' = 3 sigma(s)
__device__ __forceinline__ float potential(const Sensor& c, float s, float d) {
  const float sig3 = 3.0f * c.sigma(s);
  const float diff = fabsf(d - (s + c.bias(s)));
  const float x = diff / sig3;
  return 0.398942f / sig3 * expf(-0.5f * x * x);
}

// pixel-centre ray through the reference's symmetric GL frustum
// (src/GVDBCamera.cpp:7-32, gvdbkernels.cu:1178-1179), origin and direction
// in voxel units, and the ray-parameter -> z-depth factor (gvdbkernels.cu:837)
struct Ray {
  float o[3], d[3], mult;
};

__device__ __forceinline__ void ray_setup(const Geom& g, const Pose& P, int x, int y, Ray& r) {
  float W = (float)g.cols, H = (float)g.rows;
  float ndcx = fs(fm(2.0f, fd(fa((float)x, 0.5f), W)), 1.0f);
  float ndcy = fs(fm(2.0f, fd(fa((float)y, 0.5f), H)), 1.0f);
  float rx = fm(ndcx, fd(g.cx, g.fx));
  float ry = fm(ndcy, fd(g.cy, g.fy));
  float dw0 = fa(fa(fm(P.m[0], rx), fm(P.m[1], ry)), P.m[2]);
  float dw1 = fa(fa(fm(P.m[4], rx), fm(P.m[5], ry)), P.m[6]);
  float dw2 = fa(fa(fm(P.m[8], rx), fm(P.m[9], ry)), P.m[10]);
  float n = __fsqrt_rn(fa(fa(fm(dw0, dw0), fm(dw1, dw1)), fm(dw2, dw2)));
  r.d[0] = fd(dw0, n);
  r.d[1] = fd(dw1, n);
  r.d[2] = fd(dw2, n);
  r.o[0] = fa(fd(P.m[3], g.res), g.off[0]);
  r.o[1] = fa(fd(P.m[7], g.res), g.off[1]);
  r.o[2] = fa(fd(P.m[11], g.res), g.off[2]);
  r.mult = fm(g.res, fabsf(fa(fa(fm(P.m[2], r.d[0]), fm(P.m[6], r.d[1])), fm(P.m[10], r.d[2]))));
}

// Amanatides & Woo voxel DDA over the box [blo, bhi) of the brick grid (the
// whole grid [0, 8*NB) unless the view is confined to a scene box).  The
// next boundary time of an axis is recomputed from the integer boundary each
// step, (b - o) * (1/d), so no error accumulates along the ray; ties step x
// before y before z.
//
// A step is a few predicated instructions per axis, without a branch: a
// warp's rays step different axes.  The position inside the brick is kept as three 4-bit
// fields whose top bits show when the step left the brick; bricks change
// once in ten steps.  dda_cross leaves a whole brick at once: the exit is
// the first face in (time, axis) order, and every other axis has passed the
// boundaries that come before it in that order, so the state is the one that
// single steps reach, bit for bit.
//
// The traversals are bound by instructions and by lanes that wait.  With
// voxel-wise steps that branched on the axis and a warp per row of 32 pixels,
// a 640x480 view of 104 M incidences at 1 cm took 0.72 ms to activate, 0.94 to
// count and 1.75 to emit, a likelihood image 1.26; with brick-wise activation
// and counting, tiles, and warps that cross a brick together 0.15, 0.14, 0.93
// and 0.54.
struct Dda {
  float ox, oy, oz, ix, iy, iz;  // origin, 1 / direction (1 on an axis the ray does not move along)
  float bx, by, bz, sx, sy, sz;  // next boundaries (INFINITY ...) and their steps (+1, -1 or 0)
  float tx, ty, tz, tprev;
  int kx, ky, kz;                // brick
  int dx, dy, dz;                // steps of loc
  uint32_t loc;                  // x << 8 | y << 4 | z inside the brick
  int64_t lin;                   // brick index
  int guard;
  bool alive;
};

__device__ __forceinline__ bool dda_axis(float o, float d, int lo, int hi, float& inv, float& tn, float& tf) {
  if (d > 0.0f || d < 0.0f) {
    inv = fd(1.0f, d);
    float tA = fm(fs((float)lo, o), inv);
    float tB = fm(fs((float)hi, o), inv);
    tn = fminf(tA, tB);
    tf = fmaxf(tA, tB);
    return true;
  }
  inv = 1.0f;
  if (o < (float)lo || o >= (float)hi) return false;
  tn = -INFINITY;
  tf = INFINITY;
  return true;
}

__device__ __forceinline__ int dda_start(float o, float t0, float d, int lo, int hi) {
  int v = (int)floorf(fa(o, fm(t0, d)));
  return v < lo ? lo : (v > hi - 1 ? hi - 1 : v);
}

__device__ __forceinline__ float dda_boundary(int v, float s) {
  return s > 0.0f ? (float)(v + 1) : (s < 0.0f ? (float)v : INFINITY);
}

__device__ __forceinline__ void dda_times(Dda& r) {
  r.tx = fm(fs(r.bx, r.ox), r.ix);
  r.ty = fm(fs(r.by, r.oy), r.iy);
  r.tz = fm(fs(r.bz, r.oz), r.iz);
}

__device__ __forceinline__ bool dda_init(Dda& r, const Geom& g, const Ray& ray) {
  float tn0, tf0, tn1, tf1, tn2, tf2;
  if (!dda_axis(ray.o[0], ray.d[0], g.blo[0], g.bhi[0], r.ix, tn0, tf0)) return false;
  if (!dda_axis(ray.o[1], ray.d[1], g.blo[1], g.bhi[1], r.iy, tn1, tf1)) return false;
  if (!dda_axis(ray.o[2], ray.d[2], g.blo[2], g.bhi[2], r.iz, tn2, tf2)) return false;
  float t0 = fmaxf(fmaxf(fmaxf(0.0f, tn0), tn1), tn2);
  float t1 = fminf(fminf(fminf(INFINITY, tf0), tf1), tf2);
  if (!(t0 < t1)) return false;
  r.ox = ray.o[0]; r.oy = ray.o[1]; r.oz = ray.o[2];
  const int vx = dda_start(ray.o[0], t0, ray.d[0], g.blo[0], g.bhi[0]);
  const int vy = dda_start(ray.o[1], t0, ray.d[1], g.blo[1], g.bhi[1]);
  const int vz = dda_start(ray.o[2], t0, ray.d[2], g.blo[2], g.bhi[2]);
  r.sx = ray.d[0] > 0.0f ? 1.0f : (ray.d[0] < 0.0f ? -1.0f : 0.0f);
  r.sy = ray.d[1] > 0.0f ? 1.0f : (ray.d[1] < 0.0f ? -1.0f : 0.0f);
  r.sz = ray.d[2] > 0.0f ? 1.0f : (ray.d[2] < 0.0f ? -1.0f : 0.0f);
  // a pose with NaN: no direction or no origin, no voxels
  if (r.sx == 0.0f && r.sy == 0.0f && r.sz == 0.0f) return false;
  if (isnan(r.ox) || isnan(r.oy) || isnan(r.oz)) return false;
  r.bx = dda_boundary(vx, r.sx);
  r.by = dda_boundary(vy, r.sy);
  r.bz = dda_boundary(vz, r.sz);
  dda_times(r);
  r.tprev = t0;
  r.kx = vx >> 3;
  r.ky = vy >> 3;
  r.kz = vz >> 3;
  r.dx = (int)r.sx * 0x100;
  r.dy = (int)r.sy * 0x10;
  r.dz = (int)r.sz;
  r.loc = (uint32_t)((vx & 7) << 8 | (vy & 7) << 4 | (vz & 7));
  r.lin = ((int64_t)r.kx * g.NB[1] + r.ky) * g.NB[2] + r.kz;
  r.alive = true;
  r.guard = 2 * ((g.bhi[0] - g.blo[0]) + (g.bhi[1] - g.blo[1]) + (g.bhi[2] - g.blo[2])) + 8;
  return true;
}

// the next brick along the axis (px: x, py: y, else z)
__device__ __forceinline__ void dda_next_brick(Dda& r, const Geom& g, bool px, bool py) {
  const int s = (int)(px ? r.sx : (py ? r.sy : r.sz));
  int k;
  if (px) {
    k = (r.kx += s);
    r.lin += (int64_t)s * g.NB[1] * g.NB[2];
  } else if (py) {
    k = (r.ky += s);
    r.lin += (int64_t)s * g.NB[2];
  } else {
    k = (r.kz += s);
    r.lin += s;
  }
  const int a = px ? 0 : (py ? 1 : 2);
  r.alive = k >= (g.blo[a] >> 3) && k < (g.bhi[a] >> 3);
}

// voxel index inside the brick
__device__ __forceinline__ uint32_t dda_local(const Dda& r) {
  return (r.loc >> 2 & 0x1C0u) | (r.loc >> 1 & 0x38u) | (r.loc & 7u);
}

// leaves the current voxel: its segment length, entry and exit parameters;
// true when the step left the brick
__device__ __forceinline__ bool dda_step(Dda& r, const Geom& g, float& len, float& tin, float& texit) {
  const bool px = r.tx <= r.ty && r.tx <= r.tz;
  const bool py = !px && r.ty <= r.tz;
  tin = r.tprev;
  const float te = px ? r.tx : (py ? r.ty : r.tz);
  const float l = fs(te, tin);
  len = l < 0.0f ? 0.0f : l;  // keeps a -0
  texit = te;
  r.tprev = fmaxf(r.tprev, te);
  if (px) {
    r.bx = fa(r.bx, r.sx);
    r.tx = fm(fs(r.bx, r.ox), r.ix);
  }
  if (py) {
    r.by = fa(r.by, r.sy);
    r.ty = fm(fs(r.by, r.oy), r.iy);
  }
  if (!px && !py) {
    r.bz = fa(r.bz, r.sz);
    r.tz = fm(fs(r.bz, r.oz), r.iz);
  }
  --r.guard;
  const uint32_t old = r.loc;
  const int dl = px ? r.dx : (py ? r.dy : r.dz);
  r.loc = old + (uint32_t)dl;
  if (!(r.loc & 0x888u)) return false;
  const uint32_t field = px ? 0x700u : (py ? 0x70u : 0x7u);
  r.loc = (old & ~field) | (dl < 0 ? field : 0u);
  dda_next_brick(r, g, px, py);
  return true;
}

// an axis's next boundary after the exit at te (e: its brick face's
// boundary; before: the axis comes before the exit axis at equal times)
__device__ __forceinline__ float dda_pass(float b, float e, float s, float o, float inv, float d, float te,
                                          bool before) {
  if (s == 0.0f) return b;
  auto passed = [&](float n) {
    const float t = fm(fs(n, o), inv);
    return before ? t <= te : t < te;
  };
  // the first boundary behind the exit point up to rounding, then exactly
  float n = s * fminf(fmaxf(floorf(s * (o + te * d)) + 1.0f, s * b), s * e);
  while (n != b && !passed(n - s)) n -= s;
  while (n != e && passed(n)) n += s;
  return n;
}

// leaves the current brick: the exit parameter; steps: the voxels crossed
__device__ __forceinline__ float dda_cross(Dda& r, const Geom& g, const Ray& ray, int& steps) {
  const float ex = r.sx > 0.0f ? (float)(8 * r.kx + 8) : (r.sx < 0.0f ? (float)(8 * r.kx) : INFINITY);
  const float ey = r.sy > 0.0f ? (float)(8 * r.ky + 8) : (r.sy < 0.0f ? (float)(8 * r.ky) : INFINITY);
  const float ez = r.sz > 0.0f ? (float)(8 * r.kz + 8) : (r.sz < 0.0f ? (float)(8 * r.kz) : INFINITY);
  const float tx = fm(fs(ex, r.ox), r.ix), ty = fm(fs(ey, r.oy), r.iy), tz = fm(fs(ez, r.oz), r.iz);
  const bool px = tx <= ty && tx <= tz;
  const bool py = !px && ty <= tz;
  const float te = px ? tx : (py ? ty : tz);
  const float nx = px ? ex + r.sx : dda_pass(r.bx, ex, r.sx, r.ox, r.ix, ray.d[0], te, true);
  const float ny = py ? ey + r.sy : dda_pass(r.by, ey, r.sy, r.oy, r.iy, ray.d[1], te, !px);
  const float nz = px || py ? dda_pass(r.bz, ez, r.sz, r.oz, r.iz, ray.d[2], te, false) : ez + r.sz;
  int n = 0;
  auto move = [&](float& b, float nb, float s, int shift) {
    if (s == 0.0f) return;
    n += (int)fabsf(nb - b);
    b = nb;
    const int v = (int)(s > 0.0f ? nb - 1.0f : nb);
    r.loc = (r.loc & ~(7u << shift)) | ((uint32_t)(v & 7) << shift);
  };
  move(r.bx, nx, r.sx, 8);
  move(r.by, ny, r.sy, 4);
  move(r.bz, nz, r.sz, 0);
  dda_times(r);
  r.tprev = fmaxf(r.tprev, te);
  r.guard -= max(n, 1);
  dda_next_brick(r, g, px, py);
  steps = n;
  return te;
}

// The current voxel's coordinates as floats, from the boundaries: behind the
// next one on an axis that counts up, at it on one that counts down, and fixed
// (the boundary is INFINITY) on an axis the ray does not move along.
struct Corner {
  float ux, uy, uz, fx, fy, fz;
  __device__ __forceinline__ explicit Corner(const Dda& r) {
    ux = r.sx > 0.0f ? -1.0f : 0.0f;
    uy = r.sy > 0.0f ? -1.0f : 0.0f;
    uz = r.sz > 0.0f ? -1.0f : 0.0f;
    fx = r.sx == 0.0f ? (float)(8 * r.kx + (int)(r.loc >> 8 & 7)) : INFINITY;
    fy = r.sy == 0.0f ? (float)(8 * r.ky + (int)(r.loc >> 4 & 7)) : INFINITY;
    fz = r.sz == 0.0f ? (float)(8 * r.kz + (int)(r.loc & 7)) : INFINITY;
  }
  __device__ __forceinline__ float x(const Dda& r) const { return fminf(r.bx + ux, fx); }
  __device__ __forceinline__ float y(const Dda& r) const { return fminf(r.by + uy, fy); }
  __device__ __forceinline__ float z(const Dda& r) const { return fminf(r.bz + uz, fz); }
};

// Walks on to the next active brick: its slot, -1 at the end of the ray.
__device__ __forceinline__ int dda_next_active(Dda& r, const Geom& g, const Ray& ray) {
  while (r.alive && r.guard > 0) {
    const int slot = g.brick_slot[r.lin];
    if (slot >= 0) return slot;
    int steps;
    dda_cross(r, g, ray, steps);
  }
  return -1;
}

__device__ __forceinline__ int64_t brick_lin(const Geom& g, int vx, int vy, int vz) {
  return ((int64_t)(vx >> 3) * g.NB[1] + (vy >> 3)) * g.NB[2] + (vz >> 3);
}

__device__ __forceinline__ uint32_t voxel_local(int vx, int vy, int vz) {
  return (uint32_t)((((vx & 7) << 3) | (vy & 7)) << 3 | (vz & 7));
}

}  // namespace mrf
