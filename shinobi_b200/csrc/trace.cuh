// What the traversal engines share: the grid view, the watertight ray/triangle
// test and camera rays.
//
// The traversal (trace_coop.cuh, trace_flat.cuh) restates UniformGridTraverser (src/Control/Algorithm/SimpleGridTraverser.h:274-401)
// and TwoLevelGridTraverser (src/Control/Algorithm/TwoLevelGridTraverser.h:445-671):
// float cell coordinates, continuation while the best t exceeds the current
// cell's exit (min of tMax), exit when a coordinate reaches res or -1 within
// 0.1.  Cell lookups clamp the coordinates like the reference's tex3D did;
// each DDA level carries a step cap of res.x+res.y+res.z+3.  Any-hit stops at
// the first hit in (EPS, tmax).
//
// Two-level grids keep a reference-ordered SoA float4 copy of the triangles
// (v0[ref], v1[ref], v2[ref]; v0.w carries the triangle id), so a leaf's
// candidates are contiguous; uniform grids keep a copy of the scene's records
// and read them through indices[].
#pragma once
#include "common.cuh"

namespace shn {

struct GridView {
  Geom g;
  uint32_t kind;
  const uint2* __restrict__ cells;
  const uint2* __restrict__ leaves;
  const float4* __restrict__ rv0;
  const float4* __restrict__ rv1;
  const float4* __restrict__ rv2;
  // the scene's triangle records as they are now (48 bytes: v0 with the id in
  // w, v1, v2), indexed by the id that rv0[].w holds: for u and v
  const float4* __restrict__ src;
  // boxes (min, max) of references [32k, 32k + 32) and [1024s, 1024s + 1024)
  // of rv*, or null (no culling)
  const float4* __restrict__ cbox;
  const float4* __restrict__ sbox;
  // when not null: no reference-ordered copy; reference i is rec[3 * ridx[i]],
  // rec the records as they were at the build
  const uint32_t* __restrict__ ridx;
  const float4* __restrict__ rec;
};

struct Hit {
  float t;
  uint32_t tri;
  float u, v;
  uint32_t steps = 0, tests = 0;  // work counters (only read by the stats variants)
};

// Watertight ray/triangle test (Woop, Benthin, Wald, JCGT 2(1), 2013).
struct RayWT {
  V3 org;
  int kx, ky, kz;
  float Sx, Sy, Sz;
};

SHN_D float sel(int k, V3 v) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

SHN_D RayWT wt_setup(V3 org, V3 d) {
  RayWT r;
  r.org = org;
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  r.kz = (ax > ay) ? ((ax > az) ? 0 : 2) : ((ay > az) ? 1 : 2);
  r.kx = r.kz + 1 == 3 ? 0 : r.kz + 1;
  r.ky = r.kx + 1 == 3 ? 0 : r.kx + 1;
  if (sel(r.kz, d) < 0.f) {
    const int t = r.kx;
    r.kx = r.ky;
    r.ky = t;
  }
  const float dz = sel(r.kz, d);
  r.Sx = sel(r.kx, d) / dz;
  r.Sy = sel(r.ky, d) / dz;
  r.Sz = 1.0f / dz;
  return r;
}

SHN_D bool wt_test(const RayWT& r, float4 p0, float4 p1, float4 p2, float tmin, float tbest,
                   float& t, float& u, float& v) {
  const V3 A = sub(f4v(p0), r.org), B = sub(f4v(p1), r.org), C = sub(f4v(p2), r.org);
  const float Akz = sel(r.kz, A), Bkz = sel(r.kz, B), Ckz = sel(r.kz, C);
  // shear: one fused multiply-add per coordinate; edge functions: one product
  // rounded, then a fused multiply-add (the oracle uses fmaf identically)
  const float Ax = __fmaf_rn(-r.Sx, Akz, sel(r.kx, A));
  const float Ay = __fmaf_rn(-r.Sy, Akz, sel(r.ky, A));
  const float Bx = __fmaf_rn(-r.Sx, Bkz, sel(r.kx, B));
  const float By = __fmaf_rn(-r.Sy, Bkz, sel(r.ky, B));
  const float Cx = __fmaf_rn(-r.Sx, Ckz, sel(r.kx, C));
  const float Cy = __fmaf_rn(-r.Sy, Ckz, sel(r.ky, C));
  float U = __fmaf_rn(Cx, By, -(Cy * Bx));
  float V = __fmaf_rn(Ax, Cy, -(Ay * Cx));
  float W = __fmaf_rn(Bx, Ay, -(By * Ax));
  // exact zero of an edge function -> recompute in double; mixed signs -> miss
  // (min/max skip a NaN operand exactly as or-chains of comparisons do)
  if (fminf(fminf(fabsf(U), fabsf(V)), fabsf(W)) == 0.f) {
    U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
    V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
    W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
  }
  if (fminf(fminf(U, V), W) < 0.f && fmaxf(fmaxf(U, V), W) > 0.f) return false;
  const float det = U + V + W;
  if (det == 0.f) return false;
  const float T = __fmaf_rn(W, r.Sz * Ckz, __fmaf_rn(V, r.Sz * Bkz, U * (r.Sz * Akz)));
  const float tt = T / det;
  if (!(tt > tmin && tt < tbest)) return false;
  t = tt;
  u = V / det;
  v = W / det;
  return true;
}

// Closest hit in a range: the least (t, triangle id) below the bound from
// earlier cells, i.e. the first minimum in triangle-id order, which is what a
// strict-< loop over the references in (cell, triangle) order keeps.  The
// references of a range may be stored in another order, so a candidate may
// tie the range's running minimum (bound = next float above it) and wins on
// the smaller id.
SHN_D float next_up(float t) { return __uint_as_float(__float_as_uint(t) + 1u); }

SHN_D int min_dim(V3 t) { return (t.x < t.y) ? ((t.x < t.z) ? 0 : 2) : ((t.y < t.z) ? 1 : 2); }
SHN_D float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
SHN_D void bump(V3& v, int d, float a) {
  if (d == 0) v.x += a; else if (d == 1) v.y += a; else v.z += a;
}

// Camera::init result + RegularPixelSampler<1,1> (src/Primitive/Camera.h:67-70,
// src/Primitive/PixelSampler.h:40-52).
struct CamView {
  V3 eye, tl, sx, sy;
  float resx;
  uint32_t res_x, res_y;
};

SHN_D V3 primary_dir(const CamView& c, uint32_t id, uint32_t image_id) {
  float tmp = (float)image_id / 1.0f;
  float py = (truncf(tmp) + 0.5f) / 1.0f;
  float px = tmp - truncf(tmp) + 0.5f / 1.0f;
  tmp = (float)id / c.resx;
  py += truncf(tmp);
  px += (tmp - truncf(tmp)) * c.resx;
  return mk(c.tl.x + px * c.sx.x + py * c.sy.x, c.tl.y + px * c.sx.y + py * c.sy.y,
            c.tl.z + px * c.sx.z + py * c.sy.z);
}

// Camera ray r -> pixel: rays 32k .. 32k+31 (one warp's packet) cover the
// 8x4 pixel tile k of the image (tiles row by row); the pixels right of the
// last full tile column and below the last full tile row follow in row
// order.  A bijection of [0, resx*resy).  With packet refill the 32 rays of
// a warp are one compact tile: camera kernel 2.22 -> 2.06 ms on the
// 1M-triangle cluster at 1920x1080 (32x1 rows before).
SHN_D uint32_t tile_pixel(const CamView& c, uint32_t r) {
  const uint32_t rx = c.res_x, ry = c.res_y;
  const uint32_t W = rx & ~7u, H = ry & ~3u;
  if (r < W * H) {
    const uint32_t t = r >> 5, q = r & 31u, tw = W >> 3;
    const uint32_t ty = t / tw, tx = t - ty * tw;
    return (ty * 4 + (q >> 3)) * rx + tx * 8 + (q & 7u);
  }
  r -= W * H;
  const uint32_t sw = rx - W;
  if (r < sw * H) {
    const uint32_t y = r / sw;
    return y * rx + W + (r - y * sw);
  }
  r -= sw * H;
  return H * rx + r;
}

}  // namespace shn
