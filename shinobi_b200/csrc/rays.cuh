// Rays made on the device from a frame's primary hits: ambient occlusion and
// the shadow segments of direct illumination, for the trace kernels of both
// engines.
#pragma once
#include "trace.cuh"

namespace shn {

// Rays from arrays: coordinate c of ray i at c[i * stride].  Rays kept as
// (n, 3) arrays are read in place; copying their columns out first took six
// launches, 19 of the 74 us of a call with 1,021 rays and 78 of the 930 us of
// one with 4.0M.
struct RaysView {
  const float *ox, *oy, *oz, *dx, *dy, *dz, *tmax;
  long long so, sd, st;
  SHN_D void ray(uint32_t i, V3& o, V3& d, float& t) const {
    const long long a = i * so, b = i * sd;
    o = mk(__ldg(ox + a), __ldg(oy + a), __ldg(oz + a));
    d = mk(__ldg(dx + b), __ldg(dy + b), __ldg(dz + b));
    t = tmax ? __ldg(tmax + i * st) : FLT_MAX;
  }
};

struct AoParams {
  CamView cam;
  uint32_t image_id, spp, seed;
  float len, offset;
  const float4* stri;  // scene triangles, 48-byte records (v0, v1, v2)
  uint32_t snt;
  uint32_t npix;
};

// Occlusion ray r = sample r % spp of the hit pixel number r / spp.
struct AoRays {
  AoParams A;
  const uint32_t* ptri;
  const float* pt;
  const uint32_t* hit_idx;
  uint8_t* occ;
  SHN_D void ray(uint32_t r, V3& o, V3& dir, float& tmax) const {
    const uint32_t k = r / A.spp, s = r - k * A.spp;
    const uint32_t p = hit_idx[k];
    // a compaction whose look-back gave up (error bit set) can leave a
    // slot unwritten: such a ray becomes an empty segment, no access leaves
    // the pixel and triangle arrays
    const uint32_t tri = p < A.npix ? ptri[p] : kMiss;
    if (tri >= A.snt) {
      o = A.cam.eye;
      dir = mk(0.f, 0.f, 1.f);
      tmax = 0.f;
      return;
    }
    const float t = pt[p];
    const V3 d = primary_dir(A.cam, p, A.image_id);
    const float4* rec = A.stri + 3 * (size_t)tri;
    const V3 v0 = f4v(__ldg(rec));
    const V3 v1 = f4v(__ldg(rec + 1));
    const V3 v2 = f4v(__ldg(rec + 2));
    const V3 e1 = sub(v1, v0);
    V3 nn = normalize(cross(e1, sub(v2, v0)));
    if (dot(nn, d) > 0.f) nn = mk(-nn.x, -nn.y, -nn.z);
    const V3 tx = normalize(e1);
    const V3 ty = cross(nn, tx);
    const V3 hp = add(A.cam.eye, muls(d, t));
    o = add(hp, muls(nn, A.offset));
    const uint4 w = philox4x32(make_uint4(p, s, 0u, 0x414Fu), A.seed, 0u);
    const float u1 = u01(w.x), u2 = u01(w.y);
    float sn, cs;
    sincos_2pi(u1, sn, cs);
    const float rr = sqrtf(1.f - u2);
    const float lx = sn * rr, ly = cs * rr, lz = sqrtf(u2);
    dir = mk(tx.x * lx + ty.x * ly + nn.x * lz, tx.y * lx + ty.y * ly + nn.y * lz,
             tx.z * lx + ty.z * ly + nn.z * lz);
    tmax = A.len;
  }
  SHN_D void done(uint32_t r, const Hit& h) const { occ[r] = h.tri != kMiss ? 1 : 0; }
};

// Direct illumination from a parallelogram light (DirectIlluminationIntegrator::shade,
// src/Integrator/DirectIlluminationIntegrator.h:254-315, and computeDirectIllumination,
// src/Integrator/DirectIlluminationIntegrator.h:46-168).
struct DiParams {
  CamView cam;
  V3 lpos, le1, le2, lnrm, lint, ddef, bg;
  float larea;
  uint32_t spp, seed, image_id, nmat, npix;
  const float4* stri;        // scene triangles, 48-byte records (v0, v1, v2)
  const uint32_t* tri_mat;   // per scene triangle, or null
  const float4* diffuse;     // per material, or null
};

// Shadow segment of sample s of hit pixel p: the origin is the stored hit point
// eye + (t - EPS) d (SimpleRayBuffer::store, src/Engine/RayBuffers.h:52-55), the
// direction runs to a uniform point of the light (AreaLightShadowRayGenerator,
// src/Engine/RayGenerators.h:106-139; AreaLightSource::getPoint,
// src/Primitive/LightSource.hpp:40-43); Philox replaces the KISS generator.
SHN_D void di_segment(const DiParams& P, uint32_t p, uint32_t s, float t, V3& o, V3& L) {
  const V3 d = primary_dir(P.cam, p, P.image_id);
  o = add(P.cam.eye, muls(d, t - 1e-5f));
  const uint4 w = philox4x32(make_uint4(p, s, P.image_id, 0x444Cu), P.seed, 0u);
  const V3 lp = add(add(P.lpos, muls(P.le1, u01(w.x))), muls(P.le2, u01(w.y)));
  L = sub(lp, o);
}

struct DiRays {
  DiParams P;
  const float* pt;
  const uint32_t* hit_idx;
  uint8_t* occ;
  SHN_D void ray(uint32_t r, V3& o, V3& dir, float& tmax) const {
    const uint32_t k = r / P.spp, s = r - k * P.spp;
    const uint32_t p = hit_idx[k];
    if (p >= P.npix) {  // slot left unwritten by a look-back that gave up
      o = P.cam.eye;
      dir = mk(0.f, 0.f, 1.f);
      tmax = 0.f;
      return;
    }
    di_segment(P, p, s, pt[p], o, dir);
    tmax = 0.9999f;
  }
  SHN_D void done(uint32_t r, const Hit& h) const { occ[r] = h.tri != kMiss ? 1 : 0; }
};

}  // namespace shn
