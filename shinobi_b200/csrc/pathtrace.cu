// Wavefront path tracer.
//
// The reference runs its path tracer as a persistent megakernel in which
// finished paths leave their lanes idle until the whole warp is done
// (src/Integrator/SimplePathTracer.hpp:65-241, src/Shinobi.h:152-230).  Here
// every bounce is three kernels over the live paths: the extension rays, the
// shading (which packs the survivors for the next bounce and lists the shadow
// rays), and the shadow rays.
//
// What bounds it: the incoherent rays' walk.  One kernel that traced a path's
// extension and shadow ray lane by lane ran at 3.5-4.7 of 32 lanes after the
// first bounce; the trace kernels of uniform grids run the flat engine at
// 17-26 lanes (4.2M-triangle heightfield, 1920 x 1080 x 16 paths, depth 4: 100 ->
// 51 ms, of which the shading is 2.6 ms).
//
// Semantics (restated by the oracle path for path):
//  * path g = sample * npix + (the pixel's number in 8x4-tile order); camera ray through the pixel with a
//    Philox jitter (RandomPixelSampler, src/Primitive/PixelSampler.h:56-70);
//  * at a hit: facing geometric normal n; next-event estimation to one
//    point of the parallelogram light (shadow segment, any hit, t < 0.9999
//    as in OcclusionRayBuffer, src/Engine/RayBuffers.h:156-169); Russian
//    roulette with continuation probability = albedo from depth rr_depth
//    on; cosine-weighted bounce (CosineHemisphereSampler,
//    src/Utils/HemisphereSamplers.hpp:54-72) in the frame {e1, n x e1, n};
//  * a miss adds throughput * background;
//  * each path writes its radiance to its own slot; the image is the
//    per-pixel mean over samples summed in sample order (deterministic).
// Random numbers: Philox4x32-10, counter (pixel, sample, depth, tag), key (seed, 0).
#include "internal.h"
#include "trace_coop.cuh"
#include "trace_flat.cuh"

namespace shn {

namespace {

constexpr int kPtBlock = 128;
constexpr uint32_t kTagJitter = 0x4A49u, kTagLight = 0x4C54u, kTagDir = 0x4449u;

struct PtView {
  CamView cam;
  uint32_t npix, spp, max_depth, rr_depth, seed;
  float albedo, offset;
  V3 lpos, le1, le2, lrad, lnrm, bg;
  float larea;
  const float4* stri;
  uint32_t snt;
};

// Path record: org, beta.x | dir, beta.y | beta.z, pixel, sample.  Its
// radiance accumulates in the path's slot.  Once shaded, a record whose path
// has a shadow ray holds that: origin, c.x | segment, c.y | c.z, pixel,
// sample, where c is added to the slot if the segment is free.
struct PathRec {
  float4 r0, r1, r2;
};

struct PtHit {
  float t;
  uint32_t tri;
};

// Per bounce: live paths, shadow rays, work counters of the two trace kernels.
struct PtCount {
  uint32_t live, shadow, work0, work1;
};

__global__ void k_pt_camera(PtView P, uint64_t g0, uint32_t count, PathRec* __restrict__ out, PtCount* cnt) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) cnt->live = count;
  if (k >= count) return;
  const uint64_t g = g0 + k;
  // path g = sample s, camera ray number g - s * npix, numbered by 8x4 pixel
  // tiles: a warp's 32 paths are one compact tile of one sample
  const uint32_t s = (uint32_t)(g / P.npix);
  const uint32_t p = tile_pixel(P.cam, (uint32_t)(g - (uint64_t)s * P.npix));
  const uint4 w = philox4x32(make_uint4(p, s, 0u, kTagJitter), P.seed, 0u);
  float ox = u01(w.x), oy = u01(w.y);
  const float tmp = (float)p / P.cam.resx;
  oy = truncf(tmp) + oy;
  ox = (tmp - truncf(tmp)) * P.cam.resx + ox;
  const CamView& c = P.cam;
  const V3 d = mk(c.tl.x + ox * c.sx.x + oy * c.sy.x, c.tl.y + ox * c.sx.y + oy * c.sy.y,
                  c.tl.z + ox * c.sx.z + oy * c.sy.z);
  PathRec r;
  r.r0 = make_float4(c.eye.x, c.eye.y, c.eye.z, 1.f);
  r.r1 = make_float4(d.x, d.y, d.z, 1.f);
  r.r2 = make_float4(1.f, __uint_as_float(p), __uint_as_float(s), 0.f);
  out[k] = r;
}

// Extension rays of the live paths.
struct PtExtend {
  const PathRec* paths;
  PtHit* hits;
  SHN_D void ray(uint32_t i, V3& o, V3& d, float& tmax) const {
    const float4 a = paths[i].r0, b = paths[i].r1;
    o = f4v(a);
    d = f4v(b);
    tmax = FLT_MAX;
  }
  SHN_D void done(uint32_t i, const Hit& h) const { hits[i] = PtHit{h.t, h.tri}; }
};

// Shadow rays: rays[k] is the record that holds the k-th.
struct PtShadow {
  const PathRec* paths;
  const uint32_t* rays;
  float4* slots;
  uint32_t npix;
  SHN_D void ray(uint32_t k, V3& o, V3& d, float& tmax) const {
    const PathRec& r = paths[rays[k]];
    o = f4v(r.r0);
    d = f4v(r.r1);
    tmax = 0.9999f;
  }
  SHN_D void done(uint32_t k, const Hit& h) const {
    if (h.tri != kMiss) return;
    const PathRec& r = paths[rays[k]];
    const float4 c = r.r2;
    float4* s = slots + ((uint64_t)__float_as_uint(c.z) * npix + __float_as_uint(c.y));
    const V3 L = add(f4v(*s), mk(r.r0.w, r.r1.w, c.x));
    *s = make_float4(L.x, L.y, L.z, 0.f);
  }
};

template <bool ANY, class Rays>
__global__ void __launch_bounds__(kPtBlock, kFlatBlocks) k_pt_flat(const __grid_constant__ GridView G, Rays R, const uint32_t* n,
                                                         uint32_t* counter) {
  __shared__ FlatWarp sm[kPtBlock / 32];
  flat_trace<ANY>(
      sm, FlatGrid{&G}, *n, false, counter,
      [&](uint32_t i, V3& o, V3& d, float& tmax, uint32_t&, uint32_t&) { R.ray(i, o, d, tmax); },
      [&](uint32_t i, const Hit& h, uint32_t) { R.done(i, h); });
}

// Two-level grids.  Camera rays are taken as packets.
template <bool ANY, bool PACKET, class Rays>
__global__ void __launch_bounds__(kPtBlock, ANY ? 6 : 8) k_pt_two_level(GridView G, Rays R, const uint32_t* n,
                                                              uint32_t* counter) {
  warp_trace<1, ANY, PACKET>(
      G, *n, counter, [&](uint32_t i, V3& o, V3& d, float& tmax) { R.ray(i, o, d, tmax); },
      [&](uint32_t i, const Hit& h, uint32_t, uint32_t) { R.done(i, h); });
}

// Shades the live paths: light sample, roulette, next direction.  Survivors are
// packed into `out` and shadow rays listed by blocks of paths, one addition to
// each count per block; the order of the blocks does not show in the image.
constexpr int kShadeBlock = 256;

__global__ void __launch_bounds__(kShadeBlock) k_pt_shade(PtView P, PathRec* __restrict__ paths,
                                                          const PtHit* __restrict__ hits, PathRec* __restrict__ out,
                                                          uint32_t* __restrict__ shadow, uint32_t depth,
                                                          PtCount* cnt, float4* __restrict__ slots) {
  __shared__ uint32_t s_live[kShadeBlock / 32], s_shadow[kShadeBlock / 32];
  const uint32_t n = cnt->live;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t i0 = blockIdx.x * kShadeBlock; i0 < n; i0 += gridDim.x * kShadeBlock) {
    const uint32_t i = i0 + threadIdx.x;
    bool live = false, casts = false;
    PathRec r, sh;
    if (i < n) {
      r = paths[i];
      const PtHit h = hits[i];
      const V3 org = f4v(r.r0), dir = f4v(r.r1);
      V3 beta = mk(r.r0.w, r.r1.w, r.r2.x);
      const uint32_t p = __float_as_uint(r.r2.y), s = __float_as_uint(r.r2.z);
      float4* slot = slots + ((uint64_t)s * P.npix + p);
      if (h.tri == kMiss) {
        const V3 L = add(depth ? f4v(*slot) : mk(0.f, 0.f, 0.f), mul(beta, P.bg));
        *slot = make_float4(L.x, L.y, L.z, 0.f);
      } else {
        if (depth == 0) *slot = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* rec = P.stri + 3 * (size_t)h.tri;
        const V3 v0 = f4v(__ldg(rec));
        const V3 v1 = f4v(__ldg(rec + 1));
        const V3 v2 = f4v(__ldg(rec + 2));
        const V3 e1 = sub(v1, v0);
        V3 nn = normalize(cross(e1, sub(v2, v0)));
        if (dot(nn, dir) > 0.f) nn = mk(-nn.x, -nn.y, -nn.z);
        const V3 hp = add(org, muls(dir, h.t));
        const V3 o = add(hp, muls(nn, P.offset));
        // next-event estimation
        const uint4 wl = philox4x32(make_uint4(p, s, depth, kTagLight), P.seed, 0u);
        const float lu = u01(wl.x), lv = u01(wl.y), urr = u01(wl.z);
        const V3 lp = add(add(P.lpos, muls(P.le1, lu)), muls(P.le2, lv));
        const V3 wv = sub(lp, o);
        const float d2 = dot(wv, wv);
        const V3 l = muls(wv, 1.0f / sqrtf(d2));
        const float cs = dot(nn, l);
        const float cl = -dot(P.lnrm, l);
        if (cs > 0.f && cl > 0.f) {
          const float f = ((((P.albedo * 0.31830988618379067f) * cs) * cl) * P.larea) / d2;
          const V3 c = muls(mul(beta, P.lrad), f);
          casts = true;
          sh.r0 = make_float4(o.x, o.y, o.z, c.x);
          sh.r1 = make_float4(wv.x, wv.y, wv.z, c.y);
          sh.r2 = make_float4(c.z, r.r2.y, r.r2.z, 0.f);
        }
        // continuation
        live = depth + 1 < P.max_depth;
        if (live && depth >= P.rr_depth) {
          if (urr < P.albedo) beta = muls(beta, 1.0f / P.albedo);
          else live = false;
        }
        if (live) {
          const uint4 wd = philox4x32(make_uint4(p, s, depth, kTagDir), P.seed, 0u);
          const float u1 = u01(wd.x), u2 = u01(wd.y);
          float sn, cn;
          sincos_2pi(u1, sn, cn);
          const float rr = sqrtf(1.f - u2);
          const float lx = sn * rr, ly = cn * rr, lz = sqrtf(u2);
          const V3 tx = normalize(e1);
          const V3 ty = cross(nn, tx);
          const V3 nd = mk(tx.x * lx + ty.x * ly + nn.x * lz, tx.y * lx + ty.y * ly + nn.y * lz,
                           tx.z * lx + ty.z * ly + nn.z * lz);
          beta = muls(beta, P.albedo);
          r.r0 = make_float4(o.x, o.y, o.z, beta.x);
          r.r1 = make_float4(nd.x, nd.y, nd.z, beta.y);
          r.r2.x = beta.z;
        }
      }
    }
    const uint32_t lm = __ballot_sync(0xFFFFFFFFu, live), cm = __ballot_sync(0xFFFFFFFFu, casts);
    if (lane == 0) {
      s_live[warp] = __popc(lm);
      s_shadow[warp] = __popc(cm);
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      uint32_t* w = threadIdx.x == 0 ? s_live : s_shadow;
      uint32_t sum = 0;
      for (int k = 0; k < kShadeBlock / 32; ++k) {
        const uint32_t v = w[k];
        w[k] = sum;
        sum += v;
      }
      const uint32_t at = sum ? atomicAdd(threadIdx.x == 0 ? &cnt[1].live : &cnt->shadow, sum) : 0u;
      for (int k = 0; k < kShadeBlock / 32; ++k) w[k] += at;
    }
    __syncthreads();
    if (live) out[s_live[warp] + __popc(lm & lt)] = r;
    if (casts) {
      paths[i] = sh;
      shadow[s_shadow[warp] + __popc(cm & lt)] = i;
    }
    __syncthreads();
  }
}

__global__ void k_pt_stats(const PtCount* cnt, uint32_t depth, uint32_t* stats) {
  uint32_t shadow = 0;
  for (uint32_t d = 0; d < depth; ++d) {
    stats[d] += cnt[d].live;
    shadow += cnt[d].shadow;
  }
  stats[depth] += shadow;
}

__global__ void k_pt_resolve(const float4* __restrict__ slots, uint32_t npix, uint32_t spp,
                             float* __restrict__ img) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  float r = 0.f, g = 0.f, b = 0.f;
  for (uint32_t s = 0; s < spp; ++s) {
    const float4 v = slots[(uint64_t)s * npix + p];
    r += v.x;
    g += v.y;
    b += v.z;
  }
  img[3 * (size_t)p] = r / (float)spp;
  img[3 * (size_t)p + 1] = g / (float)spp;
  img[3 * (size_t)p + 2] = b / (float)spp;
}

template <class K>
int pt_blocks(K kernel, int num_sms) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPtBlock, 0);
  return std::max(1, per_sm) * num_sms;
}

// Extension (Rays = PtExtend) or shadow rays of one bounce.
template <bool ANY, class Rays>
void launch_rays(const GridView& G, const Rays& R, bool camera, const uint32_t* n, uint32_t* counter, uint32_t most,
                 int num_sms, cudaStream_t st) {
  const int need = (int)std::min<uint32_t>((most + kPtBlock / 32 - 1) / (kPtBlock / 32), 1u << 20);
  if (G.kind == SHN_GRID_UNIFORM) {
    static const int blocks = pt_blocks(k_pt_flat<ANY, Rays>, num_sms);
    k_pt_flat<ANY, Rays><<<std::min(blocks, need), kPtBlock, 0, st>>>(G, R, n, counter);
  } else if (!ANY && camera) {
    static const int blocks = pt_blocks(k_pt_two_level<ANY, true, Rays>, num_sms);
    k_pt_two_level<ANY, true, Rays><<<blocks, kPtBlock, 0, st>>>(G, R, n, counter);
  } else {
    static const int blocks = pt_blocks(k_pt_two_level<ANY, false, Rays>, num_sms);
    k_pt_two_level<ANY, false, Rays><<<blocks, kPtBlock, 0, st>>>(G, R, n, counter);
  }
}

}  // namespace

}  // namespace shn

using namespace shn;

extern "C" {

void shn_pt_params_default(shn_pt_params* p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->spp = 16;
  p->max_depth = 4;
  p->rr_depth = 2;
  p->albedo = 0.7f;
  const float pos[3] = {0.3f, 0.3f, 1.0f}, e1[3] = {0.f, 0.4f, 0.f}, e2[3] = {0.4f, 0.f, 0.f};
  const float rad[3] = {20.f, 20.f, 20.f}, bg[3] = {0.15f, 0.2f, 0.3f};
  memcpy(p->light_pos, pos, 12);
  memcpy(p->light_e1, e1, 12);
  memcpy(p->light_e2, e2, 12);
  memcpy(p->light_radiance, rad, 12);
  memcpy(p->background, bg, 12);
  p->offset = 1e-4f;
  p->seed = 2;
}

shn_status shn_pt_render(const shn_grid* g, const shn_scene* s, const shn_camera* cam,
                         const shn_pt_params* prm, float* d_image, uint32_t* d_stats, void* stream) {
  if (!g || !s || !cam || !prm || !d_image || prm->spp == 0 || prm->max_depth == 0) return SHN_ERR_INVALID;
  if (!g->built) return set_error(g->ctx, SHN_ERR_NOT_BUILT, "grid not built");
  grid_fence(g, (cudaStream_t)stream);
  if (!(prm->albedo > 0.f && prm->albedo <= 1.f)) return set_error(g->ctx, SHN_ERR_INVALID, "albedo must be in (0,1]");
  const uint64_t npix = (uint64_t)cam->res_x * cam->res_y;
  if (npix == 0) return SHN_OK;
  if (npix > (1u << 24)) return set_error(g->ctx, SHN_ERR_INVALID, "more than 2^24 pixels");
  const uint64_t total = npix * prm->spp;
  cudaStream_t st = (cudaStream_t)stream;
  shn_ctx* ctx = g->ctx;

  PtView P;
  P.cam = make_camera(cam);
  P.npix = (uint32_t)npix;
  P.spp = prm->spp;
  P.max_depth = prm->max_depth;
  P.rr_depth = prm->rr_depth;
  P.seed = prm->seed;
  P.albedo = prm->albedo;
  P.offset = prm->offset;
  P.lpos = mk(prm->light_pos[0], prm->light_pos[1], prm->light_pos[2]);
  P.le1 = mk(prm->light_e1[0], prm->light_e1[1], prm->light_e1[2]);
  P.le2 = mk(prm->light_e2[0], prm->light_e2[1], prm->light_e2[2]);
  P.lrad = mk(prm->light_radiance[0], prm->light_radiance[1], prm->light_radiance[2]);
  P.bg = mk(prm->background[0], prm->background[1], prm->background[2]);
  const V3 ln = cross(P.le1, P.le2);
  P.larea = sqrtf(dot(ln, ln));
  P.lnrm = normalize(ln);
  P.stri = s->tri;
  P.snt = s->nt;
  const GridView G = view_of(g);

  // Waves of at most kWave paths bound the state memory (108 bytes per path,
  // and 16 per sample of the image).
  const uint64_t kWave = 1ull << 23;
  const uint32_t wave = (uint32_t)std::min<uint64_t>(total, kWave);
  size_t bytes = 0;
  const auto part = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) & ~(size_t)255;
    return at;
  };
  const size_t bCnt = ((size_t)prm->max_depth + 1) * sizeof(PtCount);
  const size_t oa = part((size_t)wave * sizeof(PathRec)), ob = part((size_t)wave * sizeof(PathRec)),
               oh = part((size_t)wave * sizeof(PtHit)), os = part((size_t)wave * 4), ol = part((size_t)total * 16),
               oc = part(bCnt);
  char* mem = nullptr;
  cudaError_t e = dev_alloc(ctx, (void**)&mem, bytes, st);
  if (e != cudaSuccess)
    return set_error(ctx, e == cudaErrorNotPermitted ? SHN_ERR_BUDGET : SHN_ERR_OOM, "path tracer state");
  float4* slots = (float4*)(mem + ol);
  PtHit* hits = (PtHit*)(mem + oh);
  uint32_t* shadow = (uint32_t*)(mem + os);
  PtCount* cnt = (PtCount*)(mem + oc);
  if (d_stats) cudaMemsetAsync(d_stats, 0, ((size_t)prm->max_depth + 1) * 4, st);
  for (uint64_t g0 = 0; g0 < total; g0 += wave) {
    const uint32_t count = (uint32_t)std::min<uint64_t>(wave, total - g0);
    PathRec* cur = (PathRec*)(mem + oa);
    PathRec* nxt = (PathRec*)(mem + ob);
    const int shade_blocks = (int)std::min<uint32_t>((count + kShadeBlock - 1) / kShadeBlock, (uint32_t)ctx->num_sms * 8u);
    cudaMemsetAsync(cnt, 0, bCnt, st);
    k_pt_camera<<<(count + 255) / 256, 256, 0, st>>>(P, g0, count, cur, cnt);
    for (uint32_t d = 0; d < prm->max_depth; ++d) {
      PtCount* c = cnt + d;
      launch_rays<false>(G, PtExtend{cur, hits}, d == 0, &c->live, &c->work0, count, ctx->num_sms, st);
      k_pt_shade<<<shade_blocks, kShadeBlock, 0, st>>>(P, cur, hits, nxt, shadow, d, c, slots);
      launch_rays<true>(G, PtShadow{cur, shadow, slots, P.npix}, false, &c->shadow, &c->work1, count, ctx->num_sms, st);
      std::swap(cur, nxt);
    }
    if (d_stats) k_pt_stats<<<1, 1, 0, st>>>(cnt, prm->max_depth, d_stats);
  }
  k_pt_resolve<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(slots, (uint32_t)npix,
                                                               prm->spp, d_image);
  dev_free(ctx, mem, bytes, st);
  e = cudaGetLastError();
  return e == cudaSuccess ? SHN_OK : cuda_status(ctx, e, "pt_render");
}

}  // extern "C"
