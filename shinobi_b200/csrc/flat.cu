// Trace kernels of uniform grids on the flat engine: rays from arrays, camera
// rays, and the any-hit rays made from a frame's primary hits.
#include "internal.h"
#include "rays.cuh"
#include "trace_flat.cuh"

namespace shn {

namespace {

template <bool ANY, int K, bool COH>
__global__ void __launch_bounds__(kCoopBlock, K == kFlatAhead ? kFlatBlocks
                                              : ANY || COH    ? kFlatBlocksFew
                                                              : kFlatBlocksAlone)
    k_flat_rays(const __grid_constant__ GridView G, RaysView R, uint32_t n, uint32_t* counter, uint32_t* otri,
                float* ot, float* ou, float* ov, uint8_t* occ) {
  __shared__ FlatWarpOf<K> sm[kCoopBlock / 32];
  flat_trace<ANY, false, false, COH>(
      sm, FlatGrid{&G}, n, ou || ov, counter,
      [&](uint32_t i, V3& o, V3& d, float& tmax, uint32_t&, uint32_t&) {
        R.ray(i, o, d, tmax);
      },
      [&](uint32_t i, const Hit& h, uint32_t) {
        if (ANY) {
          occ[i] = h.tri != kMiss ? 1 : 0;
        } else {
          otri[i] = h.tri;
          ot[i] = h.t;
          if (ou) ou[i] = h.u;
          if (ov) ov[i] = h.v;
        }
      });
}

template <int K>
__global__ void __launch_bounds__(kCoopBlock, K == kFlatAhead ? kFlatBlocks : kFlatBlocksFew)
    k_flat_camera(const __grid_constant__ GridView G, CamView cam, uint32_t image_id, uint32_t n, uint32_t* counter,
                  uint32_t* otri, float* ot, float* ou, float* ov) {
  __shared__ FlatWarpOf<K> sm[kCoopBlock / 32];
  flat_trace<false, false, true>(
      sm, FlatGrid{&G}, n, ou || ov, counter,
      [&](uint32_t i, V3& o, V3& d, float& tmax, uint32_t&, uint32_t&) {
        o = cam.eye;
        d = primary_dir(cam, tile_pixel(cam, i), image_id);
        tmax = FLT_MAX;
      },
      [&](uint32_t r, const Hit& h, uint32_t) {
        const uint32_t i = tile_pixel(cam, r);
        otri[i] = h.tri;
        ot[i] = h.t;
        if (ou) ou[i] = h.u;
        if (ov) ov[i] = h.v;
      });
}

template <class Rays, int K>
__global__ void __launch_bounds__(kCoopBlock, K == kFlatAhead ? kFlatBlocks : kFlatBlocksFew)
    k_flat_from_hits(const __grid_constant__ GridView G, const __grid_constant__ Rays R, const uint32_t* d_m,
                     uint32_t spp, uint32_t* counter) {
  __shared__ FlatWarpOf<K> sm[kCoopBlock / 32];
  flat_trace<true>(
      sm, FlatGrid{&G}, (*d_m) * spp, false, counter,
      [&](uint32_t i, V3& o, V3& d, float& tmax, uint32_t&, uint32_t&) { R.ray(i, o, d, tmax); },
      [&](uint32_t i, const Hit& h, uint32_t) { R.done(i, h); });
}

// Persistent blocks, no more than one warp per ray needs.
template <auto KERNEL>
int flat_blocks(int num_sms, uint64_t n) {
  static const int per_sm = [] {
    int v = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, KERNEL, kCoopBlock, 0);
    return std::max(1, v);
  }();
  const uint64_t need = (n + kCoopBlock / 32 - 1) / (kCoopBlock / 32);
  return (int)std::min<uint64_t>((uint64_t)per_sm * num_sms, need);
}

}  // namespace

template <bool ANY, int K, bool COH = false>
static void flat_rays(const GridView& G, const RaysView& rays, uint32_t n, uint32_t* counter, const shn_hits& hits,
                      uint8_t* occ, int num_sms, cudaStream_t st) {
  k_flat_rays<ANY, K, COH><<<flat_blocks<k_flat_rays<ANY, K, COH>>(num_sms, n), kCoopBlock, 0, st>>>(
      G, rays, n, counter, hits.tri, hits.t, hits.u, hits.v, occ);
}

void launch_flat_closest(const GridView& G, const RaysView& rays, uint32_t n, uint32_t* counter, const shn_hits& hits,
                         int num_sms, cudaStream_t st) {
  if (n <= kFlatAlone) flat_rays<false, kFlatAheadFew>(G, rays, n, counter, hits, nullptr, num_sms, st);
  else if (n < kFlatFew) flat_rays<false, kFlatAheadFew, true>(G, rays, n, counter, hits, nullptr, num_sms, st);
  else flat_rays<false, kFlatAhead, true>(G, rays, n, counter, hits, nullptr, num_sms, st);
}

void launch_flat_any(const GridView& G, const RaysView& rays, uint32_t n, uint32_t* counter, uint8_t* occ, int num_sms,
                     cudaStream_t st) {
  if (n < kFlatFew) flat_rays<true, kFlatAheadFew>(G, rays, n, counter, shn_hits{}, occ, num_sms, st);
  else flat_rays<true, kFlatAhead>(G, rays, n, counter, shn_hits{}, occ, num_sms, st);
}

template <int K>
static void flat_camera(const GridView& G, const CamView& cam, uint32_t image_id, uint32_t n, uint32_t* counter,
                        const shn_hits& hits, int num_sms, cudaStream_t st) {
  k_flat_camera<K><<<flat_blocks<k_flat_camera<K>>(num_sms, n), kCoopBlock, 0, st>>>(
      G, cam, image_id, n, counter, hits.tri, hits.t, hits.u, hits.v);
}

void launch_flat_camera(const GridView& G, const CamView& cam, uint32_t image_id, uint32_t n, uint32_t* counter,
                        const shn_hits& hits, int num_sms, cudaStream_t st) {
  if (n < kFlatFew) flat_camera<kFlatAheadFew>(G, cam, image_id, n, counter, hits, num_sms, st);
  else flat_camera<kFlatAhead>(G, cam, image_id, n, counter, hits, num_sms, st);
}

template <class Rays, int K>
static void from_hits_k(const GridView& G, const Rays& R, const uint32_t* d_m, uint32_t spp, uint32_t* counter,
                        uint64_t most, int num_sms, cudaStream_t st) {
  k_flat_from_hits<Rays, K><<<flat_blocks<k_flat_from_hits<Rays, K>>(num_sms, most), kCoopBlock, 0, st>>>(G, R, d_m, spp,
                                                                                                     counter);
}

template <class Rays>
static void from_hits(const GridView& G, const Rays& R, const uint32_t* d_m, uint32_t spp, uint32_t* counter,
                      uint64_t most, int num_sms, cudaStream_t st) {
  if (most < kFlatFew) from_hits_k<Rays, kFlatAheadFew>(G, R, d_m, spp, counter, most, num_sms, st);
  else from_hits_k<Rays, kFlatAhead>(G, R, d_m, spp, counter, most, num_sms, st);
}

void launch_flat_from_hits(const GridView& G, const AoRays& R, const uint32_t* d_m, uint32_t spp, uint32_t* counter,
                           uint64_t most, int num_sms, cudaStream_t st) {
  from_hits(G, R, d_m, spp, counter, most, num_sms, st);
}

void launch_flat_from_hits(const GridView& G, const DiRays& R, const uint32_t* d_m, uint32_t spp, uint32_t* counter,
                           uint64_t most, int num_sms, cudaStream_t st) {
  from_hits(G, R, d_m, spp, counter, most, num_sms, st);
}

}  // namespace shn
