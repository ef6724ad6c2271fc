// Traversal engine for uniform grids.
//
// What bounds it: a ray walks ~100 cells, tests a handful of references in
// some of them, and neighbouring lanes do so at different places.  With one
// loop per lane (walk until a range is found, then test all of it) the warp
// waits for its slowest lane in both loops: 3.5 to 8 of 32 lanes were active
// per instruction on random rays, path-tracer bounces and soup frames.  Here
// the work of a warp is laid flat:
//  * setup: the warp takes 32 rays, writes the results of those that miss the
//    grid and gives the others to idle lanes;
//  * walk: every lane steps through its next kFlatAhead cells, whose ranges
//    are loaded together;
//  * test: the references of all lanes' ranges are numbered through and dealt
//    to the 32 lanes, whoever owns the ray (its origin and shear are read from
//    shared memory); a ray's least (t, cell, triangle id) is kept by atomicMin.
// 16 to 26 lanes are active per instruction, and a third of the instructions
// are left on random rays.  Measured against one loop per lane (B200): 4.0M
// random rays on a 1M-triangle soup 1.95 -> 0.82 ms; a 640 x 400 camera on a
// 200,000-triangle soup 0.33 -> 0.15 ms; C2-sized path tracing (4.2M triangles,
// 1920 x 1080 x 16, depth 4) 100 -> 52 ms; 64 scenes' random rays 1.94 -> 0.76 ms.
// What is left is latency: the random loads miss L2 (35-55 % hits), at 45-65 %
// issue.  Sizes tried: windows of 4, 6 and 8 cells (0.98, 0.93, 0.94 ms on the
// random rays, 55.9, 53.8, 53.2 ms on the path tracer), 6 to 8 blocks per SM
// (0.93, 0.92 and 0.97 ms; 53.8, 50.9 and 56 ms).  Shared memory beyond ~160 KB
// per SM costs up to 1.6x: L1 then has too few lines for the loads in flight.
//
// Crowded cells (soups at a tenth to a 2500th of the usual resolution, a ball
// of 236,000 triangles in 5 x 5 x 5 cells of a larger grid) against one loop per
// lane with long ranges tested by the warp: random rays 0.2 to 1.0 of its time,
// camera rays 0.6 to 1.02 up to ~50 references per cell and on the ball, 1.14 and
// 1.27 at ~160 and ~700 (its warps hold one packet of 32 rays at a time).
//
// The results are those of warp_trace (trace_coop.cuh), bit for bit: the cells
// are the same in the same order (see flat_enter and the end of the window), a
// range's winner is the least (t, triangle id) below the bound from earlier
// cells, and every float operation on the way is the same.
#pragma once
#include "trace_coop.cuh"

namespace shn {

// Finished lanes wait for this many before their results are written and
// their places refilled.
constexpr int kFlatRefill = 8;

// Blocks per SM of the kernels that run the engine.
constexpr int kFlatBlocks = 7;

// Groups of 32 references whose triangle ids are loaded together.
constexpr int kFlatGroups = 2;

// Cells a lane walks per step of the warp, their ranges in flight together.
// Calls of fewer rays than the device has lanes for (148 SMs x 7 blocks x 128)
// wait for one ray's chain of windows and take longer ones: 200,000-triangle
// soup, 1,021 / 16,000 / 64,000 / 130,000 rays 56 -> 50, 117 -> 86, 173 -> 159 and
// 186 -> 170 us; from 200,000 rays on the shorter ones with a block more per SM
// are as fast or faster (4.0M rays: 0.92 against 0.94 ms).  The single-grid
// calls choose by this; bounces, batches and server launches, whose ray counts
// vary, take kFlatAhead.
constexpr int kFlatAhead = 6, kFlatAheadFew = 8;
constexpr uint32_t kFlatFew = 1u << 17;

// Up to this many rays there are one or two to a warp: no neighbours to run side
// by side with (see COH), and fewer blocks per SM, whose registers keep the chain
// of windows free of spills (300 to 4,000 rays on a 65,536-triangle soup 2 us of
// 40 to 48 less than at 6 blocks; 3 blocks the same, 5 a microsecond more).
constexpr uint32_t kFlatAlone = 1u << 12;
constexpr int kFlatBlocksAlone = 4, kFlatBlocksFew = 6;

// Shared memory of one warp.  The rays live here, not in registers: the walk
// loads and stores what it needs, so that the tests have the registers.  Every
// kilobyte less leaves L1 room for lines in flight.
template <int K>
struct FlatWarpOf {
  float4 a[32];  // org, Sx
  float4 b[32];  // Sy, Sz, axis permutation (6 bits) and cells of the window that count << 8, bound (the best t so far)
  float4 c[32];  // tMax, cell
  float4 d[32];  // tDelta, direction signs (3 bits), any-hit flag, scene
  uint2 e[32];   // steps left in x and y | in z, cells ahead known to be empty
  uint32_t rid[32], best[32];
  float far_t[32];  // t of a hit that the walk may not get to (its triangle is in best)
  unsigned long long key[32];         // least (t, cell of the window, triangle id) of the ranges under test
  uint2 own[32 * K + 32];    // range under test: lane and cell | first number << 8, first reference - first number
  uint32_t wait[32];                  // rays that meet the grid and have no lane yet
  uint32_t general[96];               // < 32 when rays are taken, and at most 32 + 31 more on their way
};

using FlatWarp = FlatWarpOf<kFlatAhead>;

// Key of a candidate: t (positive: 31 bits), cell of the window (3 bits),
// triangle id (30 bits).
constexpr uint32_t kFlatMaxTris = 1u << 30;
static_assert(kFlatAhead <= 8 && kFlatAheadFew <= 8, "three bits of the key");
SHN_D unsigned long long flat_key(float t, uint32_t q, uint32_t id) {
  return ((unsigned long long)__float_as_uint(t) << 33) | ((unsigned long long)q << 30) | id;
}
SHN_D float flat_key_t(unsigned long long k) { return __uint_as_float((uint32_t)(k >> 33)); }

// Key of an any-hit ray among closest-hit ones: the first of its candidates in
// the order of the cells and their references (fewer than 2^30).  A range's
// candidate is that of warp_trace: the first hit of a short range, and of a
// long one the nearest hit (t, triangle id) among the first 32 references that
// hold any.
SHN_D unsigned long long flat_key_any(float t, uint32_t q, uint32_t ref) {
  return ((unsigned long long)q << 61) | ((unsigned long long)ref << 31) | __float_as_uint(t);
}

enum : int { FLAT_MISS = 0, FLAT_RAY = 1, FLAT_GENERAL = 2 };

// Ray setup of lane_init<0>, with the walk in integers: the cell's index, and
// per axis the number of steps until the coordinate reaches -1 or res.
//  * A start cell one outside the entry side (rounding of the entry point)
//    looks up the clamped cell, steps onto that same cell and tests it again
//    to no effect; starting on the clamped cell with tMax advanced by the same
//    addition visits the same cells under the same bounds.
//  * Every start further out, and every NaN, is left to the general walk.
// flat_enter decides; flat_queue writes the rest of a FLAT_RAY's state.
SHN_D int flat_enter(const Geom& g, V3 org, V3 dir, float tmax, V3& cell) {
  if (!(tmax > 0.f)) return FLAT_MISS;
  const V3 rcp = divv(mk(1.f, 1.f, 1.f), dir);
  const V3 t1 = mul(sub(g.gmin, org), rcp);
  V3 t2 = mul(sub(g.gmax, org), rcp);
  const V3 tmn = vmin(t1, t2);
  t2 = vmax(t1, t2);
  const float tEntry = fmaxf(fmaxf(tmn.x, tmn.y), tmn.z);
  const float tExit = fminf(fminf(t2.x, t2.y), t2.z);
  if (tExit <= tEntry || tExit < 0.f) return FLAT_MISS;
  const float te = tEntry + kEps;
  const V3 entry = (tEntry >= 0.f) ? add(org, divv(mk(te, te, te), rcp)) : org;
  cell = mul(sub(entry, g.gmin), g.rcpTrav);
  cell = mk(floorf(cell.x), floorf(cell.y), floorf(cell.z));
  const bool valid = (cell.x != (rcp.x > 0.f ? g.resf.x : -1.f)) && (cell.y != (rcp.y > 0.f ? g.resf.y : -1.f)) &&
                     (cell.z != (rcp.z > 0.f ? g.resf.z : -1.f));
  if (!valid) return FLAT_MISS;
  const bool in = cell.x >= -1.f && cell.x <= g.resf.x && cell.y >= -1.f && cell.y <= g.resf.y && cell.z >= -1.f &&
                  cell.z <= g.resf.z;
  // tMax and tDelta are numbers, and finite unless the direction component is 0
  const V3 m = mul(sub(add(mul(cell, g.cs), g.gmin), org), rcp);
  const V3 d = mul(g.cs, rcp);
  return in && m.x == m.x && m.y == m.y && m.z == m.z && d.x == d.x && d.y == d.y && d.z == d.z ? FLAT_RAY
                                                                                               : FLAT_GENERAL;
}

// One axis: tMax, tDelta, the start index and the steps left.
SHN_D void flat_axis(float gmin, float cs, int res, float org, float rcp, float cell, float& tm, float& dl, int& i,
                     uint32_t& left) {
  const bool up = rcp > 0.f;
  tm = (((cell + (up ? 1.f : 0.f)) * cs + gmin) - org) * rcp;
  dl = cs * fabsf(rcp);
  i = (int)cell;
  if (i == (up ? -1 : res)) {
    i += up ? 1 : -1;
    tm += dl;
  }
  left = (uint32_t)(up ? res - 1 - i : i);
}

template <int K>
SHN_D void flat_queue(const Geom& g, uint32_t cell0, V3 org, V3 dir, float tmax, V3 cell, uint32_t rid, uint32_t scene,
                      uint32_t anyhit, FlatWarpOf<K>& Q, uint32_t k) {
  const V3 rcp = divv(mk(1.f, 1.f, 1.f), dir);
  const RayWT w = wt_setup(org, dir);
  const uint32_t perm = (uint32_t)w.kx | ((uint32_t)w.ky << 2) | ((uint32_t)w.kz << 4);
  Q.a[k] = make_float4(org.x, org.y, org.z, w.Sx);
  Q.b[k] = make_float4(w.Sy, w.Sz, __uint_as_float(perm | (uint32_t)K << 8), tmax);
  V3 tm, dl;
  int ix, iy, iz;
  uint32_t lx, ly, lz;
  flat_axis(g.gmin.x, g.cs.x, g.res[0], org.x, rcp.x, cell.x, tm.x, dl.x, ix, lx);
  flat_axis(g.gmin.y, g.cs.y, g.res[1], org.y, rcp.y, cell.y, tm.y, dl.y, iy, ly);
  flat_axis(g.gmin.z, g.cs.z, g.res[2], org.z, rcp.z, cell.z, tm.z, dl.z, iz, lz);
  const uint32_t idx = cell0 + (uint32_t)ix + (uint32_t)iy * (uint32_t)g.res[0] + (uint32_t)iz * (uint32_t)g.res[0] * (uint32_t)g.res[1];
  const uint32_t signs = (rcp.x > 0.f ? 1u : 0u) | (rcp.y > 0.f ? 2u : 0u) | (rcp.z > 0.f ? 4u : 0u);
  Q.c[k] = make_float4(tm.x, tm.y, tm.z, __uint_as_float(idx));
  Q.d[k] = make_float4(dl.x, dl.y, dl.z, __uint_as_float(signs | (anyhit ? 8u : 0u) | scene << 4));
  Q.e[k] = make_uint2(lx | ly << 16, lz);
  Q.rid[k] = rid;
  Q.best[k] = kMiss;
}

// A ray whose walk does not start plainly: the general state machine, alone.
template <bool ANY>
__device__ __noinline__ void flat_general(const Geom& g, const uint2* cells, const Refs& R, V3 org, V3 dir, float tmax,
                                          uint32_t anyhit, Hit& h) {
  Lane L;
  uint32_t steps = 0, tests = 0;
  lane_init<0>(g, L, org, dir, tmax);
  L.anyhit = anyhit;
  while (lane_advance<0, ANY>(g, cells, nullptr, L, steps)) {
    if (!ANY && L.anyhit && L.e - L.b > kCoopThreshold) {  // the candidate of a long range, see flat_key_any
      const uint32_t end = L.e;
      L.anyhit = 0;
      for (; L.b < end && L.best == kMiss; L.b = L.e) {
        L.e = min(end, L.b + 32u);
        lane_range<false, true>(R, L, tests);
      }
      L.anyhit = 1;
    } else {
      lane_range<ANY, true>(R, L, tests);
    }
  }
  lane_result(R, L, h);
}

// The watertight test without its double-precision fallback: 0 = no hit below
// tbest, 1 = hit at t, 2 = an edge function is exactly zero (the fallback
// decides).  The operations are those of wt_test_t<3, 3, 3>.
SHN_D int flat_test(float4 a, float4 b, float4 p0, float4 p1, float4 p2, float& t) {
  const uint32_t perm = __float_as_uint(b.z);
  const uint32_t kx = perm & 3u, ky = (perm >> 2) & 3u, kz = (perm >> 4) & 3u;
  const V3 o = f4v(a), A = sub(f4v(p0), o), B = sub(f4v(p1), o), C = sub(f4v(p2), o);
  const float Akz = sel((int)kz, A), Bkz = sel((int)kz, B), Ckz = sel((int)kz, C);
  const float Ax = __fmaf_rn(-a.w, Akz, sel((int)kx, A)), Ay = __fmaf_rn(-b.x, Akz, sel((int)ky, A));
  const float Bx = __fmaf_rn(-a.w, Bkz, sel((int)kx, B)), By = __fmaf_rn(-b.x, Bkz, sel((int)ky, B));
  const float Cx = __fmaf_rn(-a.w, Ckz, sel((int)kx, C)), Cy = __fmaf_rn(-b.x, Ckz, sel((int)ky, C));
  const float U = __fmaf_rn(Cx, By, -(Cy * Bx));
  const float V = __fmaf_rn(Ax, Cy, -(Ay * Cx));
  const float W = __fmaf_rn(Bx, Ay, -(By * Ax));
  if (fminf(fminf(fabsf(U), fabsf(V)), fabsf(W)) == 0.f) return 2;
  if (fminf(fminf(U, V), W) < 0.f && fmaxf(fmaxf(U, V), W) > 0.f) return 0;
  const float det = U + V + W;
  if (det == 0.f) return 0;
  const float T = __fmaf_rn(W, b.y * Ckz, __fmaf_rn(V, b.y * Bkz, U * (b.y * Akz)));
  t = T / det;
  return t > kEps && t < b.w ? 1 : 0;
}

// Ranges of more references than this are long: loaded once for all of the
// warp's rays that wait on them, cell after cell of a ray, so that a hit ends
// the walk there.  kCoopThreshold where rays may be any-hit one by one (their
// answer depends on it, see flat_key_any), for camera rays, and for other
// coherent ones while most neighbours wait on the same range: camera rays in
// cells of ~54 references 645 us dealt out, 231 us together, but path-traced
// images of the 4.2M-triangle heightfield 51.8 ms dealt out, 66 ms as long
// ranges.  A ray that meets a range of 2^24 is left to the general walk.
constexpr uint32_t kFlatLong = 63;
constexpr uint32_t kFlatHuge = 1u << 24;

// Tests the long range [b, b + len) against the rays of the lanes in `rays`,
// which wait on it in the cells that `cell` (a lane's own) holds: each lane
// loads one reference of every 32 and tests it against each ray.  KX, KY, KZ:
// the rays' axis permutation, or 3 each where they may differ.  SAME: the rays
// have one origin, and the vertices are translated once.
template <int KX, int KY, int KZ, bool SAME, bool ANY, bool MIXED, int K>
SHN_D void flat_long_p(FlatWarpOf<K>& W, const Refs& R, uint32_t rays, uint32_t b, uint32_t len, uint32_t cell) {
  const uint32_t lane = threadIdx.x & 31;
  const V3 o0 = f4v(W.a[__ffs(rays) - 1]);
  uint32_t next = lane < len ? __ldg(R.ridx + (b + lane)) : 0u;
  for (uint32_t i0 = 0; i0 < len && rays; i0 += 32u) {
    const bool in = i0 + lane < len;
    const uint32_t id = next;
    if (i0 + 32u + lane < len) next = __ldg(R.ridx + (b + i0 + 32u + lane));
    const float4* rec = R.rec + 3 * (size_t)id;
    V3 p0 = f4v(__ldg(rec)), p1 = f4v(__ldg(rec + 1)), p2 = f4v(__ldg(rec + 2));
    if (SAME) {
      p0 = sub(p0, o0);
      p1 = sub(p1, o0);
      p2 = sub(p2, o0);
    }
    for (uint32_t m = rays; m; m &= m - 1) {
      const int r = __ffs(m) - 1;
      const float4 A = W.a[r], B = W.b[r];
      const V3 o = f4v(A);
      // below the ray's bound, or as near as its best hit so far
      float bound = B.w;
      if (!ANY && !MIXED) {
        const unsigned long long k = W.key[r];
        if (k != ~0ull) bound = next_up(flat_key_t(k));
      }
      float t;
      const uint32_t perm = __float_as_uint(B.z);
      const bool hit = in && (SAME ? wt_test_t<KX, KY, KZ>(p0, p1, p2, A.w, B.x, B.y, kEps, bound, t, perm)
                                   : wt_test_t<KX, KY, KZ>(sub(p0, o), sub(p1, o), sub(p2, o), A.w, B.x, B.y, kEps,
                                                           bound, t, perm));
      const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
      if (!hits) continue;
      if (ANY) {
        rays &= ~(1u << r);
        if (lane == 0) W.key[r] = 0ull;
        continue;
      }
      const uint32_t q = __shfl_sync(0xFFFFFFFFu, cell, r);
      if (MIXED && (__float_as_uint(W.d[r].w) & 8u)) {
        // t is positive: its bits are in its order; references are in that of the ids
        const uint32_t tb = hit ? __float_as_uint(t) : 0xFFFFFFFFu;
        const uint32_t least = __ballot_sync(0xFFFFFFFFu, tb == __reduce_min_sync(0xFFFFFFFFu, tb));
        if (lane == __ffs(least) - 1) atomicMin(&W.key[r], flat_key_any(t, q, b + i0 + lane));
        rays &= ~(1u << r);
      } else if (hit) {
        atomicMin(&W.key[r], flat_key(t, q, id));
      }
    }
    __syncwarp();
  }
}

// The long ranges: the lane's n ones stand from entry `at` on, counted from the
// end of W.own, in the order of its cells (lane and cell | length << 8, first
// reference).  Every lane waits on the first one that can still matter, and
// lanes on the same one test it together.  COH: only those whose axes are
// permuted alike, a compile-time constant of the test: camera rays in cells of
// ~700 references 1071 -> 674 us, and where rays are not coherent the copies cost
// 8 % (4.0M random rays 739 -> 803 us).
template <bool ANY, bool MIXED, bool SAME, bool COH, int K, class Acc>
SHN_D void flat_long(FlatWarpOf<K>& W, const Acc& acc, uint32_t at, uint32_t n, const float (&ex)[K]) {
  const int lane = threadIdx.x & 31;
  const uint32_t bits = MIXED && n ? __float_as_uint(W.d[lane].w) : 0u;
  const uint32_t what = COH ? (n ? __float_as_uint(W.b[lane].z) & 63u : 0u) : bits >> 4;  // axes, or the scene
  const uint32_t cells = n ? __float_as_uint(W.b[lane].z) >> 8 : 0u;
  while (true) {
    uint2 mine = make_uint2(0u, 0u);
    if (n) {
      mine = W.own[32 * K + 31 - at];
      const unsigned long long k = W.key[lane];
      const uint32_t q = (mine.x >> 5) & 7u;
      if (q >= cells) n = 0;
      if (k != ~0ull) {
        // a hit before the entry of the range's cell ends the walk before it
        float entry = -INFINITY;
#pragma unroll
        for (int i = 0; i + 1 < K; ++i)
          if (q == (uint32_t)i + 1u) entry = ex[i];
        if (ANY || (MIXED && (bits & 8u) ? (uint32_t)(k >> 61) < q : !(flat_key_t(k) > entry))) n = 0;
      }
    }
    const uint32_t todo = __ballot_sync(0xFFFFFFFFu, n != 0u);
    if (!todo) break;
    const int j = __ffs(todo) - 1;
    const uint32_t b = __shfl_sync(0xFFFFFFFFu, mine.y, j), len = __shfl_sync(0xFFFFFFFFu, mine.x, j) >> 8;
    const uint32_t like = __shfl_sync(0xFFFFFFFFu, what, j);
    const Refs R = acc.refs(MIXED ? like : 0u);
    const uint32_t rays = todo & __ballot_sync(0xFFFFFFFFu, mine.y == b && (mine.x >> 8) == len && what == like);
    const uint32_t cell = (mine.x >> 5) & 7u;
    if constexpr (COH) {
      switch (like) {
        case (1u | 2u << 2 | 0u << 4): flat_long_p<1, 2, 0, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
        case (2u | 1u << 2 | 0u << 4): flat_long_p<2, 1, 0, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
        case (2u | 0u << 2 | 1u << 4): flat_long_p<2, 0, 1, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
        case (0u | 2u << 2 | 1u << 4): flat_long_p<0, 2, 1, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
        case (0u | 1u << 2 | 2u << 4): flat_long_p<0, 1, 2, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
        default: flat_long_p<1, 0, 2, SAME, ANY, MIXED>(W, R, rays, b, len, cell); break;
      }
    } else {
      flat_long_p<3, 3, 3, SAME, ANY, MIXED>(W, R, rays, b, len, cell);
    }
    if ((rays >> lane) & 1u) {
      ++at;
      --n;
    }
    __syncwarp();
  }
}

// Rays [0, n) from *counter (zeroed).  src(i, org, dir, tmax, scene, anyhit)
// makes ray i; sink(i, hit, scene) takes its result, whose u and v are only
// computed if `uv`.  Scenes have fewer than kFlatMaxTris triangles.  MIXED:
// every scene has arrays of its own, and rays may be any-hit one by one
// (otherwise the scenes share one array of cells and one of references).  SAME:
// closest hits of rays with one origin.  COH: closest hits of rays whose
// neighbours may run side by side.
template <bool ANY, bool MIXED = false, bool SAME = false, bool COH = SAME, int K, class Acc, class Src, class Sink>
SHN_D void flat_trace(FlatWarpOf<K>* smem, const Acc& acc, uint32_t n, bool uv, uint32_t* counter, Src&& src, Sink&& sink) {
  static_assert(Acc::kIndirect, "triangles are read by id");
  static_assert(!(ANY || MIXED) || !(SAME || COH), "closest hits only");
  // A warp's first rays are its share by number (no counter to wait for: AO and
  // any-hit calls of 100,000 to 260,000 rays 89 -> 71 and 62 -> 54 us).  The rest
  // is reserved an eighth of the average share at a time, one reservation ahead
  // of its use: a quarter left one warp with the rays of a dense cell to itself
  // (camera on the ball in 5 x 5 x 5 cells 1.33 -> 1.21 ms).
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t given = min(32u, (n - 1u) / warps + 1u), grab = min(32u, max(1u, n / (8u * warps)));
  const Refs R0 = MIXED ? Refs{} : acc.refs(0u);
  const uint2* __restrict__ cells0 = MIXED ? nullptr : acc.cells(0u);
  FlatWarpOf<K>& W = smem[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  // lane 0: first ray of the reservation ahead; its rays
  uint32_t next = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * given, take = given;
  bool pool_empty = false;
  while (!pool_empty) {
    bool active = false, fin = false;  // the lane's ray: being traced; done, its result not written yet
    uint32_t waiting = 0, ngen = 0;
    while (true) {
      const uint32_t finm = __ballot_sync(0xFFFFFFFFu, fin);
      if (__popc(finm) >= kFlatRefill || !__any_sync(0xFFFFFFFFu, active)) {
        if (fin) {
          const float4 B = W.b[lane];
          Hit h{B.w, W.best[lane], 0.f, 0.f};
          if (uv && h.tri != kMiss) {
            const float4 A = W.a[lane];
            const uint32_t perm = __float_as_uint(B.z);
            RayWT w;
            w.org = mk(A.x, A.y, A.z);
            w.kx = perm & 3u;
            w.ky = (perm >> 2) & 3u;
            w.kz = (perm >> 4) & 3u;
            w.Sx = A.w;
            w.Sy = B.x;
            w.Sz = B.y;
            const float4* rec = (MIXED ? acc.refs(__float_as_uint(W.d[lane].w) >> 4).src : R0.src) + 3 * (size_t)h.tri;
            float t;
            wt_test(w, __ldg(rec), __ldg(rec + 1), __ldg(rec + 2), kEps, INFINITY, t, h.u, h.v);
          }
          sink(W.rid[lane], h, __float_as_uint(W.d[lane].w) >> 4);
          fin = false;
        }
        while (true) {
          const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !active);
          if (idle == 0u) break;
          if (waiting) {
            const uint32_t took = min(waiting, (uint32_t)__popc(idle)), rank = __popc(idle & lt);
            waiting -= took;
            if (!active && rank < took) {
              const uint32_t i = W.wait[waiting + rank];
              V3 o, d, cell;
              float tmax;
              uint32_t sc = 0, ah = 0;
              src(i, o, d, tmax, sc, ah);
              flat_enter(acc.geom(sc), o, d, tmax, cell);
              flat_queue(acc.geom(sc), acc.cell0(sc), o, d, tmax, cell, i, sc, ah, W, lane);
              active = true;
            }
            __syncwarp();
            continue;
          }
          if (pool_empty || ngen >= 32u) break;
          const uint32_t base = __shfl_sync(0xFFFFFFFFu, next, 0);
          if (base >= n) {
            pool_empty = true;
            break;
          }
          const uint32_t taken = take;
          take = grab;
          if (lane == 0) next = warps * given + atomicAdd(counter, grab);
          int what = FLAT_MISS;
          const uint32_t i = base + lane;
          if ((uint32_t)lane < taken && i < n) {
            V3 o, d, cell;
            float tmax;
            uint32_t sc = 0, ah = 0;
            src(i, o, d, tmax, sc, ah);
            what = flat_enter(acc.geom(sc), o, d, tmax, cell);
            if (what == FLAT_MISS) sink(i, Hit{tmax, kMiss, 0.f, 0.f}, sc);
          }
          const uint32_t qm = __ballot_sync(0xFFFFFFFFu, what == FLAT_RAY);
          const uint32_t gm = __ballot_sync(0xFFFFFFFFu, what == FLAT_GENERAL);
          if (what == FLAT_RAY) W.wait[__popc(qm & lt)] = i;
          if (what == FLAT_GENERAL) W.general[ngen + __popc(gm & lt)] = i;
          waiting = __popc(qm);
          ngen += __popc(gm);
          __syncwarp();
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
      }

      // ---- walk: the next K cells ------------------------------------------------
      float ex[K];  // a ray leaves a cell of the window if its bound lies beyond this
      bool on = active, again = false, some;
      uint32_t sum, longs;  // references of the short ranges; the lane's long ranges, those of lanes before << 16
      {
        uint2 r[K];
        uint32_t packed = 0;  // short ranges | their references << 9 | long ranges << 23
#pragma unroll
        for (int q = 0; q < K; ++q) {
          r[q] = make_uint2(0u, 0u);
          ex[q] = 0.f;
        }
        if (active) {
          const float4 C = W.c[lane], D = W.d[lane];
          const uint2 E = W.e[lane];
          const float bound = W.b[lane].w;
          const uint32_t bits = __float_as_uint(D.w);
          const Geom& g = acc.geom(bits >> 4);
          const uint2* __restrict__ cells = MIXED ? acc.cells(bits >> 4) : cells0;
          const int sx = bits & 1u ? 1 : -1, sy = bits & 2u ? g.res[0] : -g.res[0],
                    sz = bits & 4u ? g.res[0] * g.res[1] : -g.res[0] * g.res[1];
          float mx = C.x, my = C.y, mz = C.z;
          uint32_t idx = __float_as_uint(C.w);
          int rx = (int)(E.x & 0xFFFFu), ry = (int)(E.x >> 16), rz = (int)(E.y & 0xFFFFu), skip = (int)(E.y >> 16);
#pragma unroll
          for (int q = 0; q < K; ++q) {
            if (on && skip <= q) r[q] = __ldg(cells + idx);
            ex[q] = fminf(fminf(mx, my), mz);
            // (a ray that is not on any more may step anywhere)
            const bool xy = mx < my;
            const bool p0 = xy && mx < mz, p1 = !xy && my < mz, p2 = !p0 && !p1;
            if (p0) mx += D.x;
            if (p1) my += D.y;
            if (p2) mz += D.z;
            idx += (uint32_t)(p0 ? sx : (p1 ? sy : sz));
            if (p0) --rx;
            if (p1) --ry;
            if (p2) --rz;
            on = on && (rx | ry | rz) >= 0 && bound > ex[q];
          }
          // an empty cell may hold its distance D to the next occupied one: the
          // D - 1 cells after it are empty
          skip = max(skip - K, 0);
#pragma unroll
          for (int q = 0; q < K; ++q)
            if (r[q].y <= r[q].x) skip = max(skip, (int)r[q].x - (K - q));
          W.c[lane] = make_float4(mx, my, mz, __uint_as_float(idx));
          W.e[lane] = make_uint2((uint32_t)rx | (uint32_t)ry << 16, (uint32_t)rz | (uint32_t)skip << 16);
        }
        uint32_t longest = MIXED || SAME ? kCoopThreshold : kFlatLong;
        if (COH && !SAME) {
          uint32_t mid = ~0u - lane;  // the lane's first range of more than kCoopThreshold
#pragma unroll
          for (int q = K - 1; q >= 0; --q)
            if (r[q].y > r[q].x + kCoopThreshold) mid = r[q].x;
          const uint32_t has = __ballot_sync(0xFFFFFFFFu, mid < 1u << 30);
          if (has && 2 * __popc(__ballot_sync(0xFFFFFFFFu, __shfl_xor_sync(0xFFFFFFFFu, mid, 1) == mid)) >= __popc(has))
            longest = kCoopThreshold;
        }
#pragma unroll
        for (int q = 0; q < K; ++q) {
          if (r[q].y > r[q].x) {
            const uint32_t len = r[q].y - r[q].x;
            packed += len > longest ? 1u << 23 : len << 9 | 1u;
            again = again || len >= kFlatHuge;
          }
        }
        if (again) packed = 0;
        if (packed) W.key[lane] = ~0ull;
        if (!__any_sync(0xFFFFFFFFu, packed != 0u || again)) {
          if (active && !on) {
            active = false;
            fin = true;
          }
          continue;
        }
        some = packed != 0u;
        // number the references of all lanes' short ranges through, list the ranges
        const uint32_t incl = warp_incl_scan(packed);
        const uint32_t all = __shfl_sync(0xFFFFFFFFu, incl, 31), before = incl - packed;
        if (packed) {
          uint32_t k = before & 511u, f = (before >> 9) & 16383u, l = 32u * K + 31u - (before >> 23);
#pragma unroll
          for (int q = 0; q < K; ++q) {
            if (r[q].y > r[q].x) {
              const uint32_t len = r[q].y - r[q].x;
              if (len > longest) {
                W.own[l--] = make_uint2((uint32_t)(32 * q + lane) | len << 8, r[q].x);
              } else {
                W.own[k++] = make_uint2((uint32_t)(32 * q + lane) | f << 8, r[q].x - f);
                f += len;
              }
            }
          }
        }
        W.own[(all & 511u) + lane] = make_uint2(~0u, 0u);
        sum = (all >> 9) & 16383u;
        longs = packed >> 23 | (before >> 23) << 16;
      }
      __syncwarp();
      // the lane's ray has no result for the window yet; this is a pass for some
      // rays only, over the first of their cells (see the end of the pass)
      bool look = active, redo = false;
      do {
        // ---- test ------------------------------------------------------------------
        // The triangle ids of kFlatGroups groups of 32 references are loaded together.
        uint32_t started = 0;
        for (uint32_t j0 = 0; j0 < sum; j0 += 32u * kFlatGroups) {
          uint32_t id[kFlatGroups], slot[kFlatGroups], ref[kFlatGroups];
#pragma unroll
          for (int k = 0; k < kFlatGroups; ++k) {
            slot[k] = ~0u;
            if (k == 0 || j0 + 32u * k < sum) {
              // the ranges that start among these 32 numbers
              const uint32_t at = (W.own[started + lane].x >> 8) - (j0 + 32u * k);
              const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, at < 32u ? 1u << at : 0u);
              const uint32_t j = j0 + 32u * k + lane;
              const uint32_t rank = started + __popc(starts & (lt | (1u << lane))) - 1u;
              started += __popc(starts);
              if (j < sum) {
                const uint2 w = W.own[rank];
                slot[k] = w.x & 255u;
                const uint32_t* ridx = MIXED ? acc.refs(__float_as_uint(W.d[w.x & 31u].w) >> 4).ridx : R0.ridx;
                id[k] = __ldg(ridx + (j + w.y));
                if (MIXED) ref[k] = j + w.y;
              }
            }
          }
#pragma unroll
          for (int k = 0; k < kFlatGroups; ++k) {
            if (k != 0 && j0 + 32u * k >= sum) break;
            const uint32_t owner = slot[k] & 31u;
            // (a lane without a reference reads no ray's state: the place it would
            // look at may hold none)
            const bool mine = slot[k] != ~0u;
            const uint32_t bits = MIXED && mine ? __float_as_uint(W.d[owner].w) : 0u;
            const float4* rec = R0.rec;
            if (MIXED && mine) rec = acc.refs(bits >> 4).rec;
            rec += 3 * (size_t)(mine ? id[k] : 0u);
            int hit = 0;
            float t;
            // (numbers go up with the cells and their references, so an any-hit
            // ray's key from an earlier group stands; the long ranges come later.
            // ANY: whether a key of this group is seen makes no difference.)
            if (ANY || MIXED) __syncwarp();
            const bool done = (ANY || (MIXED && (bits & 8u))) && W.key[owner] != ~0ull;
            if (MIXED) __syncwarp();
            if (mine && !done)
              hit = flat_test(W.a[owner], W.b[owner], __ldg(rec), __ldg(rec + 1), __ldg(rec + 2), t);
            if (__any_sync(0xFFFFFFFFu, hit == 2)) {
              if (hit == 2) {
                const float4 A = W.a[owner], B = W.b[owner];
                hit = wt_test_p<3, 3, 3>(f4v(A), A.w, B.x, B.y, __ldg(rec), __ldg(rec + 1), __ldg(rec + 2), kEps, B.w, t,
                                         __float_as_uint(B.z)) ? 1 : 0;
              }
            }
            if (hit && (!redo || slot[k] >> 5 < __float_as_uint(W.b[owner].z) >> 8))
              atomicMin(&W.key[owner],
                        MIXED && (bits & 8u) ? flat_key_any(t, slot[k] >> 5, ref[k]) : flat_key(t, slot[k] >> 5, id[k]));
          }
        }
        __syncwarp();
        if (__any_sync(0xFFFFFFFFu, look && (longs & 0xFFFFu) != 0u))
          flat_long<ANY, MIXED, SAME, COH>(W, acc, longs >> 16, look ? longs & 0xFFFFu : 0u, ex);
        // ---- the window's result ------------------------------------------------------
        // The cells are visited in order while the bound lies beyond the exit of
        // the one before, so a least t beyond the entry of its cell is the result
        // of the cells visited: every earlier cell's exit lies before it.  A
        // triangle that is missing from the cell in which the ray meets it can be
        // found by a later cell, before that cell's entry; whether the walk gets
        // there depends on the cells before it, which are tested again by
        // themselves: it does unless their least t ends it.  (0.03 to 0.1 % of
        // the rays.  Traced again alone they held up whole calls: 1,021 rays
        // with one of them 59 -> 44 us, the camera on the ball of crowded cells
        // 3.0 -> 1.26 ms.)
        bool more = false;
        if (look) {
          const unsigned long long k = some ? W.key[lane] : ~0ull;
          bool end = !on;
          const uint32_t bits = MIXED ? __float_as_uint(W.d[lane].w) : 0u;
          if (MIXED && (bits & 8u)) {
            if (k != ~0ull) {
              W.best[lane] = __ldg(acc.refs(bits >> 4).ridx + ((uint32_t)(k >> 31) & 0x3FFFFFFFu));
              W.b[lane].w = __uint_as_float((uint32_t)k & 0x7FFFFFFFu);
              end = true;
            }
          } else if (k != ~0ull || redo) {
            const float t = flat_key_t(k);  // (NaN if there is no hit)
            const uint32_t q = (uint32_t)(k >> 30) & 7u;
            float entry = -INFINITY;
#pragma unroll
            for (int i = 0; i + 1 < K; ++i)
              if (q == (uint32_t)i + 1u) entry = ex[i];
            bool got = false;  // the walk gets to the cell of the hit found before
            if (redo) {
              float far = -INFINITY;
              const uint32_t cells = __float_as_uint(W.b[lane].z) >> 8;
#pragma unroll
              for (int i = 0; i + 1 < K; ++i)
                if (cells == (uint32_t)i + 1u) far = ex[i];
              got = !(t <= far);
            }
            if (got) {
              W.b[lane].w = W.far_t[lane];
              end = true;
            } else {
              W.best[lane] = (uint32_t)k & (kFlatMaxTris - 1u);
              more = !ANY && !(t > entry);
              if (more) {
                W.far_t[lane] = t;
                W.key[lane] = ~0ull;
                W.b[lane].z = __uint_as_float((__float_as_uint(W.b[lane].z) & 63u) | q << 8);
              } else {
                W.b[lane].w = t;
                end = end || ANY || !(t > ex[K - 1]);
              }
            }
          }
          if (!more && (end || again)) {
            active = false;
            fin = !again;
          }
        }
        look = more;
        if (redo || __any_sync(0xFFFFFFFFu, more || again)) {
          redo = !ANY && __any_sync(0xFFFFFFFFu, more);
          if (!more)
            W.b[lane].z = __uint_as_float((__float_as_uint(W.b[lane].z) & 63u) | (redo ? 0u : (uint32_t)K << 8));
          const uint32_t am = __ballot_sync(0xFFFFFFFFu, again);
          if (again) W.general[ngen + __popc(am & lt)] = W.rid[lane];
          ngen += __popc(am);
          again = false;
          __syncwarp();
        }
      } while (redo);
      __syncwarp();
    }
    for (uint32_t k = lane; k < ngen; k += 32) {
      const uint32_t i = W.general[k];
      V3 o, d;
      float tmax;
      uint32_t sc = 0, ah = 0;
      src(i, o, d, tmax, sc, ah);
      Hit h;
      flat_general<ANY>(acc.geom(sc), (MIXED ? acc.cells(sc) : cells0) + acc.cell0(sc), MIXED ? acc.refs(sc) : R0, o,
                             d, tmax, ah, h);
      sink(i, h, sc);
    }
    __syncwarp();
  }
}

// One uniform grid for every ray; its triangles are read by id through
// indices[].
struct FlatGrid {
  static constexpr bool kIndirect = true;
  const GridView* G;
  SHN_D const Geom& geom(uint32_t) const { return G->g; }
  SHN_D const uint2* cells(uint32_t) const { return G->cells; }
  SHN_D uint32_t cell0(uint32_t) const { return 0u; }
  SHN_D Refs refs(uint32_t) const { return refs_of(*G); }
};

}  // namespace shn
