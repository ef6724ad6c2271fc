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
// are left on random rays.  Measured (B200): 4.0M random rays on a
// 1M-triangle soup 1.95 -> 0.91 ms; 512 x 512 primary rays on a 65,536-triangle
// soup 0.32 -> 0.17 ms; C2-sized path tracing (4.2M triangles, 1920 x 1080 x 16,
// depth 4) 100 -> 51 ms; 64 scenes' random rays 1.94 -> 0.76 ms.  What is left
// is latency: the random loads miss L2 (35-55 % hits), at 45-65 % issue.
// Sizes tried: windows of 4, 6 and 8 cells (0.98, 0.93, 0.94 ms on the random
// rays, 55.9, 53.8, 53.2 ms on the path tracer), 6 to 8 blocks per SM (0.93,
// 0.92 and 0.97 ms; 53.8, 50.9 and 56 ms).  Shared memory beyond ~160 KB per SM
// costs up to 1.6x: L1 then has too few lines for the loads in flight.
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
// are as fast or faster (4.0M rays: 0.92 against 0.94 ms).
constexpr int kFlatAhead = 6, kFlatAheadFew = 8;
constexpr uint32_t kFlatFew = 1u << 17;

// Shared memory of one warp.  The rays live here, not in registers: the walk
// loads and stores what it needs, so that the tests have the registers.  Every
// kilobyte less leaves L1 room for lines in flight.
template <int K>
struct FlatWarpOf {
  float4 a[32];  // org, Sx
  float4 b[32];  // Sy, Sz, axis permutation, bound (the best t so far)
  float4 c[32];  // tMax, cell
  float4 d[32];  // tDelta, direction signs (3 bits), any-hit flag, scene
  uint2 e[32];   // steps left in x and y | in z, cells ahead known to be empty
  uint32_t rid[32], best[32];
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
  Q.b[k] = make_float4(w.Sy, w.Sz, __uint_as_float(perm), tmax);
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
template <bool ANY, bool IND>
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
        lane_range<false, IND>(R, L, tests);
      }
      L.anyhit = 1;
    } else {
      lane_range<ANY, IND>(R, L, tests);
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

// Ranges of more references than this are loaded once for all of the warp's
// rays that wait on them (kCoopThreshold where rays may be any-hit one by one:
// their answer depends on it, see flat_key_any); a ray that meets one of 2^24
// is left to the general walk.
constexpr uint32_t kFlatLong = 63, kFlatHuge = 1u << 24;

// The long ranges, listed from the end of W.own (lane and cell | length << 8,
// first reference): per distinct range, each lane loads one reference of
// every 32 and tests it against each waiting ray.
template <bool ANY, bool MIXED, int K, class Acc>
SHN_D void flat_long(FlatWarpOf<K>& W, const Acc& acc, uint32_t count) {
  const int lane = threadIdx.x & 31;
  for (uint32_t k0 = 0; k0 < count; k0 += 32) {
    uint2 mine = make_uint2(0u, 0u);
    if (k0 + lane < count) mine = W.own[32 * K + 31 - (k0 + lane)];
    const uint32_t mscene = MIXED ? __float_as_uint(W.d[mine.x & 31u].w) >> 4 : 0u;
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, k0 + lane < count);
    while (todo) {
      const int j = __ffs(todo) - 1;
      const uint32_t b = __shfl_sync(0xFFFFFFFFu, mine.y, j), len = __shfl_sync(0xFFFFFFFFu, mine.x, j) >> 8;
      const uint32_t scene = __shfl_sync(0xFFFFFFFFu, mscene, j);
      const Refs R = acc.refs(scene);
      uint32_t rays = todo & __ballot_sync(0xFFFFFFFFu, mine.y == b && (mine.x >> 8) == len && mscene == scene);
      todo &= ~rays;
      for (uint32_t i0 = 0; i0 < len && rays; i0 += 32) {
        const bool in = i0 + lane < len;
        const uint32_t id = in ? __ldg(R.ridx + (b + i0 + lane)) : 0u;
        const float4* rec = R.rec + 3 * (size_t)id;
        const float4 p0 = __ldg(rec), p1 = __ldg(rec + 1), p2 = __ldg(rec + 2);
        for (uint32_t m = rays; m; m &= m - 1) {
          const int r = __ffs(m) - 1;
          const uint32_t slot = W.own[32 * K + 31 - (k0 + r)].x & 255u, owner = slot & 31u;
          const bool first = MIXED && (__float_as_uint(W.d[owner].w) & 8u);
          if (ANY || first) {
            // answered by an earlier cell (or, ANY, by any cell)
            const unsigned long long k = W.key[owner];
            if (k != ~0ull && (ANY || (uint32_t)(k >> 61) < slot >> 5)) {
              rays &= ~(1u << r);
              continue;
            }
          }
          const float4 A = W.a[owner], B = W.b[owner];
          float t;
          const bool hit =
              in && wt_test_p<3, 3, 3>(f4v(A), A.w, B.x, B.y, p0, p1, p2, kEps, B.w, t, __float_as_uint(B.z));
          if (ANY || first) {
            const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
            if (hits) {
              // t is positive: its bits are in its order; references are in that of the ids
              const uint32_t tb = hit ? __float_as_uint(t) : 0xFFFFFFFFu;
              const uint32_t least = __ballot_sync(0xFFFFFFFFu, tb == __reduce_min_sync(0xFFFFFFFFu, tb));
              if (lane == __ffs(least) - 1)
                atomicMin(&W.key[owner], first ? flat_key_any(t, slot >> 5, b + i0 + lane) : flat_key(t, slot >> 5, id));
              rays &= ~(1u << r);
              __syncwarp();
            }
          } else if (hit) {
            atomicMin(&W.key[owner], flat_key(t, slot >> 5, id));
          }
        }
      }
    }
  }
}

// Rays [0, n) from *counter (zeroed).  src(i, org, dir, tmax, scene, anyhit)
// makes ray i; sink(i, hit, scene) takes its result, whose u and v are only
// computed if `uv`.  Scenes have fewer than kFlatMaxTris triangles.  MIXED:
// every scene has arrays of its own, and rays may be any-hit one by one
// (otherwise the scenes share one array of cells and one of references).
template <bool ANY, bool MIXED = false, int K, class Acc, class Src, class Sink>
SHN_D void flat_trace(FlatWarpOf<K>* smem, const Acc& acc, uint32_t n, bool uv, uint32_t* counter, Src&& src, Sink&& sink) {
  constexpr bool IND = true;
  constexpr uint32_t kLong = MIXED ? kCoopThreshold : kFlatLong;
  static_assert(kLong <= 63u, "the references of a window's short ranges have 14 bits");
  static_assert(Acc::kIndirect, "triangles are read by id");
  // rays reserved at a time, one reservation ahead of its use; fewer when there
  // are few rays for every warp
  const uint32_t grab = min(32u, max(1u, n / (4u * gridDim.x * (blockDim.x >> 5))));
  const Refs R0 = MIXED ? Refs{} : acc.refs(0u);
  const uint2* __restrict__ cells0 = MIXED ? nullptr : acc.cells(0u);
  FlatWarpOf<K>& W = smem[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t next = 0;  // lane 0: first ray of the reservation ahead
  if (lane == 0) next = atomicAdd(counter, grab);
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
          if (lane == 0) next = atomicAdd(counter, grab);
          int what = FLAT_MISS;
          const uint32_t i = base + lane;
          if ((uint32_t)lane < grab && i < n) {
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
      uint32_t sum, nlong;
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
          for (int q = 0; q < K; ++q) {
            if (r[q].y > r[q].x) {
              const uint32_t len = r[q].y - r[q].x;
              packed += len > kLong ? 1u << 23 : len << 9 | 1u;
              again = again || len >= kFlatHuge;
            } else {
              skip = max(skip, (int)r[q].x - (K - q));
            }
          }
          if (again) packed = 0;
          if (packed) W.key[lane] = ~0ull;
          W.c[lane] = make_float4(mx, my, mz, __uint_as_float(idx));
          W.e[lane] = make_uint2((uint32_t)rx | (uint32_t)ry << 16, (uint32_t)rz | (uint32_t)skip << 16);
        }
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
              if (len > kLong) {
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
        nlong = all >> 23;
      }
      __syncwarp();
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
          // ray's key from an earlier group stands; the long ranges come later)
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
          if (hit)
            atomicMin(&W.key[owner],
                      MIXED && (bits & 8u) ? flat_key_any(t, slot[k] >> 5, ref[k]) : flat_key(t, slot[k] >> 5, id[k]));
        }
      }
      __syncwarp();
      if (nlong) {
        flat_long<ANY, MIXED>(W, acc, nlong);
        __syncwarp();
      }
      // ---- the window's result ------------------------------------------------------
      // The cells are visited in order while the bound lies beyond the exit of
      // the one before, so a least t beyond the entry of its cell is the result
      // of the cells visited: every earlier cell's exit lies before it.  A
      // triangle that is missing from the cell in which the ray meets it can be
      // found by a later cell, before that cell's entry; whether the walk gets
      // there depends on the cells between, and the ray is traced again alone.
      if (active) {
        const unsigned long long k = some ? W.key[lane] : ~0ull;
        bool end = !on;
        const uint32_t bits = MIXED ? __float_as_uint(W.d[lane].w) : 0u;
        if (MIXED && (bits & 8u)) {
          if (k != ~0ull) {
            W.best[lane] = __ldg(acc.refs(bits >> 4).ridx + ((uint32_t)(k >> 31) & 0x3FFFFFFFu));
            W.b[lane].w = __uint_as_float((uint32_t)k & 0x7FFFFFFFu);
            end = true;
          }
        } else if (k != ~0ull) {
          const float t = flat_key_t(k);
          const uint32_t q = (uint32_t)(k >> 30) & 7u;
          float entry = -INFINITY;
#pragma unroll
          for (int i = 0; i + 1 < K; ++i)
            if (q == (uint32_t)i + 1u) entry = ex[i];
          const float last = ex[K - 1];
          W.best[lane] = (uint32_t)k & (kFlatMaxTris - 1u);
          W.b[lane].w = t;
          again = again || (!ANY && !(t > entry));
          end = end || ANY || !(t > last);
        }
        if (end || again) {
          active = false;
          fin = !again;
        }
      }
      const uint32_t am = __ballot_sync(0xFFFFFFFFu, again);
      if (again) W.general[ngen + __popc(am & lt)] = W.rid[lane];
      ngen += __popc(am);
      __syncwarp();
    }
    for (uint32_t k = lane; k < ngen; k += 32) {
      const uint32_t i = W.general[k];
      V3 o, d;
      float tmax;
      uint32_t sc = 0, ah = 0;
      src(i, o, d, tmax, sc, ah);
      Hit h;
      flat_general<ANY, IND>(acc.geom(sc), (MIXED ? acc.cells(sc) : cells0) + acc.cell0(sc), MIXED ? acc.refs(sc) : R0, o,
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
