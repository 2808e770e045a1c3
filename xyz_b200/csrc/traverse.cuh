// kd-tree closest-hit traversal for one ray (device).
//
// Semantics of the reference (xyz/geom/kdtree.cpp:82-150, 366-372):
//   * at an interior node, the plane distance e splits [t_min, t_max]; the near
//     child is the side holding the origin; e > t_max or e < 0 -> near only,
//     e < t_min -> far only, otherwise near on [t_min, e] then far on
//     [e, t_max];
//   * a leaf tests all its triangles with the double-faced Moller-Trumbore test
//     (xyz/geom/triangle.cpp:127-165): |det| < 1e-6 rejects, t must lie in the
//     interval (inclusive), barycentrics f, g >= 0 and f + g <= 1; an accepted
//     hit shrinks t_max, so among equal t the later triangle of a leaf wins;
//   * traversal stops at the first leaf (front to back) that produced a hit.
// Differences, all of which leave the closest hit unchanged: the ray is first
// clipped to the scene box, and triangles are tested against the ray's whole
// remaining interval [t_min, best_t] rather than the node's clipped interval,
// stopping once best_t <= the leaf's exit distance (robust to a hit that
// rounds across a split plane).  The plane distance uses a precomputed
// reciprocal of the direction.  A ray that starts exactly on a split plane
// continues on the side its direction points to.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "wide.cuh"

namespace xyzgpu {

struct TraceCount {
  uint32_t nodes, leaves, tris;
};

// A deferred far child: its node and exit distance.  Its entry distance is
// not stored: in front-to-back order the far child pushed last is popped
// right after the subtree that ends at its split plane, so the entry equals
// the exit distance of the leaf just finished (8 bytes per entry keep the
// local-memory stack small; it competes with node fetches for L1).
struct __align__(8) StackEntry {
  uint32_t node;
  float tf;
};

// Persistent closest-hit loop over rays [0, n) taken from a shared work
// counter, with per-lane refill: after every leaf visit the lanes whose ray
// has finished are counted with a ballot; once enough are idle, one atomicAdd
// by the first of them fetches that many new rays, and each takes its index
// from a popcount of the lanes below it.  A lane therefore never idles while its warp finishes long
// rays, which keeps the warp's lanes busy on incoherent secondary and shadow
// rays (the warp-per-batch scheme leaves most lanes waiting for the slowest
// ray of the batch).  Every lane of the warp must call this.
//   Sink::load(i, o, d, tmin, tmax)   ray i
//   Sink::store(i, hit)               result of ray i
//   Sink::scene(i)                    (kBatch) the scene of ray i; rays of one
//                                     queue may belong to different scenes
//   Sink::target(i)                   (sinks with kTarget) the triangle whose
//                                     being the closest hit is the only
//                                     question the caller asks (next-event
//                                     estimation's visibility test,
//                                     xyz/bsdf/lambert.cpp:151-155)
//
// Target queries end early, with the same answer the full closest-hit search
// gives: the target's own hit distance t_own is computed first, with the
// same arithmetic the traversal would apply to it.  If the target is not hit
// at all, it cannot be the closest hit and the ray needs no traversal.  Once
// any triangle is accepted at t < t_own, the final closest hit has t < t_own
// too, so it is not the target whatever the remaining nodes hold, and the ray
// stops (the store then sees a non-target id).  Nothing else changes: the
// target itself and hits at t >= t_own go through the unchanged closest-hit
// rules, so ties and rounding across split planes resolve as before.
constexpr int kRefillIdle = 12;

template <class S, class = void>
struct SinkHasTarget : std::false_type {};
template <class S>
struct SinkHasTarget<S, std::void_t<decltype(S::kTarget)>> : std::bool_constant<S::kTarget> {};
// Sinks with kMixed hold plain rays as well (target(i) is -1, targeted(i) false).
template <class S, class = void>
struct SinkIsMixed : std::false_type {};
template <class S>
struct SinkIsMixed<S, std::void_t<decltype(S::kMixed)>> : std::bool_constant<S::kMixed> {};
template <class Sink>
XYZ_DEV bool sink_targeted(const Sink &s, int i) {
  if constexpr (SinkIsMixed<Sink>::value)
    return s.targeted(i);
  else
    return SinkHasTarget<Sink>::value;
}
// One iteration of the persistent loop descends at most this many nodes; a lane
// still above its next leaf resumes there in the next iteration, so the warp's
// leaf tests do not wait for its longest descent (counting renders descend
// without the cap).
#ifndef XYZ_DESCEND_STEPS
#define XYZ_DESCEND_STEPS 8
#endif
constexpr int kDescendSteps = XYZ_DESCEND_STEPS;

template <bool kCount, bool kBatch = false, class Sink>
XYZ_DEV void trace_persistent(const DevScene &S, int n, int *fetch, Sink &sink, TraceCount &tc) {
  constexpr bool kTarget = SinkHasTarget<Sink>::value;
  int const lane = threadIdx.x & 31;
  unsigned const lanes_below = (1u << lane) - 1u;
  int ray = -1;
  bool exhausted = false;
  f3 o{}, d{};
  float inv[3] = {0.0f, 0.0f, 0.0f};
  float tmin = 0.0f;
  RayHit h{};
  float stop_t = 0.0f;  // target queries: the target's own hit distance
  uint32_t node = 0;
  float tn = 0.0f, tf = 0.0f;
  int sp = 0;
  StackEntry stack[kKdMaxDepthLimit];
  const DevScene *lane_scene = &S;
  for (;;) {
    bool const need = ray < 0 && !exhausted;
    // refill once at least kRefillIdle lanes are idle: refilling after every
    // finished ray costs more than it gains (measured on B200: 8..20 idle lanes
    // is best, 1 and 32 are 10 % slower)
    unsigned const idle = __ballot_sync(0xffffffffu, ray < 0);
    unsigned const want = (__popc(idle) >= kRefillIdle) ? __ballot_sync(0xffffffffu, need) : 0u;
    if (want) {
      int const leader = __ffs(want) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(fetch, __popc(want));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (need) {
        int const i = base + __popc(want & lanes_below);
        if (beyond_queue(i, n)) {
          exhausted = true;
        } else {
          float tmax;
          sink.load(i, o, d, tmin, tmax);
          if constexpr (kBatch) lane_scene = sink.scene(i);
          const DevScene &SL = kBatch ? *lane_scene : S;
          h.t = tmax;
          h.id = -1;
          h.f = h.g = 0.0f;
          h.back = 0;
          bool skip = false;
          if constexpr (kTarget) {
            stop_t = -INFINITY;
            if (sink_targeted(sink, i)) {
              RayHit own = h;
              skip = !hit_triangle(SL.tri, sink.target(i), o, d, tmin, own);
              stop_t = own.t;
              if (kCount) tc.tris++;
            }
          }
          inv[0] = __frcp_rn(d.x);
          inv[1] = __frcp_rn(d.y);
          inv[2] = __frcp_rn(d.z);
          float const org[3] = {o.x, o.y, o.z};
          float const lo[3] = {SL.bmin.x, SL.bmin.y, SL.bmin.z};
          float const hi[3] = {SL.bmax.x, SL.bmax.y, SL.bmax.z};
          float t0 = tmin, t1 = tmax;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            float const ta = (lo[k] - org[k]) * inv[k];
            float const tb = (hi[k] - org[k]) * inv[k];
            t0 = fmaxf(t0, fminf(ta, tb));
            t1 = fminf(t1, fmaxf(ta, tb));
          }
          if (skip) {
            // the target is not hit: the answer is "not the target" (h.id = -1)
            sink.store(i, h);
          } else if (!(t0 <= t1)) {
            sink.store(i, h);  // misses the scene box
          } else {
            ray = i;
            node = 0;
            tn = t0;
            tf = t1;
            sp = 0;
          }
        }
      }
    }
    if (__all_sync(0xffffffffu, exhausted && ray < 0)) break;
    if (ray < 0) continue;
    const uint2 *__restrict__ nodes = kBatch ? lane_scene->nodes : S.nodes;
    // descend to a leaf
    uint2 nd = __ldg(&nodes[node]);
    if (kCount) tc.nodes++;
    int steps = 0;
    while ((nd.y & 3u) != kKdLeafTag && (kCount || steps < kDescendSteps)) {
      ++steps;
      uint32_t const ax = nd.y & 3u;
      float const split = __uint_as_float(nd.x);
      uint32_t const child = nd.y >> 2;
      float const oa = ax == 0 ? o.x : (ax == 1 ? o.y : o.z);
      float const ia = ax == 0 ? inv[0] : (ax == 1 ? inv[1] : inv[2]);
      float const da = ax == 0 ? d.x : (ax == 1 ? d.y : d.z);
      float const tp = (split - oa) * ia;
      uint32_t const above_first = (oa < split || (oa == split && da <= 0.0f)) ? 0u : 1u;
      uint32_t const first = child + above_first;
      uint32_t const second = child + (above_first ^ 1u);
      if ((tp > tf) || (tp <= 0.0f)) {
        node = first;
      } else if (tp < tn) {
        node = second;
      } else {
        stack[sp] = StackEntry{second, tf};
        ++sp;
        node = first;
        tf = tp;
      }
      nd = __ldg(&nodes[node]);
      if (kCount) tc.nodes++;
    }
    if ((nd.y & 3u) != kKdLeafTag) continue;  // resumes at `node` in the next iteration
    // test the leaf
    uint32_t const cnt = nd.y >> 2;
    if (kCount) {
      tc.leaves++;
      tc.tris += cnt;
    }
    const int32_t *__restrict__ refs = kBatch ? lane_scene->refs : S.refs;
    const float4 *__restrict__ tris = kBatch ? lane_scene->tri : S.tri;
    int32_t t_next = cnt > 0 ? __ldg(&refs[nd.x]) : 0;
    for (uint32_t j = 0; j < cnt; ++j) {
      int32_t const t = t_next;
      if (j + 1 < cnt) t_next = __ldg(&refs[nd.x + j + 1]);
      hit_triangle(tris, t, o, d, tmin, h);
      if (kTarget && h.t < stop_t) break;
    }
    // next leaf (entered at this leaf's exit), or done
    bool const done = (h.id >= 0 && h.t <= tf) || sp == 0 || (kTarget && h.t < stop_t);
    if (!done) {
      --sp;
      StackEntry const e = stack[sp];
      node = e.node;
      tn = tf;
      tf = e.tf;
    }
    if (done) {
      sink.store(ray, h);
      ray = -1;
    }
  }
}

// ---------------------------------------------------------------- wide tree
// Persistent closest-hit loop over the wide tree (wide.cuh), with the answers
// of the kd-tree loop above, bit for bit.
//
// Both loops apply the same triangle test, so they can differ only where the
// order of the tests or the choice of the cells decides: a hit so close to an
// edge of its triangle that rounding decides whether the ray's kd cells hold
// it, or two hits whose distances differ by less than their rounding.  Such
// rays are recognised while they are traced (wide_take: 0.1 to 1 % of them on a
// 1M-triangle mesh, nearly all where rays are 10,000 times as long as the
// triangles), and the leaf of the kd-tree in which the kd loop would stop says
// what it would answer (wide_leaf_answer).  Where that leaf does not decide (one
// of 10,000 of them), and for rays the wide tree cannot serve (wide_usable),
// the ray goes into a list of the warp in shared memory and is
// traced through the kd-tree once the list is full or the queue is empty.
//
// The claim rests on every triangle being tested that the kd loop could accept
// (wide_triangle and the slack of wide_test) and leaves out one kind of ray: one
// nearly in the plane of a triangle that passes it beside an edge.  The test may
// then report a hit far beyond the edge; the kd loop takes it where the ray's
// cells hold the triangle, this loop where the ray meets its box.  A ray that does
// so in the plane itself goes to the kd-tree (wide_parallel).
//
// Why: a cosine bounce on a 1M-triangle mesh takes the kd loop 44 dependent node
// loads and 15 triangle tests, at 8 of 32 lanes and 351 warp instructions a ray (the
// second bounce of a render); a wide node costs one round of uniform arithmetic on
// eight boxes for three 32-byte loads, and the ray needs eight of them and five
// tests, at 17 lanes and 173 instructions.
constexpr int kWideRetry = 128;  // list entries per warp; 64 + one refill + the lanes under way fit
constexpr int kWideRetryFull = 64;

template <class Sink>
struct RetrySink {
  static constexpr bool kTarget = SinkHasTarget<Sink>::value;
  static constexpr bool kMixed = SinkIsMixed<Sink>::value;
  Sink *s;
  const int32_t *list;
  XYZ_DEV void load(int i, f3 &o, f3 &d, float &tmin, float &tmax) const { s->load(list[i], o, d, tmin, tmax); }
  XYZ_DEV const DevScene *scene(int i) const { return s->scene(list[i]); }
  XYZ_DEV int32_t target(int i) const { return s->target(list[i]); }
  XYZ_DEV bool targeted(int i) const { return sink_targeted(*s, list[i]); }
  XYZ_DEV void store(int i, const RayHit &h) { s->store(list[i], h); }
};

XYZ_DEV void wide_load8(const uint32_t *p, uint32_t *w) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
      : "l"(p));
}

// Triangle tests run once kWideWait lanes wait for one, or fewer than kWideStep
// could take a node step; a lane tests at most kWideTris before its warp goes
// on.  Rays are taken once kWideRefill lanes are idle.  Measured on 2^22 second
// bounces of a 1M-triangle mesh / an indoor room / box stacks (ms): tests
// as they come, two at a time, 1.50 / 1.39 / 1.34; waiting for 8, 10, 14
// lanes 1.38 / 1.26 / 1.19, 1.35 / 1.23 / 1.17, 1.38 / 1.20 / 1.15; eight
// tests at a time 1.43 / 1.26 / 1.22; refill at 8 or 16 idle lanes +-2 %, but in
// a room of 36 triangles, whose rays take one node step and a dozen tests, 16
// keeps the warp's rays together: camera rays and two bounces 0.38 / 0.46 / 0.47
// ms at 12, 0.38 / 0.41 / 0.44 at 16, 0.36 / 0.41 / 0.44 at 20.
constexpr int kWideTris = 4;
constexpr int kWideWait = 12;
constexpr int kWideStep = 8;
constexpr int kWideRefill = 12, kWideRefillTiny = 16;
constexpr int kWideTinyNodes = 64;

// Rays a CTA of four warps needs to be worth launching: eight a warp.
constexpr int kRaysPerCta = 32;

// A lane holds one ray through three states: under way (live), finished with
// its answer still in registers, and empty.  Answers are written and new rays
// taken together, once enough lanes are not under way, so that neither runs
// for a lane or two at a time.
template <bool kBatch = false, class Sink>
XYZ_DEV void trace_wide(const DevScene &S, int n, int *fetch, Sink &sink, int32_t *list, float *list_t, int *list_fetch,
                        int warps) {
  constexpr bool kTarget = SinkHasTarget<Sink>::value;
  int const lane = threadIdx.x & 31;
  unsigned const lanes_below = (1u << lane) - 1u;
  // short queues: fewer lanes per warp, so that all warps have a share and a
  // warp's rays wait for fewer others
  int const width = min(32, max(1, ceil_div(n, warps)));
  int const refill_at = width < 32 ? 0 : 32 - ((kBatch || S.n_wide > kWideTinyNodes) ? kWideRefill : kWideRefillTiny);
  bool exhausted = lane >= width;
  bool kd_only = false;  // the same on every lane
  const DevScene *lane_scene = &S;
  for (;;) {
    int n_list = 0;  // entries of the warp's list (the same on every lane)
    int ray = -1;
    bool live = false;
    f3 d{};
    WideRay R{};
    float tmin = 0.0f, tlim = 0.0f;
    RayHit h{};
    float slack = 0.0f;  // > 0: rounding could decide the answer (wide_take)
    uint32_t base = 0, group = 0;             // node group: first child, hits (visiting order) << 8 | inner slots
    uint32_t tri_base = 0, tri_valid = 0, tri_hits = 0;
    int sp = 0;
    uint2 stack[kWideStack];
    for (;;) {
      unsigned under_way = __ballot_sync(0xffffffffu, live);
      if (__popc(under_way) <= refill_at) {
        int retry = -1;
        float retry_t = __int_as_float(0x7fffffff);  // a hit's distance, or no number
        if (ray >= 0 && !live) {
          if (tmin < 0.0f) {
            retry = ray;
          } else if (h.id >= 0 && slack > 0.0f) {
            retry = ray;
            retry_t = h.t;
          } else {
            sink.store(ray, h);
          }
          ray = -1;
        }
        // a full list is traced before more rays are taken
        unsigned const want =
            n_list <= kWideRetryFull ? __ballot_sync(0xffffffffu, ray < 0 && retry < 0 && !exhausted) : 0u;
        if (want) {
          int const leader = __ffs(want) - 1;
          int first = 0;
          if (lane == leader) first = atomicAdd(fetch, __popc(want));
          first = __shfl_sync(0xffffffffu, first, leader);
          if (want & (1u << lane)) {
            int const i = first + __popc(want & lanes_below);
            if (beyond_queue(i, n)) {
              exhausted = true;
            } else {
              float tmax;
              f3 o;
              sink.load(i, o, d, tmin, tmax);
              if constexpr (kBatch) lane_scene = sink.scene(i);
              const DevScene &SL = kBatch ? *lane_scene : S;
              h.t = tmax;
              h.f = h.g = 0.0f;
              h.id = -1;
              h.back = 0;
              tlim = tmax;
              slack = 0.0f;
              if (!SL.wide || !wide_usable(sub3(o, SL.wide_mid), d, SL.wide_reach) || !(0.0f <= tmin && tmin <= tmax)) {
                retry = i;
              } else {
                ray = i;
                live = true;
                R = wide_ray(o, d);
                // the root is the only child of a group
                base = 0;
                group = (1u << (8 + R.octinv)) | 1u;
                tri_hits = 0;
                sp = 0;
                if constexpr (kTarget) {
                  // the target's own hit: what could hide it lies before it;
                  // if it is not hit, the answer is "not the target"
                  if (sink_targeted(sink, i)) {
                    int32_t const own = sink.target(i);
                    float4 const a = __ldg(&SL.tri[3 * own]), b = __ldg(&SL.tri[3 * own + 1]),
                                 c = __ldg(&SL.tri[3 * own + 2]);
                    float t, f, g, det;
                    live = test_triangle(a, b, c, o, d, tmin, tmax, &t, &f, &g, &det);
                    if (live) {
                      float m, dt;
                      float const l1 = norm1(xyz3(b)), l2 = norm1(xyz3(c));
                      wide_margin(t, norm1(d), l1 + l2, norm1(mk3(a.w, b.w, c.w)) + l1 * l2, reciprocal(det), &m, &dt);
                      if (f < m || g < m || 1.0f - (f + g) < m || t < tmin + dt || tmax < t + dt) slack = dt;
                      h.t = t;
                      h.f = f;
                      h.g = g;
                      h.id = own;
                      h.back = det > 0.0f;
                      tlim = t + dt;
                    }
                  }
                }
              }
            }
          }
        }
        unsigned const again = __ballot_sync(0xffffffffu, retry >= 0);
        if (retry >= 0) {
          int const at = n_list + __popc(again & lanes_below);
          list[at] = retry;
          list_t[at] = retry_t;
        }
        n_list += __popc(again);
        // a whole warp of rays that the tree cannot serve: the rest of the queue
        // is taken to be like them
        if (__all_sync(0xffffffffu, retry >= 0 && !(retry_t == retry_t))) {
          kd_only = true;
          break;
        }
        under_way = __ballot_sync(0xffffffffu, live);
        // nothing under way: the list is traced and the rest of the queue
        // taken, or (not yet full) more rays are taken first
        if (under_way == 0u) {
          if (__all_sync(0xffffffffu, ray < 0 && (exhausted || n_list > kWideRetryFull))) break;
          continue;
        }
      }
      if (live && tri_hits == 0) {
        const uint32_t *__restrict__ nodes = kBatch ? lane_scene->wide : S.wide;
        // the group's next child in visiting order
        int const bit = 31 - __clz(static_cast<int>(group));
        group &= ~(1u << bit);
        uint32_t const slot = static_cast<uint32_t>(bit - 8) ^ R.octinv;
        uint32_t const child = base + __popc(group & ((1u << slot) - 1u));
        if (group >> 8) {
          stack[sp] = make_uint2(base, group);
          ++sp;
        }
        uint32_t w[kWideWords];
        const uint32_t *const p = nodes + static_cast<size_t>(child) * kWideWords;
        wide_load8(p, w);
        wide_load8(p + 8, w + 8);
        wide_load8(p + 16, w + 16);
        uint32_t const hit = wide_test(w, R, tmin, tlim);
        uint32_t const inner = w[8] & 0xffu;
        base = w[3];
        group = (wide_order(hit & inner, R.octinv) << 8) | inner;
        tri_base = w[7];
        tri_valid = w[8] >> 8;
        tri_hits = wide_spread(hit) & tri_valid;
      }
      // triangle tests once enough lanes wait for them
      unsigned const wait = __ballot_sync(0xffffffffu, live && tri_hits != 0);
      if (__popc(wait) >= kWideWait || __popc(under_way & ~wait) < kWideStep) {
        const float4 *__restrict__ tris = kBatch ? lane_scene->wide_tri : S.wide_tri;
#pragma unroll 1
        for (int k = 0; k < kWideTris && live && tri_hits; ++k) {
          int const bit = __ffs(static_cast<int>(tri_hits)) - 1;
          tri_hits &= tri_hits - 1u;
          uint32_t const rec = tri_base + __popc(tri_valid & ((1u << bit) - 1u));
          uint32_t w[16];
          const uint32_t *const p = reinterpret_cast<const uint32_t *>(tris + static_cast<size_t>(rec) * kWideTriVec);
          wide_load8(p, w);
          wide_load8(p + 8, w + 8);
          auto vec = [&](int q) {
            return make_float4(__uint_as_float(w[4 * q]), __uint_as_float(w[4 * q + 1]), __uint_as_float(w[4 * q + 2]),
                               __uint_as_float(w[4 * q + 3]));
          };
          float t, f, g, det;
          // such a ray is marked by its tmin, so that no branch and no register is
          // needed (a test of its own: 5 to 13 % of a small scene's traces)
          if (wide_parallel(dot3(d, mk3(vec(0).w, vec(1).w, vec(2).w)), __uint_as_float(w[15]))) tmin = -1.0f;
          if (test_triangle(vec(0), vec(1), vec(2), R.o, d, tmin, tlim, &t, &f, &g, &det)) {
            int32_t const id = static_cast<int32_t>(w[12]);
            float m, dt;
            wide_margin(t, norm1(d), __uint_as_float(w[13]), __uint_as_float(w[14]), reciprocal(det), &m, &dt);
            if (kTarget && id != h.id && t + dt < h.t && f >= m && g >= m && 1.0f - (f + g) >= m && t >= tmin + dt &&
                sink_targeted(sink, ray)) {
              // certainly before the target: the ray is answered
              h.id = -1;
              live = false;
            } else if (id != h.id) {
              wide_take(t, f, g, id, det > 0.0f, m, dt, tmin, h, tlim, slack);
            }
          }
        }
      }
      if (live && tri_hits == 0 && (group >> 8) == 0) {
        if (sp == 0) {
          live = false;
        } else {
          --sp;
          uint2 const e = stack[sp];
          base = e.x;
          group = e.y;
        }
      }
    }
    __syncwarp();
    int n_kd = 0;
    for (int j0 = 0; j0 < n_list; j0 += 32) {
      int i = j0 + lane < n_list ? list[j0 + lane] : -1;
      if (i >= 0) {
        RayHit a{list_t[j0 + lane], 0.0f, 0.0f, -1, 0};
        if (a.t == a.t) {
          f3 o, dir;
          float t0, t1;
          sink.load(i, o, dir, t0, t1);
          const DevScene *SL = &S;
          if constexpr (kBatch) SL = sink.scene(i);
          if (wide_leaf_answer(*SL, o, dir, t0, a)) {
            sink.store(i, a);
            i = -1;
          }
        }
      }
      unsigned const kept = __ballot_sync(0xffffffffu, i >= 0);
      if (i >= 0) list[n_kd + __popc(kept & lanes_below)] = i;
      n_kd += __popc(kept);
    }
    if (n_kd > 0) {
      if (lane == 0) *list_fetch = 0;
      __syncwarp();
      RetrySink<Sink> again{&sink, list};
      TraceCount tc{};
      trace_persistent<false, kBatch>(S, n_kd, list_fetch, again, tc);
      __syncwarp();
    }
    if (kd_only) {
      TraceCount tc{};
      trace_persistent<false, kBatch>(S, n, fetch, sink, tc);
      return;
    }
    if (__all_sync(0xffffffffu, exhausted)) return;
  }
}

// The retry lists of a CTA's warps.
constexpr int kTraceWarps = 4;
struct WideList {
  int32_t entry[kTraceWarps][kWideRetry];
  float t[kTraceWarps][kWideRetry];
  int fetch[kTraceWarps];
};

// The grid's warps, which share a launch's queues.
XYZ_DEV int grid_warps() { return static_cast<int>((gridDim.x * blockDim.x) >> 5); }

// Closest hits through the wide tree, or the kd-tree of a scene without one, of
// a queue that `warps` warps work on.
template <bool kBatch = false, class Sink>
XYZ_DEV void trace_closest_hits(const DevScene &S, int n, int *fetch, Sink &sink, WideList &L,
                                int warps = grid_warps()) {
  if (kBatch || S.wide) {
    int const w = threadIdx.x >> 5;
    trace_wide<kBatch>(S, n, fetch, sink, L.entry[w], L.t[w], &L.fetch[w], warps);
  } else {
    TraceCount tc{};
    trace_persistent<false, kBatch>(S, n, fetch, sink, tc);
  }
}

}  // namespace xyzgpu
