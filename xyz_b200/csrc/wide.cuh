// Eight-wide bounding-box tree over a scene's triangles, derived from its
// kd-tree: the structure the traversal kernels walk (traverse.cuh).
//
// Every triangle belongs to the one kd leaf that holds its centroid, so the
// kd-tree's split hierarchy becomes a hierarchy of triangle sets (no triangle
// is referenced twice) with tight boxes.  Groups of its nodes are merged into
// nodes of up to eight children (the child of largest surface is opened until
// eight are found), after Ylitie, Karras and Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017): child boxes
// as 8-bit steps of a per-node power-of-two grid, children placed in octant
// slots so that a ray visits them front to back in the order slot ^ octant.
//
// Node: 24 words (96 bytes, three 32-byte loads):
//   0..2   grid origin          3   index of the first inner child
//   4..6   grid step (x, y, z)  7   index of the node's first triangle record
//   8      inner-child slots (8 bits) | triangle bits << 8 (3 per slot, low bits first)
//   12..17 box minima, 8 bytes per axis (byte s = slot s); 18..23 box maxima
// Inner children lie consecutively in slot order, triangle records in bit order.
// Triangle record: 64 bytes, (v0, n.x) (e1, n.y) (e2, n.z) as in DevScene::tri,
// then the triangle id and the lengths for the error margins (WideTri).
//
// A 1M-triangle mesh: 11 MB of nodes and 63 MB of records, where the kd-tree
// keeps 38 MB of nodes, 35 MB of references and 47 MB of triangles.
//
// The functions are __host__ __device__: the host builds and walks the same
// tree in the tests' CPU check.
#pragma once

#include <cmath>
#include <cstring>

#include "common.cuh"

namespace xyzgpu {

constexpr int kWideWords = 24;       // 32-bit words of a node
constexpr int kWideLeafTris = 3;     // triangles of a leaf child
constexpr int kWideStack = 64;       // node groups a ray may hold: the tree is no deeper
constexpr int kWideTriVec = 4;       // float4 per triangle record
// While a ray is tested the boxes grow by kWideSlack of their distance from its
// origin (wide_test), which is small beside the triangles wherever the scene lies
// and however far it reaches.  An allowance for the longest possible ray, as a
// share of the largest coordinate S, is not (boxes grown by 2^-18 S / this, us for
// 2^21 rays between two points):
// an 80,000-triangle terrain 2 wide at coordinates of 0 / 1,000 / 10,000
// 1,203 / 1,938 / 17,649 and 1,215 / 1,238 / 1,368; a 1M-triangle object 6 wide in a
// ground of half width 300 / 1,000 / 3,000 2,390 / 3,516 / 8,022 and 1,391 / 1,445 /
// 1,454 (the kd loop 2,550 to 2,490).  Where it buys nothing it costs 2 %.  Rays
// from all over such a ground at the object's triangles, 10^4 to 10^5 times as long
// as these, are close calls to the last one: 5,455 / 7,388 / 13,718 and 2,101 /
// 2,965 / 5,588 (the kd loop 2,470 to 2,540, which is faster from 1,000 on).
// Rays from beyond kWideReach * S of the scene, or kWideFar times the median
// triangle's extent (WideTri::e), do not use the tree (wide_reach).
constexpr float kWideSlack = 1.0f / 524288.0f;
constexpr float kWidePad = 1.0f / 8388608.0f;  // of S: for boxes whose corners are rounded to nearest
constexpr float kWideReach = 65536.0f;
constexpr float kWideFar = 16384.0f;

// Triangle sets of the kd-tree's (breadth-first) nodes while the tree is built.
struct WideSets {
  uint4 *lo = nullptr;       // ordered keys of the box minimum
  uint4 *hi = nullptr;       // of the maximum; w: triangles below the node
  int32_t *first = nullptr;  // first triangle of the node in depth-first order
};

// A wide node to be built: `cnt` triangles from `first` under kd node `node`
// (all of it, or for a leaf with many triangles a range).
struct WideTask {
  int32_t node, first, cnt;
};

XYZ_HD uint32_t float_key(float f) {
#ifdef __CUDA_ARCH__
  uint32_t const u = __float_as_uint(f);
#else
  uint32_t u;
  std::memcpy(&u, &f, 4);
#endif
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
XYZ_HD float key_float(uint32_t k) {
  uint32_t const u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, 4);
  return f;
#endif
}
// The sum, rounded down and up.
XYZ_HD float add_down(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rd(a, b);
#else
  float const r = a + b;
  return static_cast<long double>(r) > static_cast<long double>(a) + b ? std::nextafter(r, -INFINITY) : r;
#endif
}
XYZ_HD float add_up(float a, float b) { return -add_down(-a, -b); }
XYZ_HD uint32_t wide_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u;
#endif
}
XYZ_HD float wide_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  std::memcpy(&f, &u, 4);
  return f;
#endif
}

// The kd leaf that holds the point: at a split plane, the side above.
XYZ_HD int32_t wide_leaf_of(const uint2 *nodes, f3 p) {
  uint32_t i = 0;
  uint2 nd = nodes[0];
  while ((nd.y & 3u) != kKdLeafTag) {
    uint32_t const ax = nd.y & 3u;
    float const v = ax == 0 ? p.x : (ax == 1 ? p.y : p.z);
    i = (nd.y >> 2) + (v < wide_float(nd.x) ? 0u : 1u);
    nd = nodes[i];
  }
  return static_cast<int32_t>(i);
}

// Opens a task into two, descending past kd nodes with all triangles on one
// side; a kd leaf's range is halved.  cnt > kWideLeafTris.
XYZ_HD void wide_open(const uint2 *nodes, const WideSets &T, WideTask t, WideTask *a, WideTask *b) {
  for (;;) {
    uint2 const nd = nodes[t.node];
    if ((nd.y & 3u) == kKdLeafTag) {
      int const h = t.cnt >> 1;
      *a = WideTask{t.node, t.first, h};
      *b = WideTask{t.node, t.first + h, t.cnt - h};
      return;
    }
    int32_t const c = static_cast<int32_t>(nd.y >> 2);
    int32_t const nl = static_cast<int32_t>(T.hi[c].w), nr = static_cast<int32_t>(T.hi[c + 1].w);
    if (nl > 0 && nr > 0) {
      *a = WideTask{c, t.first, nl};
      *b = WideTask{c + 1, t.first + nl, nr};
      return;
    }
    t.node = nl > 0 ? c : c + 1;
  }
}

struct WideBox {
  float lo[3], hi[3];
};

XYZ_HD WideBox wide_box(const WideSets &T, int32_t node) {
  uint4 const l = T.lo[node], h = T.hi[node];
  return WideBox{{key_float(l.x), key_float(l.y), key_float(l.z)}, {key_float(h.x), key_float(h.y), key_float(h.z)}};
}

// A triangle's box and the lengths its error margins need (wide_margin).
//
// The box holds every point that the triangle test may report, so that the walk
// tests each triangle the kd loop could accept.  The test divides by
// det = d.n, and n carries the rounding of its products (2.8 u |e1||e2|, u =
// 2^-24) as do the sums (3 u each): an accepted ray passes the triangle in its
// plane within 12 u e |e1||e2| |d| / |det| (e the longer edge), the part that
// grows with the ray's length left to wide_test.  For a well-shaped triangle
// that is a millionth of its size, for a sliver of width q e it is 12 u e / q:
// beyond its far edge rays are accepted that miss it by many times its width.
// |det| is at least kEpsilon (of a ray of |d| <= 2 here), and slopes below 1/16
// are left out: a box grown for every slope would have no bound.
// 200 slivers 1e-4 / 1e-5 as wide as long, 2 M rays aimed beside their edges: the
// box of the corners alone misses 1 / 47 hits that the kd loop reports, this one
// none of 16 M; triangle tests a ray 9.7 -> 12.6 / 10.2 -> 46.3.
struct WideTri {
  float lo[3], hi[3];
  float e, n;      // |e1| + |e2| and |n| + |e1||e2| (1-norms)
  float parallel;  // kWideParallel |n|, 0 below kEpsilon (wide_parallel)
};

// Rays in a triangle's plane, to 2^-15: the determinant is then of the size of its
// own rounding, and so are the sums that it divides, so that the test may accept
// triangles of that plane which the ray does not come near.  The kd loop's answer
// is what such triangles its cells hold; it is asked where a ray meets one.
// (Where the rounding stays below kEpsilon the test rejects them all.)
// Without this rule 112 of 135 M rays between two points of a surface (turned
// boxes, strips, plane figures) got another answer.
constexpr float kWideParallel = 1.0f / 32768.0f;

// Triangles by extent, four ranges to the octave: bucket of an extent, and the
// least extent of a bucket.
constexpr int kWideExtents = 1024;
XYZ_HD int wide_extent_bucket(float e) { return static_cast<int>(wide_bits(e) >> 21) & (kWideExtents - 1); }
inline float wide_extent_of(int bucket) { return wide_float(static_cast<uint32_t>(bucket) << 21); }

// How far from the middle of a scene (half extent `half`, largest coordinate S, n
// triangles counted by extent) rays may start to use the tree.  From further the
// slack of wide_test, a share of the distance, reaches the size of the triangles:
// nearly every hit is then a close call, and the triangle test's own error at a
// slope below the 0.17 that the slack allows for exceeds it.  2^21 rays at the
// triangles of a 1M-triangle mesh / an 80,000-triangle terrain / 6,000 triangles of
// boxes from 2^12, 2^14, 2^16, 2^18 extents, us: 1,117 / 1,157 / 1,008, 1,405 / 1,429
// / 1,338, 1,971 / 2,099 / 2,013, 4,971 / 6,266 / 4,804 by the wide tree, 1,730 / 1,320
// / 905 by the kd-tree at any distance.
inline float wide_reach_of(float half, float S, const uint32_t *extents, uint32_t n) {
  uint32_t below = 0;
  int b = 0;
  while (b < kWideExtents - 1 && (below += extents[b]) <= n / 2) ++b;
  return half + std::fmin(kWideReach * S, kWideFar * wide_extent_of(b));
}

constexpr float kWideGrow = 12.0f / 16777216.0f;

XYZ_HD WideTri wide_triangle(f3 v0, f3 e1, f3 e2, f3 n) {
  WideTri w;
  float const a = norm1(e1), b = norm1(e2), l1 = sqrtf(dot3(e1, e1)), l2 = sqrtf(dot3(e2, e2));
  float const top = fmaxf(fmaxf(fabsf(n.x), fabsf(n.y)), fabsf(n.z));
  f3 const u = top > 0.0f ? scl3(n, 1.0f / top) : n;
  float const uu = dot3(u, u), ln = top * sqrtf(uu);
  w.e = a + b;
  w.n = norm1(n) + a * b;
  w.parallel = kWideParallel * ln > kEpsilon ? kWideParallel * ln : 0.0f;
  float const grow = kWideGrow * fmaxf(l1, l2) * (l1 * l2) / fmaxf(0.5f * kEpsilon, 0.0625f * ln);
  for (int k = 0; k < 3; ++k) {
    float const x = comp3(v0, k), p = comp3(e1, k), q = comp3(e2, k), c = comp3(u, k);
    // in the triangle's plane: an axis along the normal needs none
    float const along = sqrtf(fmaxf(0.0f, 1.0f - c * c / uu)) + 4.0f / 16777216.0f * (l1 * l2) / ln;
    float const g = top > 0.0f ? grow * fminf(1.0f, along) : 0.0f;
    w.lo[k] = add_down(fminf(x, fminf(add_down(x, p), add_down(x, q))), -g);
    w.hi[k] = add_up(fmaxf(x, fmaxf(add_up(x, p), add_up(x, q))), g);
  }
  return w;
}

// The smallest power of two s >= 2^-100 with 252 s >= extent (the grid starts
// 1/32 step before the boxes and each bound may round one step outwards).
XYZ_HD float wide_step(float extent) {
  float const r = extent * (1.0f / 252.0f);
  uint32_t e = (wide_bits(r) >> 23) & 0xffu;
  if (wide_bits(r) & 0x7fffffu) ++e;
  if (e < 27u) e = 27u;
  return wide_float(e << 23);
}

// Builds one node of the tree from the boxes of T, grown by `pad`.
// alloc_nodes(k) / alloc_tris(k) reserve k consecutive node / record indices;
// put_task(i, t) names the task of inner node i, put_tri(pos, rec) the record of
// the triangle at depth-first position pos.
template <class AllocNodes, class AllocTris, class PutTask, class PutTri>
XYZ_HD void wide_make_node(const uint2 *nodes, const WideSets &T, WideTask root, float pad, uint32_t *w,
                           AllocNodes alloc_nodes, AllocTris alloc_tris, PutTask put_task, PutTri put_tri) {
  WideTask it[8];
  float area[8];
  int m = 1;
  it[0] = root;
  area[0] = INFINITY;
  while (m < 8) {
    // the largest child that cannot be a leaf, then (into slots that would stay
    // empty) the largest leaf of several triangles
    int best = -1;
    for (int i = 0; i < m; ++i)
      if (it[i].cnt > kWideLeafTris && (best < 0 || area[i] > area[best])) best = i;
    if (best < 0)
      for (int i = 0; i < m; ++i)
        if (it[i].cnt > 1 && (best < 0 || area[i] > area[best])) best = i;
    if (best < 0) break;
    WideTask a, b;
    wide_open(nodes, T, it[best], &a, &b);
    it[best] = a;
    it[m] = b;
    for (int k = 0; k < 2; ++k) {
      int const i = k == 0 ? best : m;
      WideBox const x = wide_box(T, it[i].node);
      float const dx = x.hi[0] - x.lo[0], dy = x.hi[1] - x.lo[1], dz = x.hi[2] - x.lo[2];
      area[i] = dx * dy + dy * dz + dz * dx;
    }
    ++m;
  }
  WideBox box[8], all;
  for (int k = 0; k < 3; ++k) {
    all.lo[k] = INFINITY;
    all.hi[k] = -INFINITY;
  }
  for (int i = 0; i < m; ++i) {
    box[i] = wide_box(T, it[i].node);
    for (int k = 0; k < 3; ++k) {
      box[i].lo[k] -= pad;
      box[i].hi[k] += pad;
      all.lo[k] = fminf(all.lo[k], box[i].lo[k]);
      all.hi[k] = fmaxf(all.hi[k], box[i].hi[k]);
    }
  }
  // octant slots: the (child, slot) pair that fits best, until all are placed
  int slot_child[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
  uint32_t todo = (1u << m) - 1u;
  while (todo) {
    float best = -INFINITY;
    int bc = -1, bs = -1;
    for (int i = 0; i < m; ++i) {
      if (!(todo & (1u << i))) continue;
      float c[3];
      for (int k = 0; k < 3; ++k) c[k] = (box[i].lo[k] + box[i].hi[k]) - (all.lo[k] + all.hi[k]);
      for (int s = 0; s < 8; ++s) {
        if (slot_child[s] >= 0) continue;
        float const v = ((s & 1) ? c[0] : -c[0]) + ((s & 2) ? c[1] : -c[1]) + ((s & 4) ? c[2] : -c[2]);
        if (bc < 0 || v > best) {
          best = v;
          bc = i;
          bs = s;
        }
      }
    }
    slot_child[bs] = bc;
    todo &= ~(1u << bc);
  }
  for (int k = 0; k < kWideWords; ++k) w[k] = 0u;
  float step[3], org[3];
  for (int k = 0; k < 3; ++k) {
    // (2^-22 of the coordinate: the rounding of the origin)
    step[k] = wide_step(all.hi[k] - all.lo[k] + fmaxf(fabsf(all.lo[k]), fabsf(all.hi[k])) * (1.0f / 4194304.0f));
    org[k] = add_down(all.lo[k], step[k] * (-1.0f / 32.0f));
    w[k] = wide_bits(org[k]);
    w[4 + k] = wide_bits(step[k]);
  }
  int n_inner = 0, n_tris = 0;
  for (int s = 0; s < 8; ++s) {
    int const i = slot_child[s];
    if (i < 0) continue;
    if (it[i].cnt > kWideLeafTris)
      ++n_inner;
    else
      n_tris += it[i].cnt;
  }
  uint32_t const nb = n_inner ? alloc_nodes(n_inner) : 0u;
  uint32_t const tb = n_tris ? alloc_tris(n_tris) : 0u;
  w[3] = nb;
  w[7] = tb;
  uint32_t meta = 0u;
  int ni = 0, ti = 0;
  for (int s = 0; s < 8; ++s) {
    int const i = slot_child[s];
    if (i < 0) continue;
    if (it[i].cnt > kWideLeafTris) {
      meta |= 1u << s;
      put_task(nb + ni, it[i]);
      ++ni;
    } else {
      for (int c = 0; c < it[i].cnt; ++c) {
        meta |= 1u << (8 + 3 * s + c);
        put_tri(it[i].first + c, tb + ti);
        ++ti;
      }
    }
    for (int k = 0; k < 3; ++k) {
      // wide_test places a plane to 1/128 step (its bytes are read as 65536 +
      // byte): a bound rounds outwards from 1/64 step beyond the box
      float const ql = floorf((box[i].lo[k] - org[k]) / step[k] - (1.0f / 64.0f));
      float const qh = ceilf((box[i].hi[k] - org[k]) / step[k] + (1.0f / 64.0f));
      uint32_t const bl = static_cast<uint32_t>(fminf(fmaxf(ql, 0.0f), 255.0f));
      uint32_t const bh = static_cast<uint32_t>(fminf(fmaxf(qh, 0.0f), 255.0f));
      w[12 + 2 * k + (s >> 2)] |= bl << (8 * (s & 3));
      w[18 + 2 * k + (s >> 2)] |= bh << (8 * (s & 3));
    }
  }
  w[8] = meta;
}

// ---------------------------------------------------------------- walking
// What the box tests of a ray need: origin, reciprocal direction (components
// below 1e-18 replaced by 1e-18 of their sign) and the order its octant gives
// the slots.
struct WideRay {
  f3 o, inv;
  uint32_t octinv;  // bit k set: the direction's component k is >= 0
};

XYZ_HD float wide_inv(float d) {
  float const a = fabsf(d) < 1e-18f ? copysignf(1e-18f, d) : d;
#ifdef __CUDA_ARCH__
  return __frcp_rn(a);
#else
  return 1.0f / a;
#endif
}

XYZ_HD WideRay wide_ray(f3 o, f3 d) {
  WideRay r;
  r.o = o;
  r.inv = mk3(wide_inv(d.x), wide_inv(d.y), wide_inv(d.z));
  r.octinv = (r.inv.x >= 0.0f ? 1u : 0u) | (r.inv.y >= 0.0f ? 2u : 0u) | (r.inv.z >= 0.0f ? 4u : 0u);
  return r;
}

// Rays the tree answers (o: from the scene's middle): within reach, no component so
// small that its reciprocal is infinite: such a ray can lie in a split plane of
// the kd-tree, whose distance is then not a number, and the kd loop's choice of
// cells is its own.
XYZ_HD bool wide_usable(f3 o, f3 d, float reach) {
  float const dd = dot3(d, d);
  return fabsf(o.x) <= reach && fabsf(o.y) <= reach && fabsf(o.z) <= reach && dd <= 1e12f && dd >= 1e-12f &&
         fminf(fminf(fabsf(d.x), fabsf(d.y)), fabsf(d.z)) >= 1e-37f;
}

// Byte j of w as the float 65536 + byte: the byte times 128 added to the bits
// of 65536 (an integer dot product: it runs on the FMA pipe, where the
// bit-moving forms would add to the ALU pipe that the comparisons fill).
template <int J>
XYZ_HD float wide_byte(uint32_t w) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(__dp4a(w, 128u << (8 * J), 0x47800000u));
#else
  return 65536.0f + static_cast<float>((w >> (8 * J)) & 0xffu);
#endif
}

XYZ_HD float wide_max3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fmaxf(fmaxf(a, b), c);
#endif
}
XYZ_HD float wide_min3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fminf(fminf(a, b), c);
#endif
}

XYZ_HD float wide_fma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// Two fused multiply-adds q * a + c of one axis (packed FP32 on the device).
XYZ_HD void wide_fma2(float q0, float q1, float a, float c, float *t0, float *t1) {
#ifdef __CUDA_ARCH__
  unsigned long long q, aa, cc, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(q0), "f"(q1));
  asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
  asm("mov.b64 %0, {%1, %1};" : "=l"(cc) : "f"(c));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(q), "l"(aa), "l"(cc));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*t0), "=f"(*t1) : "l"(r));
#else
  *t0 = std::fma(q0, a, c);
  *t1 = std::fma(q1, a, c);
#endif
}

// Slots kSlot + J and kSlot + J + 1 of a node (bytes J, J + 1 of the words n, f):
// 2^slot added to m where the ray's box interval meets [tmin, tlim].
template <int kSlot, int J>
XYZ_HD float wide_pair(const uint32_t n[3], const uint32_t f[3], const float a[3], const float cn[3], const float cf[3],
                       float tmin, float tlim, float m) {
  float tn[3][2], tf[3][2];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    wide_fma2(wide_byte<J>(n[k]), wide_byte<J + 1>(n[k]), a[k], cn[k], &tn[k][0], &tn[k][1]);
    wide_fma2(wide_byte<J>(f[k]), wide_byte<J + 1>(f[k]), a[k], cf[k], &tf[k][0], &tf[k][1]);
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    float const t0 = fmaxf(wide_max3(tn[0][s], tn[1][s], tn[2][s]), tmin);
    float const t1 = fminf(wide_min3(tf[0][s], tf[1][s], tf[2][s]), tlim);
    if (t0 <= t1) m += static_cast<float>(1 << (kSlot + J + s));
  }
  return m;
}

// Slots of node w whose boxes the ray meets within [tmin, tlim].  Empty slots
// may report a hit (their box is the grid's first cell): neither an inner bit
// nor a triangle bit of the node belongs to them.
XYZ_HD uint32_t wide_test(const uint32_t *w, const WideRay &r, float tmin, float tlim) {
  float a[3], cn[3], cf[3];
  float const inv[3] = {r.inv.x, r.inv.y, r.inv.z}, o[3] = {r.o.x, r.o.y, r.o.z};
  uint32_t near0[3], near1[3], far0[3], far1[3];
  // The boxes are widened by kWideSlack of their distance (32 u, u = 2^-24): the
  // plane distances err by 3 u of it, and the triangle test, whose differences and
  // products are as long as the ray, reports hits up to 4.9 u of it beside an edge,
  // over the slope of the ray to the triangle (above 0.17 here).
  float const slack =
      kWideSlack * fmaxf(fmaxf(fabsf(wide_float(w[0]) - o[0]), fabsf(wide_float(w[1]) - o[1])), fabsf(wide_float(w[2]) - o[2]));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a[k] = wide_float(w[4 + k]) * inv[k];
    // (origin - o) * inv - 65536 * a: the bytes are read as 65536 + byte
    float const po = wide_float(w[k]) - o[k];
    float const c = wide_fma(-65536.0f, a[k], po * inv[k]);
    cn[k] = wide_fma(-slack, fabsf(inv[k]), c);
    cf[k] = wide_fma(slack, fabsf(inv[k]), c);
    bool const pos = (r.octinv >> k) & 1u;
    near0[k] = pos ? w[12 + 2 * k] : w[18 + 2 * k];
    near1[k] = pos ? w[13 + 2 * k] : w[19 + 2 * k];
    far0[k] = pos ? w[18 + 2 * k] : w[12 + 2 * k];
    far1[k] = pos ? w[19 + 2 * k] : w[13 + 2 * k];
  }
  float m = 8388608.0f;  // 2^23: the sum's low mantissa bits are the slots
  m = wide_pair<0, 0>(near0, far0, a, cn, cf, tmin, tlim, m);
  m = wide_pair<0, 2>(near0, far0, a, cn, cf, tmin, tlim, m);
  m = wide_pair<4, 0>(near1, far1, a, cn, cf, tmin, tlim, m);
  m = wide_pair<4, 2>(near1, far1, a, cn, cf, tmin, tlim, m);
  return wide_bits(m) & 0xffu;
}

// Slot bits to visiting order: bit s moves to bit s ^ octinv; the highest bit
// is visited first.
XYZ_HD uint32_t wide_order(uint32_t h, uint32_t octinv) {
  if (octinv & 1u) h = ((h & 0x55u) << 1) | ((h >> 1) & 0x55u);
  if (octinv & 2u) h = ((h & 0x33u) << 2) | ((h >> 2) & 0x33u);
  if (octinv & 4u) h = ((h & 0x0fu) << 4) | (h >> 4);
  return h;
}

// Slot bits to triangle bits (three per slot).
XYZ_HD uint32_t wide_spread(uint32_t h) {
  h = (h | (h << 8)) & 0x00f00fu;
  h = (h | (h << 4)) & 0x0c30c3u;
  h = (h | (h << 2)) & 0x249249u;
  return h * 7u;
}

// ---------------------------------------------------------------- hits
struct RayHit {
  float t, f, g;
  int32_t id;    // -1 = miss
  int32_t back;  // 1 = hit from the back side (det > 0)
};

#ifdef __CUDA_ARCH__
#define XYZ_LDG(x) __ldg(&(x))
#else
#define XYZ_LDG(x) (x)
#endif

XYZ_HD float reciprocal(float x) {
#ifdef __CUDA_ARCH__
  return __frcp_rn(x);
#else
  return 1.0f / x;
#endif
}

// FindIntersectionDF (xyz/geom/triangle.cpp:127-165) on a packed triangle
// (a, b, c): the hit within [tmin, tmax] and det (positive: from the back side).
XYZ_HD bool test_triangle(float4 a, float4 b, float4 c, f3 o, f3 d, float tmin, float tmax, float *t_out,
                          float *f_out, float *g_out, float *det_out) {
  f3 const e2xe1 = mk3(a.w, b.w, c.w);
  float const det = dot3(d, e2xe1);
  if (fabsf(det) < kEpsilon) return false;
  float const inv_det = reciprocal(det);
  f3 const vmo = sub3(xyz3(a), o);
  float const t = inv_det * dot3(vmo, e2xe1);
  if ((t < tmin) || (tmax < t)) return false;
  f3 const dxvmo = cross3(d, vmo);
  float const f = inv_det * dot3(xyz3(c), dxvmo);
  if ((f < 0.0f) || (f > 1.0f)) return false;
  float const g = inv_det * -dot3(xyz3(b), dxvmo);
  if ((g < 0.0f) || ((f + g) > 1.0f)) return false;
  *t_out = t;
  *f_out = f;
  *g_out = g;
  *det_out = det;
  return true;
}

// The test on triangle i of the scene; updates best_t on acceptance.
XYZ_HD bool hit_triangle(const float4 *__restrict__ tri, int32_t i, f3 o, f3 d, float tmin, RayHit &h) {
  float t, f, g, det;
  if (!test_triangle(XYZ_LDG(tri[3 * i + 0]), XYZ_LDG(tri[3 * i + 1]), XYZ_LDG(tri[3 * i + 2]), o, d, tmin, h.t, &t,
                     &f, &g, &det))
    return false;
  h = RayHit{t, f, g, i, det > 0.0f};
  return true;
}

// Whether a ray lies in the triangle's plane (WideTri::parallel); its direction
// counts as if of length 1.
XYZ_HD bool wide_parallel(float det, float parallel) { return fabsf(det) < parallel; }

// Error bounds of an accepted hit of a ray with |d| = s (1-norm): `dt` in its
// distance, `m` in its barycentric coordinates.  The sums over the differences of
// the ray's and the triangle's coordinates, at most t s + |e| long, round by 3 u
// of their terms (u = 2^-24), the normal by 2.8 u |e1||e2|: 7 u |n| + 5.7 u |e1||e2|
// and 5.7 u t s |e| + 18 u |e1||e2| over det, both below the 8 u of w.n and w.e.
XYZ_HD void wide_margin(float t, float s, float e, float n, float inv_det, float *m, float *dt) {
  float const r = (fabsf(t) * s + e) * fabsf(inv_det) * (1.0f / 2097152.0f);
  *m = r * e * s;
  *dt = r * n;
}

// Takes a hit of triangle id into the ray's answer h: the nearest, and of equal
// distances the highest id.  The walk goes on to tlim, the answer's distance and
// its error; slack is positive where rounding could decide the kd loop's answer:
// the hit closer to an edge (or to tmin), or a second hit closer in distance,
// than its error.
XYZ_HD void wide_take(float t, float f, float g, int32_t id, int32_t back, float m, float dt, float tmin, RayHit &h,
                      float &tlim, float &slack) {
  bool const edge = f < m || g < m || 1.0f - (f + g) < m || t < tmin + dt;
  float const both = fmaxf(fmaxf(slack, tlim - h.t), dt);
  if (t < h.t || (t == h.t && id > h.id)) {
    slack = h.t <= t + dt ? both : (edge ? dt : 0.0f);
    h = RayHit{t, f, g, id, back};
    tlim = t + dt;
  } else {
    slack = both;
  }
}

// The kd loop's answer where h is the nearest hit of all triangles, if one leaf
// decides it.  The loop stops at the latest in the leaf whose interval of
// distances, as it computes them, holds h.t: if that leaf refers to h's
// triangle, or to others hit at the same distance, the last of them is the
// answer (a leaf's triangles are tested in order, and equal distances replace).
// False where it refers to none: the answer then depends on the leaves before.
XYZ_HD bool wide_leaf_answer(const DevScene &S, f3 o, f3 d, float tmin, RayHit &h) {
  f3 const inv = mk3(reciprocal(d.x), reciprocal(d.y), reciprocal(d.z));
  float tn = tmin, tf = INFINITY;
  for (int k = 0; k < 3; ++k) {
    float const ta = (comp3(S.bmin, k) - comp3(o, k)) * comp3(inv, k);
    float const tb = (comp3(S.bmax, k) - comp3(o, k)) * comp3(inv, k);
    tn = fmaxf(tn, fminf(ta, tb));
    tf = fminf(tf, fmaxf(ta, tb));
  }
  if (!(tn <= tf && tn <= h.t)) return false;
  uint2 nd = XYZ_LDG(S.nodes[0]);
  while ((nd.y & 3u) != kKdLeafTag) {
    int const ax = static_cast<int>(nd.y & 3u);
    float const split = wide_float(nd.x), oa = comp3(o, ax);
    float const tp = (split - oa) * comp3(inv, ax);
    uint32_t const first = (oa < split || (oa == split && comp3(d, ax) <= 0.0f)) ? 0u : 1u;
    bool in_first = true;
    if (!(tp > tf || tp <= 0.0f)) {
      if (tp < tn) {
        in_first = false;
      } else if (h.t <= tp) {
        tf = tp;
      } else {
        in_first = false;
        tn = tp;
      }
    }
    nd = XYZ_LDG(S.nodes[(nd.y >> 2) + (in_first ? first : first ^ 1u)]);
  }
  RayHit a = h;
  a.id = -1;
  for (uint32_t j = 0; j < (nd.y >> 2); ++j) hit_triangle(S.tri, XYZ_LDG(S.refs[nd.x + j]), o, d, tmin, a);
  if (a.id < 0 || a.t < h.t) return false;
  h = a;
  return true;
}

}  // namespace xyzgpu
