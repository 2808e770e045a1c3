// Host check of the wide tree's answers against the kd loop's: builds both trees
// of a scene, walks them for the same rays with the device's functions
// (xyz_b200/csrc/wide.cuh) and compares every bit of the hits.  Rays are aimed at
// or just beside the edges and corners of a triangle, where rounding decides.
//   wide_kd_check SCENE RAYS KIND        (see main)
// Prints  rays hits unsettled differ  nodes tests  kd_nodes kd_tests  (the last
// four per ray); exit code 1 if the scene cannot be built.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../xyz_b200/csrc/kdtree.h"
#include "../../xyz_b200/csrc/wide.cuh"

using namespace xyzgpu;

namespace {

struct Trees {
  std::vector<float4> tri;
  KdTreeHost kd;
  std::vector<uint2> nodes;
  std::vector<uint32_t> wide;
  std::vector<int> record;  // triangle of a record
  std::vector<WideTri> lengths;
  DevScene S{};
};

bool build(const std::vector<f3> &V, Trees &B) {
  int const n = static_cast<int>(V.size() / 3);
  std::vector<float> trv(9 * static_cast<size_t>(n));
  for (int i = 0; i < n; ++i) {
    f3 const v0 = V[3 * i], e1 = sub3(V[3 * i + 1], v0), e2 = sub3(V[3 * i + 2], v0), c = cross3(e2, e1);
    B.tri.push_back(make_float4(v0.x, v0.y, v0.z, c.x));
    B.tri.push_back(make_float4(e1.x, e1.y, e1.z, c.y));
    B.tri.push_back(make_float4(e2.x, e2.y, e2.z, c.z));
    f3 const p[3] = {v0, add3(v0, e1), add3(v0, e2)};
    for (int k = 0; k < 9; ++k) trv[9 * static_cast<size_t>(i) + k] = comp3(p[k / 3], k % 3);
  }
  BuildConfig cfg;
  cfg.max_depth = kd_resolve_max_depth(0, n);
  cfg.max_refs = 6ll * n + 1024;
  std::string err;
  if (!kd_build_host(trv.data(), n, cfg, &B.kd, &err)) return false;
  int const nn = static_cast<int>(B.kd.nodes.size() / 2);
  for (int i = 0; i < nn; ++i) B.nodes.push_back(make_uint2(B.kd.nodes[2 * i], B.kd.nodes[2 * i + 1]));
  const std::vector<uint2> &nd = B.nodes;
  std::vector<uint4> lo(nn, make_uint4(~0u, ~0u, ~0u, ~0u)), hi(nn, make_uint4(0, 0, 0, 0));
  std::vector<int32_t> first(nn, 0), owner(n);
  std::vector<uint32_t> extents(kWideExtents, 0u);
  for (int i = 0; i < n; ++i) {
    f3 const v0 = V[3 * i], e1 = xyz3(B.tri[3 * i + 1]), e2 = xyz3(B.tri[3 * i + 2]);
    WideTri const w =
        wide_triangle(v0, e1, e2, mk3(B.tri[3 * i].w, B.tri[3 * i + 1].w, B.tri[3 * i + 2].w));
    B.lengths.push_back(w);
    ++extents[wide_extent_bucket(w.e)];
    f3 const sum = add3(add3(v0, add3(v0, e1)), add3(v0, e2));
    int const l = owner[i] = wide_leaf_of(nd.data(), scl3(sum, 1.0f / 3.0f));
    uint32_t *const L = &lo[l].x, *const H = &hi[l].x;
    for (int k = 0; k < 3; ++k) {
      L[k] = std::min(L[k], float_key(w.lo[k]));
      H[k] = std::max(H[k], float_key(w.hi[k]));
    }
    ++H[3];
  }
  for (int i = nn - 1; i >= 0; --i) {
    if ((nd[i].y & 3u) == kKdLeafTag) continue;
    int const c = static_cast<int>(nd[i].y >> 2);
    for (int k = 0; k < 3; ++k) {
      (&lo[i].x)[k] = std::min((&lo[c].x)[k], (&lo[c + 1].x)[k]);
      (&hi[i].x)[k] = std::max((&hi[c].x)[k], (&hi[c + 1].x)[k]);
    }
    hi[i].w = hi[c].w + hi[c + 1].w;
  }
  for (int i = 0; i < nn; ++i) {
    if ((nd[i].y & 3u) == kKdLeafTag) continue;
    int const c = static_cast<int>(nd[i].y >> 2);
    first[c] = first[i];
    first[c + 1] = first[i] + static_cast<int>(hi[c].w);
  }
  float reach = 0.0f;
  for (int k = 0; k < 3; ++k) reach = std::max({reach, std::fabs(B.kd.bmin[k]), std::fabs(B.kd.bmax[k])});
  WideSets const W{lo.data(), hi.data(), first.data()};
  size_t const max_nodes = n / 4 + (n + n / 4) / 7 + 64;
  B.wide.resize(max_nodes * kWideWords);
  std::vector<WideTask> task(max_nodes);
  std::vector<int32_t> dst(n, -1);
  uint32_t made = 1, recs = 0;
  task[0] = WideTask{0, 0, n};
  for (uint32_t b = 0; b < made; ++b) {
    if (made > max_nodes) return false;
    wide_make_node(
        nd.data(), W, task[b], 0.0f, &B.wide[static_cast<size_t>(b) * kWideWords],
        [&](int k) { return (made += k) - k; }, [&](int k) { return (recs += k) - k; },
        [&](uint32_t at, WideTask t) { task[at] = t; }, [&](int32_t at, uint32_t r) { dst[at] = static_cast<int>(r); });
  }
  B.record.assign(n, -1);
  std::vector<int> fill(nn, 0);
  for (int i = 0; i < n; ++i) B.record[dst[first[owner[i]] + fill[owner[i]]++]] = i;
  B.S.tri = B.tri.data();
  B.S.nodes = B.nodes.data();
  B.S.refs = B.kd.refs.data();
  B.S.bmin = mk3(B.kd.bmin[0], B.kd.bmin[1], B.kd.bmin[2]);
  B.S.bmax = mk3(B.kd.bmax[0], B.kd.bmax[1], B.kd.bmax[2]);
  f3 const half = scl3(sub3(B.S.bmax, B.S.bmin), 0.5f);
  B.S.wide_mid = add3(B.S.bmin, half);
  B.S.wide_reach = wide_reach_of(std::max({half.x, half.y, half.z}), reach, extents.data(), static_cast<uint32_t>(n));
  return true;
}

// The kd loop of traverse.cuh for one ray.
RayHit kd_loop(const DevScene &S, f3 o, f3 d, float tmin, float tmax, double *nodes, double *tests) {
  RayHit h{tmax, 0.0f, 0.0f, -1, 0};
  float const inv[3] = {1.0f / d.x, 1.0f / d.y, 1.0f / d.z};
  float t0 = tmin, t1 = tmax;
  for (int k = 0; k < 3; ++k) {
    float const ta = (comp3(S.bmin, k) - comp3(o, k)) * inv[k], tb = (comp3(S.bmax, k) - comp3(o, k)) * inv[k];
    t0 = fmaxf(t0, fminf(ta, tb));
    t1 = fminf(t1, fmaxf(ta, tb));
  }
  if (!(t0 <= t1)) return h;
  std::vector<std::pair<uint32_t, float>> stack;
  uint32_t node = 0;
  float tn = t0, tf = t1;
  for (;;) {
    uint2 nd = S.nodes[node];
    for (; (nd.y & 3u) != kKdLeafTag; nd = S.nodes[node]) {
      int const ax = static_cast<int>(nd.y & 3u);
      float const split = wide_float(nd.x), oa = comp3(o, ax), tp = (split - oa) * inv[ax];
      uint32_t const above = (oa < split || (oa == split && comp3(d, ax) <= 0.0f)) ? 0u : 1u, c = nd.y >> 2;
      *nodes += 1;
      node = c + above;
      if (tp > tf || tp <= 0.0f) continue;
      if (tp < tn) {
        node = c + (above ^ 1u);
      } else {
        stack.push_back({c + (above ^ 1u), tf});
        tf = tp;
      }
    }
    *nodes += 1;
    for (uint32_t j = 0; j < (nd.y >> 2); ++j) {
      *tests += 1;
      hit_triangle(S.tri, S.refs[nd.x + j], o, d, tmin, h);
    }
    if ((h.id >= 0 && h.t <= tf) || stack.empty()) return h;
    node = stack.back().first;
    tn = tf;
    tf = stack.back().second;
    stack.pop_back();
  }
}

// The wide loop for one ray that the tree takes; false: it leaves the ray to the kd loop.
bool wide_loop(const Trees &B, f3 o, f3 d, float tmin, float tmax, RayHit &h, double *nodes, double *tests) {
  h = RayHit{tmax, 0.0f, 0.0f, -1, 0};
  float tlim = tmax, slack = 0.0f;
  WideRay const R = wide_ray(o, d);
  uint32_t base = 0, group = (1u << (8 + R.octinv)) | 1u;
  std::vector<uint2> stack;
  for (;;) {
    int const bit = 31 - __builtin_clz(group);
    group &= ~(1u << bit);
    uint32_t const slot = static_cast<uint32_t>(bit - 8) ^ R.octinv;
    uint32_t const child = base + __builtin_popcount(group & ((1u << slot) - 1u));
    if (group >> 8) stack.push_back(make_uint2(base, group));
    const uint32_t *w = &B.wide[static_cast<size_t>(child) * kWideWords];
    *nodes += 1;
    uint32_t const hit = wide_test(w, R, tmin, tlim), valid = w[8] >> 8;
    base = w[3];
    group = (wide_order(hit & w[8] & 0xffu, R.octinv) << 8) | (w[8] & 0xffu);
    for (uint32_t th = wide_spread(hit) & valid; th; th &= th - 1) {
      int const id = B.record[w[7] + __builtin_popcount(valid & ((1u << __builtin_ctz(th)) - 1u))];
      float t, f, g, det, m, dt;
      *tests += 1;
      if (wide_parallel(dot3(d, mk3(B.tri[3 * id].w, B.tri[3 * id + 1].w, B.tri[3 * id + 2].w)), B.lengths[id].parallel))
        return false;
      if (!test_triangle(B.tri[3 * id], B.tri[3 * id + 1], B.tri[3 * id + 2], o, d, tmin, tlim, &t, &f, &g, &det))
        continue;
      wide_margin(t, norm1(d), B.lengths[id].e, B.lengths[id].n, reciprocal(det), &m, &dt);
      wide_take(t, f, g, id, det > 0.0f, m, dt, tmin, h, tlim, slack);
    }
    if (group >> 8) continue;
    if (stack.empty()) break;
    base = stack.back().x;
    group = stack.back().y;
    stack.pop_back();
  }
  return !(h.id >= 0 && slack > 0.0f) || wide_leaf_answer(B.S, o, d, tmin, h);
}

void quad(std::vector<f3> &v, f3 a, f3 b, f3 c, f3 d) {
  for (f3 p : {a, b, c, a, c, d}) v.push_back(p);
}

// A 2 x 2 height field of 2 m^2 triangles about (at, 0, at).
void terrain(std::vector<f3> &v, int m, float at) {
  auto P = [&](int i, int j) {
    float const x = -1 + 2.0f * i / m, z = -1 + 2.0f * j / m;
    return mk3(at + x, 0.1f * std::sin(7 * x) * std::cos(5 * z) + 0.004f * std::sin(311.0f * i + 173.0f * j), at + z);
  };
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) quad(v, P(i, j), P(i + 1, j), P(i + 1, j + 1), P(i, j + 1));
}

}  // namespace

// scenes: sliver:WIDTH (200 long thin triangles), soup:SIZE, terrain:OFFSET, grid:SIDE (a terrain of so many squares
// a side), ground:HALF (a terrain patch above a ground that wide), boxes, turned (the boxes 30 times as large, about
// a slanted axis)
// kinds: edge (rays at a point 1e-7 to 1e-1 of a triangle inside or beyond one of its edges, from near and far),
// plane (rays between two points of a box's face), far (the same as edge, from 10 to 30,000 scene sizes), local (rays between two points of the scene's finely divided part)
int main(int argc, char **argv) {
  if (argc != 4) return 1;
  std::string const scene = argv[1], kind = argv[3];
  float const arg = scene.find(':') == std::string::npos ? 0.0f : std::stof(scene.substr(scene.find(':') + 1));
  std::mt19937 g(1);
  std::uniform_real_distribution<float> U(-1, 1);
  std::normal_distribution<float> N;
  auto unit = [](f3 a) { return scl3(a, 1.0f / std::sqrt(dot3(a, a))); };
  std::vector<f3> v;
  if (scene.rfind("sliver", 0) == 0) {
    for (int i = 0; i < 200; ++i) {
      f3 const c = mk3(U(g), U(g), U(g)), a = unit(mk3(N(g), N(g), N(g))), b = unit(cross3(a, mk3(N(g), N(g), N(g))));
      float const l = 0.65f + 0.35f * U(g), s = 0.65f + 0.35f * U(g);
      for (f3 p : {c, add3(c, scl3(a, l)), add3(add3(c, scl3(a, l * s)), scl3(b, arg * l))}) v.push_back(p);
    }
  } else if (scene.rfind("soup", 0) == 0) {
    for (int i = 0; i < 1000; ++i) {
      f3 const c = mk3(U(g), U(g), U(g));
      for (int k = 0; k < 3; ++k) v.push_back(add3(c, mk3(arg * U(g), arg * U(g), arg * U(g))));
    }
  } else if (scene.rfind("terrain", 0) == 0) {
    terrain(v, 120, arg);
  } else if (scene.rfind("grid", 0) == 0) {
    terrain(v, static_cast<int>(arg), 0.0f);
  } else if (scene.rfind("ground", 0) == 0) {
    terrain(v, 120, 0.0f);
    quad(v, mk3(-arg, -1, -arg), mk3(arg, -1, -arg), mk3(arg, -1, arg), mk3(-arg, -1, arg));
  } else {
    for (int i = 0; i < 80; ++i) {
      f3 const a = mk3(0.5f * (i % 9), 0.4f * (i % 4), 0.5f * (i / 9)), b = add3(a, mk3(0.45f, 0.4f, 0.45f));
      auto P = [&](int k) { return mk3(k & 1 ? b.x : a.x, k & 2 ? b.y : a.y, k & 4 ? b.z : a.z); };
      for (const int *q : {(const int[]){0, 1, 3, 2}, (const int[]){4, 6, 7, 5}, (const int[]){0, 4, 5, 1},
                           (const int[]){2, 3, 7, 6}, (const int[]){0, 2, 6, 4}, (const int[]){1, 5, 7, 3}})
        quad(v, P(q[0]), P(q[1]), P(q[2]), P(q[3]));
    }
  }
  if (scene == "turned")
    for (f3 &p : v) {
      f3 const a = unit(mk3(1.0f, 2.0f, 3.0f)), q = scl3(p, 30.0f);  // Rodrigues' rotation by 0.7
      p = add3(add3(scl3(q, std::cos(0.7f)), scl3(cross3(a, q), std::sin(0.7f))),
               scl3(a, dot3(a, q) * (1.0f - std::cos(0.7f))));
    }
  Trees B;
  if (!build(v, B)) return 1;
  int const fine = static_cast<int>(v.size() / 3) - (scene.rfind("ground", 0) == 0 ? 2 : 0);
  long rays = 0, hits = 0, unsettled = 0, differ = 0;
  double n[4] = {0, 0, 0, 0};
  f3 const half = scl3(sub3(B.S.bmax, B.S.bmin), 0.5f);
  float const size = std::fmax(half.x, std::fmax(half.y, half.z));
  auto point = [&](int i, float a, float b) {
    return add3(add3(v[3 * i], scl3(sub3(v[3 * i + 1], v[3 * i]), a)), scl3(sub3(v[3 * i + 2], v[3 * i]), b));
  };
  for (long r = std::atol(argv[2]); r > 0; --r) {
    int const i = static_cast<int>(g() % fine);
    f3 o, d;
    if (kind == "edge" || kind == "far") {
      int const k = static_cast<int>(g() % 3);
      f3 const a = v[3 * i + k], b = v[3 * i + (k + 1) % 3], c = v[3 * i + (k + 2) % 3];
      float const past = std::pow(10.0f, -4 + 3 * U(g)) * (g() % 4 ? 1.0f : -1.0f);
      f3 const e = add3(a, scl3(sub3(b, a), 0.5f + 0.5f * U(g)));
      d = unit(mk3(N(g), N(g), N(g)));
      o = sub3(add3(e, scl3(sub3(e, c), past)), scl3(d, size * std::pow(10.0f, kind == "far" ? 2.75f + 1.75f * U(g) : -0.5f + U(g))));
    } else if (kind == "plane") {
      float const a = 0.5f + 0.5f * U(g), b = (0.5f + 0.5f * U(g)) * (1 - a), c = 0.5f + 0.5f * U(g);
      o = point(i, a, b);
      d = unit(sub3(point(i ^ 1, c, (0.5f + 0.5f * U(g)) * (1 - c)), o));
    } else {
      float const a = 0.5f + 0.5f * U(g), b = (0.5f + 0.5f * U(g)) * (1 - a);
      o = add3(point(static_cast<int>(g() % fine), 0.3f, 0.3f), mk3(0, 0.3f + 0.2f * U(g), 0));
      d = unit(sub3(point(i, a, b), o));
    }
    RayHit w, k = kd_loop(B.S, o, d, kRayTMin, INFINITY, &n[2], &n[3]);
    ++rays;
    hits += k.id >= 0;
    if (!wide_usable(sub3(o, B.S.wide_mid), d, B.S.wide_reach)) continue;
    if (!wide_loop(B, o, d, kRayTMin, INFINITY, w, &n[0], &n[1]))
      ++unsettled;
    else
      differ += std::memcmp(&w, &k, sizeof w) != 0;
  }
  std::printf("%ld %ld %ld %ld %.2f %.2f %.2f %.2f\n", rays, hits, unsettled, differ, n[0] / rays, n[1] / rays,
              n[2] / rays, n[3] / rays);
  return 0;
}
