// Host check of the wide tree (xyz_b200/csrc/wide.cuh): builds it from a host
// kd-tree with the device's functions, checks that every triangle has exactly
// one record and that the walk stays inside the tree, and compares the walk's
// closest hit with a test of every triangle.  Prints one line per scene;
// exit code 1 on a difference.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../../xyz_b200/csrc/kdtree.h"
#include "../../xyz_b200/csrc/wide.cuh"

using namespace xyzgpu;

namespace {

struct Tri {
  f3 v0, e1, e2, n;
};

bool test(const Tri &T, f3 o, f3 d, float tmax, float *t_out) {
  float const det = dot3(d, T.n);
  if (std::fabs(det) < kEpsilon) return false;
  float const inv = 1.0f / det;
  f3 const vmo = sub3(T.v0, o);
  float const t = inv * dot3(vmo, T.n);
  if (t < kRayTMin || tmax < t) return false;
  f3 const x = cross3(d, vmo);
  float const f = inv * dot3(T.e2, x);
  if (f < 0 || f > 1) return false;
  float const g = inv * -dot3(T.e1, x);
  if (g < 0 || f + g > 1) return false;
  *t_out = t;
  return true;
}

bool run(const char *name, const std::vector<f3> &V, int rays, int leaf_max) {
  int const n = static_cast<int>(V.size() / 3);
  std::vector<Tri> T(n);
  std::vector<float> trv(9 * static_cast<size_t>(n));
  for (int i = 0; i < n; ++i) {
    T[i].v0 = V[3 * i];
    T[i].e1 = sub3(V[3 * i + 1], V[3 * i]);
    T[i].e2 = sub3(V[3 * i + 2], V[3 * i]);
    T[i].n = cross3(T[i].e2, T[i].e1);
    f3 const p[3] = {T[i].v0, add3(T[i].v0, T[i].e1), add3(T[i].v0, T[i].e2)};
    for (int k = 0; k < 9; ++k) trv[9 * i + k] = comp3(p[k / 3], k % 3);
  }
  BuildConfig cfg;
  cfg.leaf_max_tris = leaf_max;
  cfg.max_depth = kd_resolve_max_depth(0, n);
  cfg.bins = 64;
  cfg.empty_bonus = 0.0f;
  cfg.max_refs = 6ll * n + 1024;
  KdTreeHost K;
  std::string err;
  if (!kd_build_host(trv.data(), n, cfg, &K, &err)) return false;
  int const nn = static_cast<int>(K.nodes.size() / 2);
  std::vector<uint2> nd(nn);
  for (int i = 0; i < nn; ++i) nd[i] = make_uint2(K.nodes[2 * i], K.nodes[2 * i + 1]);
  std::vector<uint4> lo(nn, make_uint4(~0u, ~0u, ~0u, ~0u)), hi(nn, make_uint4(0, 0, 0, 0));
  std::vector<int32_t> first(nn, 0), owner(n);
  for (int i = 0; i < n; ++i) {
    f3 const v0 = T[i].v0, v1 = add3(v0, T[i].e1), v2 = add3(v0, T[i].e2);
    int const l = owner[i] = wide_leaf_of(nd.data(), scl3(add3(add3(v0, v1), v2), 1.0f / 3.0f));
    uint32_t *const L = &lo[l].x, *const H = &hi[l].x;
    for (int k = 0; k < 3; ++k) {
      float const x = comp3(v0, k), y = comp3(v1, k), z = comp3(v2, k);
      L[k] = std::min(L[k], float_key(std::fmin(std::fmin(x, y), z)));
      H[k] = std::max(H[k], float_key(std::fmax(std::fmax(x, y), z)));
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
  WideSets const W{lo.data(), hi.data(), first.data()};
  float reach = 0.0f;
  for (int k = 0; k < 3; ++k) reach = std::max({reach, std::fabs(K.bmin[k]), std::fabs(K.bmax[k])});
  // the device's bound on the node count (wide_max_nodes)
  size_t const max_nodes = n / 4 + (n + n / 4) / 7 + 64;
  std::vector<uint32_t> out(max_nodes * kWideWords);
  std::vector<WideTask> task(max_nodes);
  std::vector<int32_t> dst(n, -1);
  uint32_t nodes = 1, recs = 0, levels = 0;
  bool ok = true;
  task[0] = WideTask{0, 0, n};
  for (uint32_t b = 0; b < nodes && ok; ++levels) {
    uint32_t const e = nodes;
    for (; b < e && ok; ++b)
      wide_make_node(
          nd.data(), W, task[b], reach * kWidePad, &out[static_cast<size_t>(b) * kWideWords],
          [&](int k) {
            uint32_t const r = nodes;
            nodes += k;
            ok = ok && nodes <= max_nodes;
            return r;
          },
          [&](int k) {
            uint32_t const r = recs;
            recs += k;
            return r;
          },
          [&](uint32_t at, WideTask t) {
            if (at < max_nodes) task[at] = t;
          },
          [&](int32_t at, uint32_t r) {
            if (at < 0 || at >= n || dst[at] >= 0)
              ok = false;
            else
              dst[at] = static_cast<int32_t>(r);
          });
  }
  if (!ok || recs != static_cast<uint32_t>(n) || levels > static_cast<uint32_t>(kWideStack)) return false;
  std::vector<int> rec(n, -1), fill(nn, 0);
  for (int i = 0; i < n; ++i) {
    int const p = dst[first[owner[i]] + fill[owner[i]]++];
    if (p < 0 || p >= n || rec[p] >= 0) return false;
    rec[p] = i;
  }
  std::mt19937_64 rng(n + 1);
  std::uniform_real_distribution<float> U(-1, 1);
  std::normal_distribution<float> N;
  int hits = 0, wrong = 0;
  f3 const c = mk3((K.bmin[0] + K.bmax[0]) / 2, (K.bmin[1] + K.bmax[1]) / 2, (K.bmin[2] + K.bmax[2]) / 2);
  f3 const h = mk3((K.bmax[0] - K.bmin[0]) / 2, (K.bmax[1] - K.bmin[1]) / 2, (K.bmax[2] - K.bmin[2]) / 2);
  for (int r = 0; r < rays; ++r) {
    float const far = r % 7 == 0 ? 5.0f : 1.2f;
    f3 const o = mk3(c.x + far * h.x * U(rng), c.y + far * h.y * U(rng), c.z + far * h.z * U(rng));
    f3 d = mk3(N(rng), N(rng), N(rng));
    if (r % 3 == 0) {  // at a triangle's inside, edge or vertex
      const Tri &t = T[rng() % n];
      float const a = r % 2 ? 0.0f : std::fabs(U(rng));
      float const b = r % 5 == 0 ? 0.0f : std::fabs(U(rng)) * (1 - a);
      d = sub3(add3(add3(t.v0, scl3(t.e1, a)), scl3(t.e2, b)), o);
    }
    if (r % 11 == 0) d.x = 0.0f;
    if (r % 13 == 0) d.y = -0.0f;
    float const l = std::sqrt(dot3(d, d));
    if (!(l > 0)) continue;
    d = scl3(d, 1 / l);
    if (!wide_usable(o, d, reach * kWideReach)) continue;
    float best = INFINITY, t;
    for (int i = 0; i < n; ++i)
      if (test(T[i], o, d, best, &t)) best = t;
    float found = INFINITY;
    WideRay const R = wide_ray(o, d);
    uint32_t base = 0, group = (1u << (8 + R.octinv)) | 1u;
    std::vector<uint2> stack;
    for (;;) {
      if (group < 256u) return false;
      int const bit = 31 - __builtin_clz(group);
      group &= ~(1u << bit);
      uint32_t const slot = static_cast<uint32_t>(bit - 8) ^ R.octinv;
      uint32_t const child = base + __builtin_popcount(group & ((1u << slot) - 1u));
      if (child >= nodes || stack.size() >= static_cast<size_t>(kWideStack)) return false;
      if (group >> 8) stack.push_back(make_uint2(base, group));
      const uint32_t *w = &out[static_cast<size_t>(child) * kWideWords];
      uint32_t const hit = wide_test(w, R, kRayTMin, found);
      uint32_t const valid = w[8] >> 8;
      base = w[3];
      group = (wide_order(hit & w[8] & 0xffu, R.octinv) << 8) | (w[8] & 0xffu);
      for (uint32_t th = wide_spread(hit) & valid; th; th &= th - 1) {
        uint32_t const p = w[7] + __builtin_popcount(valid & ((1u << __builtin_ctz(th)) - 1u));
        if (p >= static_cast<uint32_t>(n)) return false;
        if (test(T[rec[p]], o, d, found, &t)) found = t;
      }
      if (group >> 8) continue;
      if (stack.empty()) break;
      base = stack.back().x;
      group = stack.back().y;
      stack.pop_back();
    }
    hits += best < INFINITY;
    wrong += !(found == best);
  }
  std::printf("%s: %d triangles, %u nodes, %u levels, %d hits, %d wrong\n", name, n, nodes, levels, hits, wrong);
  return hits > 0 && wrong == 0;
}

}  // namespace

int main() {
  std::mt19937 g(1);
  std::uniform_real_distribution<float> U(-1, 1);
  bool ok = true;
  for (int n : {1, 2, 3, 4, 5, 8, 9, 25, 200, 2000}) {
    std::vector<f3> v;
    float const size = n > 100 ? 0.1f : 0.5f;
    for (int i = 0; i < n; ++i) {
      f3 const c = mk3(U(g), U(g), U(g));
      for (int k = 0; k < 3; ++k) v.push_back(add3(c, mk3(size * U(g), size * U(g), size * U(g))));
    }
    ok = run("soup", v, 2000, 4) && ok;
  }
  {
    std::vector<f3> v;  // more triangles in one place than any leaf holds
    for (int i = 0; i < 300; ++i)
      for (f3 p : {mk3(0, 0, 0), mk3(1, 0, 0), mk3(0, 1, 0)}) v.push_back(p);
    ok = run("coincident", v, 1000, 4) && ok;
  }
  {
    std::vector<f3> v;  // a flat grid: boxes without thickness, shared edges
    int const m = 24;
    auto P = [&](int a, int b) { return mk3(-1 + 2.0f * a / m, 0, -1 + 2.0f * b / m); };
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j)
        for (f3 p : {P(i, j), P(i + 1, j), P(i + 1, j + 1), P(i, j), P(i + 1, j + 1), P(i, j + 1)}) v.push_back(p);
    ok = run("grid", v, 2000, 8) && ok;
  }
  {
    std::vector<f3> v;  // sizes over five decades
    for (int i = 0; i < 400; ++i) {
      float const s = std::pow(10.0f, 2.5f * U(g) - 1.0f);
      f3 const c = mk3(20 * U(g), 20 * U(g), 20 * U(g));
      for (int k = 0; k < 3; ++k) v.push_back(add3(c, mk3(s * U(g), s * U(g), s * U(g))));
    }
    ok = run("uneven", v, 2000, 4) && ok;
  }
  return ok ? 0 : 1;
}
