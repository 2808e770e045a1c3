// Closest-hit entry point (xyzgpu_trace_closest): the batch form of
// Scene::FindIntersection (xyz/core/scene.hpp:277-295).
//
// Persistent warps with per-lane refill (trace_wide in traverse.cuh; counting calls
// and long queues of axis-parallel rays or of tiny scenes walk the kd-tree with
// trace_persistent):
// rays are taken from a global counter as lanes free up, so long and short rays
// balance across lanes and SMs.  Rays are read as two 16-byte vectors and hits
// written as one.
#include <algorithm>

#include "scene.h"
#include "traverse.cuh"

namespace xyzgpu {
namespace {

constexpr int kTraceThreads = 128;

// Rays as 8 floats (o, tmin, d, tmax); hits as (t, f, g, id << 1 | back).
struct ApiSink {
  const float4 *__restrict__ rays;
  float4 *__restrict__ hits;
  uint32_t n_rays, n_hits;
  XYZ_DEV void load(int i, f3 &o, f3 &d, float &tmin, float &tmax) const {
    float4 const a = __ldg(&rays[2 * i + 0]);
    float4 const b = __ldg(&rays[2 * i + 1]);
    o = xyz3(a);
    d = xyz3(b);
    tmin = a.w;
    tmax = b.w;
  }
  XYZ_DEV void store(int i, const RayHit &h) {
    int32_t const code = h.id >= 0 ? ((h.id << 1) | h.back) : -1;
    hits[i] = make_float4(h.id >= 0 ? h.t : 0.0f, h.f, h.g, __int_as_float(code));
    ++n_rays;
    n_hits += h.id >= 0;
  }
};

// Whether 32 rays spread over the queue are all rays that the wide tree cannot
// serve (a grid of axis-parallel rays): every warp of the grid finds the same.
XYZ_DEV bool kd_queue(const DevScene &S, const ApiSink &sink, int n) {
  f3 o, d;
  float tmin, tmax;
  sink.load(static_cast<int>(threadIdx.x & 31) * (n / 32), o, d, tmin, tmax);
  return __all_sync(0xffffffffu, !S.wide || !wide_usable(sub3(o, S.wide_mid), d, S.wide_reach) || !(0.0f <= tmin && tmin <= tmax));
}

// The kd-tree's kernel for such queues: the loop takes 9 CTAs per SM where the
// wide loop takes 8, in which it is 11 to 15 % slower (2^21 axis-parallel rays of
// a 1M-triangle mesh / a room / box stacks: 1,708 / 1,281 / 1,110 us in 9,
// 1,926 / 1,502 / 1,247 in 8).  Launched after the wide kernel where the
// queue fills the grid twice; it finds the queue empty in 2 us otherwise.
__global__ void __launch_bounds__(kTraceThreads, 9)
    k_trace_kd(DevScene S, const float4 *__restrict__ rays, int n, float4 *__restrict__ hits, int *__restrict__ fetch) {
  TraceCount c{0u, 0u, 0u};
  ApiSink sink{rays, hits, 0u, 0u};
  trace_persistent<false>(S, n, fetch, sink, c);
}

// Scenes of a few triangles in a closed room: the walls' boxes overlap in the
// corners and a ray tests most of the triangles, where the kd-tree's cells divide
// them.  Queues that fill the kd kernel's grid go to it: 2^21 rays of a 36-triangle
// room, wide / kd, us: from the middle 300 / 247, from anywhere inside 226 / 193,
// between two surface points 401 / 210, from outside 309 / 155; 4 M camera and
// bounce rays 391 / 377; 262,144 rays 53 / 50, 49 / 47, 73 / 55, 59 / 43.  (Renders,
// whose rays keep together, are 10 to 25 % faster by the wide tree; shorter queues
// too.)
constexpr int kKdTris = 64;

template <bool kCount>
__global__ void __launch_bounds__(kTraceThreads, kCount ? 9 : 8)
    k_trace_api(DevScene S, const float4 *__restrict__ rays, int n, float4 *__restrict__ hits,
                int *__restrict__ fetch, unsigned long long *__restrict__ counts, int kd_follows) {
  int const lane = threadIdx.x & 31;
  TraceCount c{0u, 0u, 0u};
  ApiSink sink{rays, hits, 0u, 0u};
  if constexpr (kCount) {
    trace_persistent<true>(S, n, fetch, sink, c);
  } else {
    if (kd_follows && kd_queue(S, sink, n)) return;
    __shared__ WideList s_list;
    trace_closest_hits(S, n, fetch, sink, s_list);
  }
  uint32_t const n_rays = sink.n_rays, n_hits = sink.n_hits;
  if (kCount) {
    unsigned long long v[5] = {n_rays, c.nodes, c.leaves, c.tris, n_hits};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      unsigned long long x = v[k];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
      if (lane == 0) atomicAdd(&counts[k], x);
    }
  }
}

template <class Kernel>
int grid_for(Kernel k, int &blocks, int device) {
  if (blocks == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTraceThreads, 0) != cudaSuccess ||
        per_sm <= 0)
      per_sm = 4;
    blocks = per_sm * sm_count(device);
  }
  return blocks;
}

}  // namespace

int trace_api_launch(SceneImpl &s, const float *rays, int n, float *hits, cudaStream_t st,
                     xyzgpu_trace_counters *counters) {
  if (counters) *counters = xyzgpu_trace_counters{0, 0, 0, 0, 0};
  if (n == 0) return XYZGPU_OK;
  XYZ_CUDA_TRY(cudaSetDevice(s.device));
  XYZ_CUDA_TRY(cudaMemsetAsync(s.d_fetch, 0, sizeof(int32_t), st));
  const float4 *r4 = reinterpret_cast<const float4 *>(rays);
  float4 *h4 = reinterpret_cast<float4 *>(hits);
  if (counters) {
    XYZ_CUDA_TRY(cudaMemsetAsync(s.d_trace_counts, 0, 8 * sizeof(unsigned long long), st));
    static int counted_grid = 0;
    k_trace_api<true><<<grid_for(k_trace_api<true>, counted_grid, s.device), kTraceThreads, 0, st>>>(
        s.dev, r4, n, h4, s.d_fetch, s.d_trace_counts, 0);
    XYZ_CUDA_TRY(cudaGetLastError());
    unsigned long long c[8];
    XYZ_CUDA_TRY(cudaMemcpyAsync(c, s.d_trace_counts, sizeof(c), cudaMemcpyDeviceToHost, st));
    XYZ_CUDA_TRY(cudaStreamSynchronize(st));
    counters->rays = c[0];
    counters->nodes_visited = c[1];
    counters->leaves_visited = c[2];
    counters->tri_tests = c[3];
    counters->hits = c[4];
  } else {
    static int wide_grid = 0, kd_grid = 0;
    int const kd_full = grid_for(k_trace_kd, kd_grid, s.device);
    if (s.n_tris <= kKdTris && n / kTraceThreads >= kd_full) {
      k_trace_kd<<<kd_full, kTraceThreads, 0, st>>>(s.dev, r4, n, h4, s.d_fetch);
      XYZ_CUDA_TRY(cudaGetLastError());
      return XYZGPU_OK;
    }
    int const full = grid_for(k_trace_api<false>, wide_grid, s.device);
    int const grid = std::min(full, ceil_div(n, kRaysPerCta));
    bool const kd_follows = n / (2 * kTraceThreads) >= full;
    k_trace_api<false><<<grid, kTraceThreads, 0, st>>>(s.dev, r4, n, h4, s.d_fetch, nullptr, kd_follows);
    XYZ_CUDA_TRY(cudaGetLastError());
    if (kd_follows) {
      k_trace_kd<<<kd_full, kTraceThreads, 0, st>>>(s.dev, r4, n, h4, s.d_fetch);
      XYZ_CUDA_TRY(cudaGetLastError());
    }
  }
  return XYZGPU_OK;
}

}  // namespace xyzgpu
