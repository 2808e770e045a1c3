// Device kd-tree builder (XYZGPU_BUILD_DEVICE): the binned-SAH build of
// kdbuild_host.cpp performed breadth first on the GPU, one level at a time,
// producing the identical flattened tree (same float operations in the same
// order, --fmad=false; integer histograms and scans are order independent).
//
// Per level (m nodes, R references, each node's references contiguous):
//   classify   nodes with >= kBigRefs references are listed ("big"): their
//              histograms, left / right counts and emit run on up to 128 CTAs
//              each (slices of the references), the SAH decision on one CTA
//              each; the rest get one warp each
//   decide     binned start/end histograms per axis in shared memory
//              (shared-memory atomics), exclusive prefix per axis, SAH cost of
//              every candidate plane, arg-min with the host's tie-break
//              (lowest axis, then lowest plane), exact left/right counts
//   scan       exclusive scan over nodes of (split, leaf refs, next refs,
//              empty leaf) -> child pair index, leaf offset, child ref offset
//   emit       node words, next-level node bounds and ranges, and a stable
//              scatter of references into the children (ballot / block scans,
//              and per-slice counts for big nodes, keep the parent's order) or
//              into the leaf reference array
// The host reads once per level (the scan totals and the next level's big-node
// count) to size the next level; everything else stays on the device.
//
// Layout (kd_layout_depth_first, after either builder): the breadth-first
// array is permuted so that every subtree occupies one contiguous range, in
// depth-first order of child pairs: a pair (first, second) is followed by
// the first child's descendants, then the second's.  A ray descending into
// the first child finds that child's pair in the next bytes, usually the
// same 32-byte sector, and rays working in one region of space read one
// region of the array.  Node words keep their format; only child indices
// change.
//
// The same two sweeps over the levels give the wide tree (wide.cuh) its
// triangle sets: boxes and counts of the kd nodes from the deepest level up,
// positions in depth-first order from the root down; k_wide_nodes then builds
// the wide nodes level by level and k_wide_tris writes the triangle records.
#include <algorithm>
#include <cstddef>
#include <vector>

#include "scene.h"
#include "wide.cuh"

namespace xyzgpu {
namespace {

// References from which a node is split by CTAs: a warp needs 30 us for the
// decision and 65 us for the emit of 2,000 references (9 and 10 us for 500), the
// CTAs' five launches 20 us in all.  Device time of the build kernels below,
// 247,042 triangles: 1,200 us at 2,048, 1,060 at 1,024, 920 at 512 (the
// decision as it was before), at 256 as at 512.
constexpr int kBigRefs = 512;
// References a lane of the small nodes' kernels has in flight: both kernels 696
// us at 2, 725 at 4 (registers).
constexpr int kRefUnroll = 2;
constexpr int kBigThreads = 256;
constexpr int kBigSlicesMax = 128;     // CTAs per big node when emitting
constexpr int kBigSliceBudget = 1024;  // CTAs per emit launch (about)
constexpr int kWarpsPerBlock = 4;
constexpr int kScanThreads = 256;
constexpr int kFirstLevelNodes = 8192;  // 0.6 MB a set of level arrays
constexpr int kScanPerThread = 8;
constexpr int kScanPerBlock = kScanThreads * kScanPerThread;

struct RefArrays {
  int32_t *tri;
  float *lo[3];
  float *hi[3];
};

struct LevelArrays {
  float4 *blo, *bhi;  // node bounds
  int32_t *begin, *count;
  int32_t *axis;      // -1: leaf
  float *plane;
  int32_t *nl, *nr;
  uint4 *scan;        // in: (split, leaf refs, next refs, empty leaf); out: exclusive prefix
};

// What the host reads of a level.
struct LevelTotals {
  uint4 scan;        // splits, leaf refs, next refs, empty leaves
  int32_t next_big;  // the next level's big nodes
  int32_t pad[3];
};

struct BuildArgs {
  int leaf_max, max_depth, bins, depth;
  float ct, ci, eb;
};

XYZ_DEV float half_area3(float e0, float e1, float e2) { return e0 * e1 + e1 * e2 + e2 * e0; }
XYZ_DEV float comp4(float4 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

__global__ void k_init_refs(const float4 *__restrict__ tri, int n, RefArrays R) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 const a = tri[3 * i], b = tri[3 * i + 1], c = tri[3 * i + 2];
    // vertices as the intersection test sees them: v0, v0 + e1, v0 + e2
    float const v[3][3] = {{a.x, a.y, a.z}, {a.x + b.x, a.y + b.y, a.z + b.z},
                           {a.x + c.x, a.y + c.y, a.z + c.z}};
    R.tri[i] = i;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      R.lo[k][i] = fminf(fminf(v[0][k], v[1][k]), v[2][k]);
      R.hi[k][i] = fmaxf(fmaxf(v[0][k], v[1][k]), v[2][k]);
    }
  }
}

__global__ void k_init_root(LevelArrays L, float4 lo, float4 hi, int n, int32_t *big_count) {
  L.blo[0] = lo;
  L.bhi[0] = hi;
  L.begin[0] = 0;
  L.count[0] = n;
  *big_count = 0;
}

__host__ __device__ inline bool eligible(const BuildArgs &a, int n) { return n > a.leaf_max && a.depth < a.max_depth; }

__global__ void k_classify(LevelArrays L, int m, BuildArgs a, int32_t *big_list, int32_t *big_count) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
    int const n = L.count[j];
    if (n >= kBigRefs && eligible(a, n)) big_list[atomicAdd(big_count, 1)] = j;
  }
}

// SAH over the exclusive prefix sums pre[a][0][i] (starts) and pre[a][1][i]
// (ends) of bins [0, i).  Candidate c = a * (B - 1) + (i - 1).  Returns the
// cost; +inf for invalid candidates.
XYZ_DEV float candidate_cost(const BuildArgs &A, int B, const uint32_t *pre, int c, int n, const float ext[3],
                             float4 lo4, float4 hi4, float sa, float *plane_out, int *nl_out) {
  int const a = c / (B - 1);
  int const i = c - a * (B - 1) + 1;
  if (!(ext[a] > 0.0f)) return INFINITY;
  float const lo = comp4(lo4, a);
  float const step = ext[a] / static_cast<float>(B);
  float const plane = lo + static_cast<float>(i) * step;
  uint32_t const nl = pre[(a * 2 + 0) * (kKdMaxBins + 1) + i];
  uint32_t const ended = pre[(a * 2 + 1) * (kKdMaxBins + 1) + i];
  int const nr = n - static_cast<int>(ended);
  float el[3] = {ext[0], ext[1], ext[2]};
  float er[3] = {ext[0], ext[1], ext[2]};
  el[a] = plane - lo;
  er[a] = comp4(hi4, a) - plane;
  float const sal = half_area3(el[0], el[1], el[2]);
  float const sar = half_area3(er[0], er[1], er[2]);
  float cost = A.ct + A.ci * (sal * static_cast<float>(nl) + sar * static_cast<float>(nr)) / sa;
  if (nl == 0 || nr == 0) cost = cost * (1.0f - A.eb);
  *plane_out = plane;
  *nl_out = static_cast<int>(nl);
  return cost;
}

XYZ_DEV void classify_ref(float lo, float hi, float plane, bool *l, bool *r) {
  bool const flat_on = (lo == plane) && (hi == plane);
  *l = (lo < plane) || flat_on;
  *r = (hi > plane) || flat_on;
}

XYZ_DEV int bin_of(float x, float lo, float scale, int B) {
  int b = static_cast<int>((x - lo) * scale);
  return min(max(b, 0), B - 1);
}

// Smaller (cost, candidate) first.
XYZ_DEV bool better(float c0, int i0, float c1, int i1) { return c0 < c1 || (c0 == c1 && i0 < i1); }

// ---- decide: one warp per small node
// The cost of candidate i of axis kA: candidate_cost with the axis known.
template <int kA>
XYZ_DEV float plane_cost(const BuildArgs &A, int i, int nl, int nr, f3 ext, float lo, float hi, float step, float sa) {
  float const plane = lo + static_cast<float>(i) * step;
  float const dl = plane - lo, dr = hi - plane;
  float const sal = half_area3(kA == 0 ? dl : ext.x, kA == 1 ? dl : ext.y, kA == 2 ? dl : ext.z);
  float const sar = half_area3(kA == 0 ? dr : ext.x, kA == 1 ? dr : ext.y, kA == 2 ? dr : ext.z);
  float cost = A.ct + A.ci * (sal * static_cast<float>(nl) + sar * static_cast<float>(nr)) / sa;
  if (nl == 0 || nr == 0) cost = cost * (1.0f - A.eb);
  return cost;
}

// The order of finite costs and infinity as unsigned numbers; a NaN comes last.
XYZ_DEV uint32_t cost_key(float c) {
  if (!(c == c)) return 0xffffffffu;
  uint32_t const u = __float_as_uint(c + 0.0f);
  return u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
}
XYZ_DEV float key_cost(uint32_t k) { return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xffffffffu)); }

// Deep levels hold 100,000 nodes of a few references and are bound by
// instructions; shallow ones hold a few hundred nodes of up to kBigRefs, whose
// warps wait for their loads.  So: up to 32 bins, lane i holds plane i + 1 of
// each axis and the counts before it, starts and ends packed in 16 bits each
// (three histograms and scans instead of six, nothing written back); the loads
// of kRefUnroll references are in flight together; up to that many stay in
// registers for the children's counts.  All 30 levels of a 247,042-triangle
// build: 618 -> 400 us (843 with nodes of up to 2,047 references).
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    k_decide_small(LevelArrays L, int m, RefArrays R, BuildArgs A, LevelTotals *totals, int32_t *big_count) {
  static_assert(kBigRefs <= 0xffff, "packed counts");
  __shared__ uint32_t hist[kWarpsPerBlock][3 * (kKdMaxBins + 1)];
  // counters of the next level (this level's list is complete)
  if (blockIdx.x == 0 && threadIdx.x == 0) totals->next_big = *big_count = 0;
  int const lane = threadIdx.x & 31;
  int const wib = threadIdx.x >> 5;
  uint32_t *h = hist[wib];
  int const warp = blockIdx.x * kWarpsPerBlock + wib;
  int const nwarps = gridDim.x * kWarpsPerBlock;
  for (int j = warp; j < m; j += nwarps) {
    int const n = L.count[j];
    int const B = kd_node_bins(A.bins, n);
    if (n >= kBigRefs && eligible(A, n)) continue;  // a CTA decides this node
    float4 const lo4 = L.blo[j], hi4 = L.bhi[j];
    int const rb = L.begin[j];
    f3 const ext = mk3(hi4.x - lo4.x, hi4.y - lo4.y, hi4.z - lo4.z);
    float const sa = half_area3(ext.x, ext.y, ext.z);
    if (!eligible(A, n) || !(sa > 0.0f)) {
      if (lane == 0) {
        L.axis[j] = -1;
        L.nl[j] = L.nr[j] = 0;
      }
      continue;
    }
    float const bins = static_cast<float>(B);
    f3 const scale = mk3(bins / ext.x, bins / ext.y, bins / ext.z);
    f3 const step = mk3(ext.x / bins, ext.y / bins, ext.z / bins);
    // the three rows' first B entries (the rest is never read)
    for (int t = lane; t < B; t += 32) h[t] = h[kKdMaxBins + 1 + t] = h[2 * (kKdMaxBins + 1) + t] = 0u;
    __syncwarp();
    float v[kRefUnroll][6];
    for (int r0 = 0; r0 < n; r0 += 32 * kRefUnroll) {
#pragma unroll
      for (int u = 0; u < kRefUnroll; ++u) {
        int const r = rb + min(r0 + 32 * u + lane, n - 1);
        if (u == 0 || r0 + 32 * u < n) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            v[u][2 * a] = R.lo[a][r];
            v[u][2 * a + 1] = R.hi[a][r];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kRefUnroll; ++u) {
        if (r0 + 32 * u + lane < n) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            float const e = a == 0 ? ext.x : (a == 1 ? ext.y : ext.z);
            float const o = comp4(lo4, a), sc = a == 0 ? scale.x : (a == 1 ? scale.y : scale.z);
            if (e > 0.0f) {
              atomicAdd(&h[a * (kKdMaxBins + 1) + bin_of(v[u][2 * a], o, sc, B)], 1u);
              atomicAdd(&h[a * (kKdMaxBins + 1) + bin_of(v[u][2 * a + 1], o, sc, B)], 0x10000u);
            }
          }
        }
      }
    }
    __syncwarp();
    // plane i + 1 has the bins up to i on its left: inclusive scans over the
    // lanes, 32 bins at a time
    float best = INFINITY;
    int best_c = 0x7fffffff;
    uint32_t carry[3] = {0u, 0u, 0u};
    for (int base = 0; base < B - 1; base += 32) {
      int const i = base + lane + 1;
      uint32_t incl[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) incl[a] = i <= B ? h[a * (kKdMaxBins + 1) + i - 1] : 0u;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          uint32_t const t = __shfl_up_sync(0xffffffffu, incl[a], off);
          if (lane >= off) incl[a] += t;
        }
#pragma unroll
      for (int a = 0; a < 3; ++a) incl[a] += carry[a];
      if (i < B) {
        auto consider = [&](float e, float cost, int c) {
          if (e > 0.0f && better(cost, c, best, best_c)) {
            best = cost;
            best_c = c;
          }
        };
        auto left = [&](int a) { return static_cast<int>(incl[a] & 0xffffu); };
        auto right = [&](int a) { return n - static_cast<int>(incl[a] >> 16); };
        consider(ext.x, plane_cost<0>(A, i, left(0), right(0), ext, lo4.x, hi4.x, step.x, sa), i - 1);
        consider(ext.y, plane_cost<1>(A, i, left(1), right(1), ext, lo4.y, hi4.y, step.y, sa), (B - 1) + i - 1);
        consider(ext.z, plane_cost<2>(A, i, left(2), right(2), ext, lo4.z, hi4.z, step.z, sa), 2 * (B - 1) + i - 1);
      }
      if (base + 32 < B - 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) carry[a] = __shfl_sync(0xffffffffu, incl[a], 31);
    }
    // smallest cost, then smallest candidate
    uint32_t const key = cost_key(best);
    uint32_t const min_key = __reduce_min_sync(0xffffffffu, key);
    best_c = static_cast<int>(
        __reduce_min_sync(0xffffffffu, key == min_key ? static_cast<uint32_t>(best_c) : 0x7fffffffu));
    int axis = -1;
    float plane = 0.0f;
    int nl = 0, nr = 0;
    if (key_cost(min_key) < A.ci * static_cast<float>(n)) {
      axis = best_c / (B - 1);
      int const i = best_c - axis * (B - 1) + 1;
      float const s = axis == 0 ? step.x : (axis == 1 ? step.y : step.z);
      plane = comp4(lo4, axis) + static_cast<float>(i) * s;
      if (n <= 32 * kRefUnroll) {
#pragma unroll
        for (int u = 0; u < kRefUnroll; ++u) {
          float const lo = axis == 0 ? v[u][0] : (axis == 1 ? v[u][2] : v[u][4]);
          float const hi = axis == 0 ? v[u][1] : (axis == 1 ? v[u][3] : v[u][5]);
          bool l = false, r = false;
          if (32 * u + lane < n) classify_ref(lo, hi, plane, &l, &r);
          nl += __popc(__ballot_sync(0xffffffffu, l));
          nr += __popc(__ballot_sync(0xffffffffu, r));
        }
      } else {
        const float *const lo = rb + (axis == 0 ? R.lo[0] : (axis == 1 ? R.lo[1] : R.lo[2]));
        const float *const hi = rb + (axis == 0 ? R.hi[0] : (axis == 1 ? R.hi[1] : R.hi[2]));
#pragma unroll 4
        for (int r = lane; r < n; r += 32) {
          bool l, rr;
          classify_ref(lo[r], hi[r], plane, &l, &rr);
          nl += l;
          nr += rr;
        }
        nl = __reduce_add_sync(0xffffffffu, nl);
        nr = __reduce_add_sync(0xffffffffu, nr);
      }
    }
    if (lane == 0) {
      L.axis[j] = axis;
      L.plane[j] = plane;
      L.nl[j] = nl;
      L.nr[j] = nr;
    }
    __syncwarp();
  }
}

// ---- decide: one CTA per big node
// Big nodes use `slices` CTAs each for their O(n) passes; CTA g of a node
// takes the g-th contiguous slice of its references.
__device__ __forceinline__ void big_slice(int n, int slices, int g, int *b, int *e) {
  int const s = (n + slices - 1) / slices;
  *b = min(n, g * s);
  *e = min(n, *b + s);
}

constexpr int kHistWords = 3 * 2 * (kKdMaxBins + 1);

// Start / end bin histograms of a big node, one slice per CTA, added into the
// node's histogram in global memory (integer counts: the sum does not depend
// on the order of the slices).
__global__ void __launch_bounds__(kBigThreads) k_decide_big_hist(LevelArrays L, const int32_t *__restrict__ big_list,
                                                                 RefArrays R, BuildArgs A, int slices,
                                                                 uint32_t *__restrict__ gh) {
  __shared__ uint32_t h[kHistWords];
  int const ib = blockIdx.x / slices, g = blockIdx.x % slices;
  int const j = big_list[ib];
  int const n = L.count[j];
  int const B = kd_node_bins(A.bins, n);
  int const tid = threadIdx.x;
  float4 const lo4 = L.blo[j], hi4 = L.bhi[j];
  float const ext[3] = {hi4.x - lo4.x, hi4.y - lo4.y, hi4.z - lo4.z};
  if (!(half_area3(ext[0], ext[1], ext[2]) > 0.0f)) return;  // k_decide_big makes it a leaf
  for (int t = tid; t < kHistWords; t += kBigThreads) h[t] = 0u;
  __syncthreads();
  int b, e;
  big_slice(n, slices, g, &b, &e);
  int const rb = L.begin[j];
  for (int a = 0; a < 3; ++a) {
    if (!(ext[a] > 0.0f)) continue;
    float const scale = static_cast<float>(B) / ext[a];
    float const lo = comp4(lo4, a);
    for (int r = b + tid; r < e; r += kBigThreads) {
      int const b0 = bin_of(R.lo[a][rb + r], lo, scale, B);
      int const b1 = bin_of(R.hi[a][rb + r], lo, scale, B);
      atomicAdd(&h[(a * 2 + 0) * (kKdMaxBins + 1) + b0], 1u);
      atomicAdd(&h[(a * 2 + 1) * (kKdMaxBins + 1) + b1], 1u);
    }
  }
  __syncthreads();
  for (int t = tid; t < kHistWords; t += kBigThreads)
    if (h[t]) atomicAdd(&gh[static_cast<int64_t>(ib) * kHistWords + t], h[t]);
}

__global__ void __launch_bounds__(kBigThreads)
    k_decide_big(LevelArrays L, const int32_t *__restrict__ big_list, BuildArgs A,
                 const uint32_t *__restrict__ gh) {
  __shared__ uint32_t h[kHistWords];
  __shared__ float s_cost[kBigThreads / 32];
  __shared__ int s_idx[kBigThreads / 32];
  int const j = big_list[blockIdx.x];
  int const n = L.count[j];
  int const B = kd_node_bins(A.bins, n);
  int const tid = threadIdx.x;
  float4 const lo4 = L.blo[j], hi4 = L.bhi[j];
  float const ext[3] = {hi4.x - lo4.x, hi4.y - lo4.y, hi4.z - lo4.z};
  float const sa = half_area3(ext[0], ext[1], ext[2]);
  if (!(sa > 0.0f)) {
    if (tid == 0) {
      L.axis[j] = -1;
      L.nl[j] = L.nr[j] = 0;
    }
    return;
  }
  // the node's histograms, summed over its slices by k_decide_big_hist
  for (int t = tid; t < kHistWords; t += kBigThreads) h[t] = gh[static_cast<int64_t>(blockIdx.x) * kHistWords + t];
  __syncthreads();
  if (tid < 6) {
    uint32_t *row = h + tid * (kKdMaxBins + 1);
    uint32_t acc = 0u;
    for (int b = 0; b < B; ++b) {
      uint32_t const v = row[b];
      row[b] = acc;
      acc += v;
    }
    row[B] = acc;
  }
  __syncthreads();
  float best = INFINITY;
  int best_c = 0x7fffffff;
  for (int c = tid; c < 3 * (B - 1); c += kBigThreads) {
    float pl;
    int nl;
    float const cost = candidate_cost(A, B, h, c, n, ext, lo4, hi4, sa, &pl, &nl);
    if (better(cost, c, best, best_c)) {
      best = cost;
      best_c = c;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    float const oc = __shfl_xor_sync(0xffffffffu, best, off);
    int const oi = __shfl_xor_sync(0xffffffffu, best_c, off);
    if (better(oc, oi, best, best_c)) {
      best = oc;
      best_c = oi;
    }
  }
  if ((tid & 31) == 0) {
    s_cost[tid >> 5] = best;
    s_idx[tid >> 5] = best_c;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kBigThreads / 32; ++w)
      if (better(s_cost[w], s_idx[w], best, best_c)) {
        best = s_cost[w];
        best_c = s_idx[w];
      }
    s_cost[0] = best;
    s_idx[0] = best_c;
  }
  __syncthreads();
  best = s_cost[0];
  best_c = s_idx[0];
  int axis = -1;
  float plane = 0.0f;
  if (best < A.ci * static_cast<float>(n)) {
    int nl_bin;
    candidate_cost(A, B, h, best_c, n, ext, lo4, hi4, sa, &plane, &nl_bin);
    axis = best_c / (B - 1);
  }
  // exact left / right counts: k_emit_big_count per slice, k_big_totals per node
  if (tid == 0) {
    L.axis[j] = axis;
    L.plane[j] = plane;
  }
}

__global__ void k_flags(LevelArrays L, int m, int force_leaves, BuildArgs next, LevelTotals *totals) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
    if (force_leaves) L.axis[j] = -1;
    int const split = L.axis[j] >= 0;
    int const n = L.count[j];
    if (split) {
      int const nl = L.nl[j], nr = L.nr[j];
      int const big = (nl >= kBigRefs && eligible(next, nl)) + (nr >= kBigRefs && eligible(next, nr));
      if (big) atomicAdd(&totals->next_big, big);
    }
    L.scan[j] = make_uint4(split, split ? 0u : static_cast<uint32_t>(n),
                           split ? static_cast<uint32_t>(L.nl[j] + L.nr[j]) : 0u, (!split && n == 0) ? 1u : 0u);
  }
}

// ---- exclusive scan of uint4 (three kernels)
XYZ_DEV uint4 add4(uint4 a, uint4 b) { return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

XYZ_DEV uint4 block_exclusive(uint4 v, uint4 *total) {
  __shared__ uint4 warp_sums[kScanThreads / 32];
  int const lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint4 inc = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    uint4 o;
    o.x = __shfl_up_sync(0xffffffffu, inc.x, off);
    o.y = __shfl_up_sync(0xffffffffu, inc.y, off);
    o.z = __shfl_up_sync(0xffffffffu, inc.z, off);
    o.w = __shfl_up_sync(0xffffffffu, inc.w, off);
    if (lane >= off) inc = add4(inc, o);
  }
  if (lane == 31) warp_sums[w] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint4 acc = make_uint4(0, 0, 0, 0);
    for (int k = 0; k < kScanThreads / 32; ++k) {
      uint4 const s = warp_sums[k];
      warp_sums[k] = acc;
      acc = add4(acc, s);
    }
    *total = acc;
  }
  __syncthreads();
  uint4 const ex = make_uint4(inc.x - v.x, inc.y - v.y, inc.z - v.z, inc.w - v.w);
  uint4 const r = add4(ex, warp_sums[w]);
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_blocks(uint4 *data, int m, uint4 *block_sums) {
  __shared__ uint4 total;
  int const base = blockIdx.x * kScanPerBlock + threadIdx.x * kScanPerThread;
  uint4 loc[kScanPerThread];
  uint4 sum = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int k = 0; k < kScanPerThread; ++k) {
    loc[k] = base + k < m ? data[base + k] : make_uint4(0, 0, 0, 0);
    sum = add4(sum, loc[k]);
  }
  uint4 off = block_exclusive(sum, &total);
#pragma unroll
  for (int k = 0; k < kScanPerThread; ++k) {
    if (base + k < m) data[base + k] = off;
    off = add4(off, loc[k]);
  }
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_totals(uint4 *block_sums, int nb, uint4 *grand) {
  __shared__ uint4 total;
  uint4 carry = make_uint4(0, 0, 0, 0);
  for (int base = 0; base < nb; base += kScanThreads) {
    int const i = base + threadIdx.x;
    uint4 const v = i < nb ? block_sums[i] : make_uint4(0, 0, 0, 0);
    uint4 const ex = block_exclusive(v, &total);
    if (i < nb) block_sums[i] = add4(ex, carry);
    __syncthreads();
    carry = add4(carry, total);
    __syncthreads();
  }
  if (threadIdx.x == 0) *grand = carry;
}

__global__ void k_scan_add(uint4 *data, int m, const uint4 *block_sums) {
  int const i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) data[i] = add4(data[i], block_sums[i / kScanPerBlock]);
}

// ---- emit
struct EmitArgs {
  LevelArrays L, N;  // this level, next level
  RefArrays R, RN;   // this level's refs, next level's refs
  uint2 *nodes;
  int32_t *leaf_refs;
  int64_t level_base, next_base, leaf_base;
  int m;
};

XYZ_DEV void write_split_node(const EmitArgs &E, int j, int axis, float plane) {
  uint4 const sc = E.L.scan[j];
  int64_t const child = E.next_base + 2 * static_cast<int64_t>(sc.x);
  E.nodes[E.level_base + j] = make_uint2(__float_as_uint(plane),
                                         (static_cast<uint32_t>(child) << 2) | static_cast<uint32_t>(axis));
  int const c = 2 * static_cast<int>(sc.x);
  float4 lo = E.L.blo[j], hi = E.L.bhi[j];
  float4 hl = hi, lr = lo;
  if (axis == 0) hl.x = plane, lr.x = plane;
  if (axis == 1) hl.y = plane, lr.y = plane;
  if (axis == 2) hl.z = plane, lr.z = plane;
  E.N.blo[c] = lo;
  E.N.bhi[c] = hl;
  E.N.blo[c + 1] = lr;
  E.N.bhi[c + 1] = hi;
  E.N.begin[c] = static_cast<int32_t>(sc.z);
  E.N.count[c] = E.L.nl[j];
  E.N.begin[c + 1] = static_cast<int32_t>(sc.z) + E.L.nl[j];
  E.N.count[c + 1] = E.L.nr[j];
}

// One reference of a child: its box (lo, hi per axis) cut at the plane.
XYZ_DEV void put_ref(const RefArrays &D, int dst, int32_t tri, const float *box, int axis, float plane, bool left) {
  D.tri[dst] = tri;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float lo = box[2 * k], hi = box[2 * k + 1];
    if (k == axis) {
      if (left)
        hi = fminf(hi, plane);
      else
        lo = fmaxf(lo, plane);
    }
    D.lo[k][dst] = lo;
    D.hi[k][dst] = hi;
  }
}

XYZ_DEV void write_ref(const RefArrays &D, int dst, const RefArrays &S, int src, int axis, float plane,
                       bool left) {
  float box[6];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    box[2 * k] = S.lo[k][src];
    box[2 * k + 1] = S.hi[k][src];
  }
  put_ref(D, dst, S.tri[src], box, axis, plane, left);
}

__global__ void __launch_bounds__(32 * kWarpsPerBlock) k_emit_small(EmitArgs E, BuildArgs A) {
  int const lane = threadIdx.x & 31;
  int const warp = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  int const nwarps = gridDim.x * kWarpsPerBlock;
  for (int j = warp; j < E.m; j += nwarps) {
    int const n = E.L.count[j];
    if (n >= kBigRefs && eligible(A, n)) continue;  // emitted by k_emit_big
    int const axis = E.L.axis[j];
    int const rb = E.L.begin[j];
    if (axis < 0) {
      uint4 const sc = E.L.scan[j];
      int64_t const off = E.leaf_base + sc.y;
      if (lane == 0)
        E.nodes[E.level_base + j] = make_uint2(static_cast<uint32_t>(off),
                                               (static_cast<uint32_t>(n) << 2) | kKdLeafTag);
      for (int r = lane; r < n; r += 32) E.leaf_refs[off + r] = E.R.tri[rb + r];
      continue;
    }
    float const plane = E.L.plane[j];
    if (lane == 0) write_split_node(E, j, axis, plane);
    int const lbase = static_cast<int>(E.L.scan[j].z);
    int const rbase = lbase + E.L.nl[j];
    int nl_run = 0, nr_run = 0;
    unsigned const below = (1u << lane) - 1u;
    for (int r0 = 0; r0 < n; r0 += 32 * kRefUnroll) {
      float v[kRefUnroll][6];
      int32_t tri[kRefUnroll];
#pragma unroll
      for (int u = 0; u < kRefUnroll; ++u) {
        int const r = rb + min(r0 + 32 * u + lane, n - 1);
        if (u > 0 && r0 + 32 * u >= n) break;  // the same on every lane
        tri[u] = E.R.tri[r];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          v[u][2 * k] = E.R.lo[k][r];
          v[u][2 * k + 1] = E.R.hi[k][r];
        }
      }
#pragma unroll
      for (int u = 0; u < kRefUnroll; ++u) {
        if (u > 0 && r0 + 32 * u >= n) break;
        float const *const w = v[u];
        float const lo = axis == 0 ? w[0] : (axis == 1 ? w[2] : w[4]);
        float const hi = axis == 0 ? w[1] : (axis == 1 ? w[3] : w[5]);
        bool l = false, rr = false;
        if (r0 + 32 * u + lane < n) classify_ref(lo, hi, plane, &l, &rr);
        unsigned const ml = __ballot_sync(0xffffffffu, l);
        unsigned const mr = __ballot_sync(0xffffffffu, rr);
        if (l) put_ref(E.RN, lbase + nl_run + __popc(ml & below), tri[u], w, axis, plane, true);
        if (rr) put_ref(E.RN, rbase + nr_run + __popc(mr & below), tri[u], w, axis, plane, false);
        nl_run += __popc(ml);
        nr_run += __popc(mr);
      }
    }
  }
}

// Big nodes are emitted by `slices` CTAs each: CTA g of a node takes the g-th
// contiguous slice of its references.  A counting pass records each slice's
// left and right counts; the scatter pass starts each slice after the counts
// of the node's earlier slices and keeps the order within the slice, so the
// children receive the parent's references in the parent's order, as from a
// single CTA.

__global__ void __launch_bounds__(kBigThreads)
    k_emit_big_count(LevelArrays L, RefArrays R, const int32_t *__restrict__ big_list, int slices,
                     int2 *__restrict__ cnt) {
  __shared__ int s_red[2][kBigThreads / 32];
  int const j = big_list[blockIdx.x / slices], g = blockIdx.x % slices;
  int const axis = L.axis[j];
  if (axis < 0) return;  // leaf: its references are copied, not counted
  int const n = L.count[j], rb = L.begin[j];
  float const plane = L.plane[j];
  int b, e;
  big_slice(n, slices, g, &b, &e);
  int const tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int cl = 0, cr = 0;
  for (int r = b + tid; r < e; r += kBigThreads) {
    bool l = false, rr = false;
    classify_ref(R.lo[axis][rb + r], R.hi[axis][rb + r], plane, &l, &rr);
    cl += l;
    cr += rr;
  }
  for (int o = 16; o > 0; o >>= 1) {
    cl += __shfl_down_sync(0xffffffffu, cl, o);
    cr += __shfl_down_sync(0xffffffffu, cr, o);
  }
  if (lane == 0) {
    s_red[0][w] = cl;
    s_red[1][w] = cr;
  }
  __syncthreads();
  if (tid == 0) {
    int tl = 0, tr = 0;
    for (int k = 0; k < kBigThreads / 32; ++k) {
      tl += s_red[0][k];
      tr += s_red[1][k];
    }
    cnt[blockIdx.x] = make_int2(tl, tr);
  }
}

// A big node's exact left / right reference counts: the sum of its slices'.
__global__ void k_big_totals(LevelArrays L, const int32_t *__restrict__ big_list, int slices,
                             const int2 *__restrict__ cnt) {
  int const j = big_list[blockIdx.x];
  int const lane = threadIdx.x;
  bool const split = L.axis[j] >= 0;
  int nl = 0, nr = 0;
  if (split)
    for (int k = lane; k < slices; k += 32) {
      int2 const c = cnt[blockIdx.x * slices + k];
      nl += c.x;
      nr += c.y;
    }
  for (int o = 16; o > 0; o >>= 1) {
    nl += __shfl_down_sync(0xffffffffu, nl, o);
    nr += __shfl_down_sync(0xffffffffu, nr, o);
  }
  if (lane == 0) {
    L.nl[j] = split ? nl : 0;
    L.nr[j] = split ? nr : 0;
  }
}

__global__ void __launch_bounds__(kBigThreads)
    k_emit_big(EmitArgs E, const int32_t *__restrict__ big_list, int slices, const int2 *__restrict__ cnt) {
  __shared__ int s_warp[2][kBigThreads / 32];
  __shared__ int s_run[2];
  int const first = (blockIdx.x / slices) * slices, g = blockIdx.x - first;
  int const j = big_list[blockIdx.x / slices];
  int const n = E.L.count[j];
  int const axis = E.L.axis[j];
  int const rb = E.L.begin[j];
  int const tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int b, e;
  big_slice(n, slices, g, &b, &e);
  if (axis < 0) {
    uint4 const sc = E.L.scan[j];
    int64_t const off = E.leaf_base + sc.y;
    if (g == 0 && tid == 0)
      E.nodes[E.level_base + j] = make_uint2(static_cast<uint32_t>(off),
                                             (static_cast<uint32_t>(n) << 2) | kKdLeafTag);
    for (int r = b + tid; r < e; r += kBigThreads) E.leaf_refs[off + r] = E.R.tri[rb + r];
    return;
  }
  float const plane = E.L.plane[j];
  if (g == 0 && tid == 0) write_split_node(E, j, axis, plane);
  if (w == 0) {
    // references of the node's earlier slices
    int pl = 0, pr = 0;
    for (int k = lane; k < g; k += 32) {
      int2 const c = cnt[first + k];
      pl += c.x;
      pr += c.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
      pl += __shfl_down_sync(0xffffffffu, pl, o);
      pr += __shfl_down_sync(0xffffffffu, pr, o);
    }
    if (lane == 0) {
      s_run[0] = pl;
      s_run[1] = pr;
    }
  }
  __syncthreads();
  int const lbase = static_cast<int>(E.L.scan[j].z);
  int const rbase = lbase + E.L.nl[j];
  for (int r0 = b; r0 < e; r0 += kBigThreads) {
    int const r = r0 + tid;
    bool l = false, rr = false;
    if (r < e) classify_ref(E.R.lo[axis][rb + r], E.R.hi[axis][rb + r], plane, &l, &rr);
    unsigned const ml = __ballot_sync(0xffffffffu, l);
    unsigned const mr = __ballot_sync(0xffffffffu, rr);
    if (lane == 0) {
      s_warp[0][w] = __popc(ml);
      s_warp[1][w] = __popc(mr);
    }
    __syncthreads();
    int pl = s_run[0], pr = s_run[1];
    for (int k = 0; k < w; ++k) {
      pl += s_warp[0][k];
      pr += s_warp[1][k];
    }
    unsigned const below = (1u << lane) - 1u;
    if (l) write_ref(E.RN, lbase + pl + __popc(ml & below), E.R, rb + r, axis, plane, true);
    if (rr) write_ref(E.RN, rbase + pr + __popc(mr & below), E.R, rb + r, axis, plane, false);
    __syncthreads();
    if (tid == 0) {
      for (int k = 0; k < kBigThreads / 32; ++k) {
        s_run[0] += s_warp[0][k];
        s_run[1] += s_warp[1][k];
      }
    }
    __syncthreads();
  }
}

// ---- device buffers
// Device buffer from the stream-ordered pool (the scene's build stream).
template <class T>
struct DevBuf {
  T *p = nullptr;
  int64_t cap = 0;
  cudaStream_t st = nullptr;
  ~DevBuf() {
    if (p) cudaFreeAsync(p, st);
  }
  // Grows to at least n elements, keeping the first `keep` elements.
  cudaError_t reserve(int64_t n, int64_t keep = 0) {
    if (n <= cap) return cudaSuccess;
    int64_t const nc = std::max<int64_t>(n, cap + cap / 2);
    T *q = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&q), nc * sizeof(T), st);
    if (e != cudaSuccess) return e;
    if (keep > 0 && p) {
      e = cudaMemcpyAsync(q, p, keep * sizeof(T), cudaMemcpyDeviceToDevice, st);
      if (e != cudaSuccess) {
        cudaFreeAsync(q, st);
        return e;
      }
    }
    if (p) cudaFreeAsync(p, st);
    p = q;
    cap = nc;
    return cudaSuccess;
  }
  T *release() {
    T *q = p;
    p = nullptr;
    cap = 0;
    return q;
  }
};

struct RefBufs {
  DevBuf<int32_t> tri;
  DevBuf<float> c[6];
  cudaError_t reserve(int64_t n) {
    cudaError_t e = tri.reserve(n);
    for (int k = 0; k < 6 && e == cudaSuccess; ++k) e = c[k].reserve(n);
    return e;
  }
  RefArrays view() {
    RefArrays r;
    r.tri = tri.p;
    for (int k = 0; k < 3; ++k) {
      r.lo[k] = c[k].p;
      r.hi[k] = c[3 + k].p;
    }
    return r;
  }
};

struct LevelBufs {
  DevBuf<float4> blo, bhi;
  DevBuf<int32_t> begin, count, axis, nl, nr;
  DevBuf<float> plane;
  DevBuf<uint4> scan;
  cudaError_t reserve(int64_t n) {
    cudaError_t e = blo.reserve(n);
    if (e == cudaSuccess) e = bhi.reserve(n);
    if (e == cudaSuccess) e = begin.reserve(n);
    if (e == cudaSuccess) e = count.reserve(n);
    if (e == cudaSuccess) e = axis.reserve(n);
    if (e == cudaSuccess) e = nl.reserve(n);
    if (e == cudaSuccess) e = nr.reserve(n);
    if (e == cudaSuccess) e = plane.reserve(n);
    if (e == cudaSuccess) e = scan.reserve(n);
    return e;
  }
  LevelArrays view() {
    return LevelArrays{blo.p, bhi.p, begin.p, count.p, axis.p, plane.p, nl.p, nr.p, scan.p};
  }
};

int grid_for(int64_t work, int threads, int device) {
  int64_t const want = (work + threads - 1) / threads;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(want, int64_t{sm_count(device)} * 16)));
}

// ---- depth-first layout
// Descendant count of node i (its children lie in deeper levels, counted
// before) and, with sets, the box and triangle count of what lies below it.
XYZ_DEV void layout_up(const uint2 *__restrict__ nodes, int64_t i, int32_t *desc, const WideSets &T) {
  uint2 const nd = nodes[i];
  if ((nd.y & 3u) == kKdLeafTag) {
    desc[i] = 0;
    return;
  }
  uint32_t const c = nd.y >> 2;
  desc[i] = 2 + desc[c] + desc[c + 1];
  if (T.lo) {
    uint4 const a = T.lo[c], b = T.lo[c + 1], p = T.hi[c], q = T.hi[c + 1];
    T.lo[i] = make_uint4(min(a.x, b.x), min(a.y, b.y), min(a.z, b.z), 0u);
    T.hi[i] = make_uint4(max(p.x, q.x), max(p.y, q.y), max(p.z, q.z), p.w + q.w);
  }
}

// New positions of node i's children: the pair at base(parent); the first
// child's descendants from base + 2, the second's after them.  With sets, the
// positions of their triangles: the first child's, then the second's.
XYZ_DEV void layout_down(const uint2 *__restrict__ nodes, int64_t i, const int32_t *__restrict__ desc, int32_t *pos,
                         int32_t *base, const WideSets &T) {
  uint2 const nd = nodes[i];
  if ((nd.y & 3u) == kKdLeafTag) return;
  uint32_t const c = nd.y >> 2;
  int32_t const b = base[i];
  pos[c] = b;
  pos[c + 1] = b + 1;
  base[c] = b + 2;
  base[c + 1] = b + 2 + desc[c];
  if (T.lo) {
    int32_t const f = T.first[i];
    T.first[c] = f;
    T.first[c + 1] = f + static_cast<int32_t>(T.hi[c].w);
  }
}

__global__ void k_layout_desc(const uint2 *__restrict__ nodes, int64_t begin, int64_t end, int32_t *desc, WideSets T) {
  for (int64_t i = begin + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < end;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    layout_up(nodes, i, desc, T);
}

__global__ void k_layout_place(const uint2 *__restrict__ nodes, int64_t begin, int64_t end,
                               const int32_t *__restrict__ desc, int32_t *pos, int32_t *base, WideSets T) {
  for (int64_t i = begin + blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < end;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    layout_down(nodes, i, desc, pos, base, T);
}

// Both sweeps of the top levels in one CTA: a level of at most kTopNodes nodes
// takes one CTA no longer than a launch of its own takes.
constexpr int kTopLevels = 16;
constexpr int64_t kTopNodes = 2048;
struct TopLevels {
  int64_t start[kTopLevels + 1];
  int n;
};

__global__ void __launch_bounds__(1024)
    k_layout_top(const uint2 *__restrict__ nodes, TopLevels V, int32_t *desc, int32_t *pos, int32_t *base, WideSets T) {
  for (int l = V.n - 1; l >= 0; --l) {
    for (int64_t i = V.start[l] + threadIdx.x; i < V.start[l + 1]; i += blockDim.x) layout_up(nodes, i, desc, T);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    pos[0] = 0;
    base[0] = 1;
    if (T.lo) T.first[0] = 0;
  }
  __syncthreads();
  for (int l = 0; l < V.n; ++l) {
    for (int64_t i = V.start[l] + threadIdx.x; i < V.start[l + 1]; i += blockDim.x)
      layout_down(nodes, i, desc, pos, base, T);
    __syncthreads();
  }
}

__global__ void k_layout_scatter(const uint2 *__restrict__ nodes, int64_t n, const int32_t *__restrict__ pos,
                                 const int32_t *__restrict__ base, uint2 *__restrict__ out) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint2 nd = nodes[i];
    if ((nd.y & 3u) != kKdLeafTag) nd.y = (static_cast<uint32_t>(base[i]) << 2) | (nd.y & 3u);
    out[pos[i]] = nd;
  }
}


// ---- wide tree
// Each triangle joins the kd leaf that holds its centroid: the leaf's box and
// count take it in.
__global__ void __launch_bounds__(256)
    k_wide_assign(const float4 *__restrict__ tri, int n, const uint2 *__restrict__ nodes, WideSets T,
                  int32_t *__restrict__ owner, uint32_t *extents) {
  __shared__ uint32_t s_extents[kWideExtents];
  for (int i = threadIdx.x; i < kWideExtents; i += blockDim.x) s_extents[i] = 0u;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 const a = tri[3 * i], b = tri[3 * i + 1], c = tri[3 * i + 2];
    // vertices as the intersection test sees them: v0, v0 + e1, v0 + e2
    f3 const v0 = xyz3(a), e1 = xyz3(b), e2 = xyz3(c);
    int32_t const leaf = wide_leaf_of(nodes, scl3(add3(add3(v0, add3(v0, e1)), add3(v0, e2)), 1.0f / 3.0f));
    WideTri const w = wide_triangle(v0, e1, e2, mk3(a.w, b.w, c.w));
    owner[i] = leaf;
    atomicAdd(&s_extents[wide_extent_bucket(w.e)], 1u);
    uint32_t *const lo = reinterpret_cast<uint32_t *>(T.lo + leaf);
    uint32_t *const hi = reinterpret_cast<uint32_t *>(T.hi + leaf);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      atomicMin(lo + k, float_key(w.lo[k]));
      atomicMax(hi + k, float_key(w.hi[k]));
    }
    atomicAdd(hi + 3, 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kWideExtents; i += blockDim.x)
    if (s_extents[i]) atomicAdd(&extents[i], s_extents[i]);
}

// State of the level-by-level construction: nodes and records handed out, the
// node range [level[l], level[l + 1]) of every level, and per level the CTAs
// that have finished (the last one closes the next level's range).
struct WideCounters {
  uint32_t nodes, tris;
  uint32_t level[kWideStack + 3];
  uint32_t done[kWideStack + 1];
  uint32_t extents[kWideExtents];  // triangles by extent (k_wide_assign)
};

constexpr int kWideThreads = 64;

__global__ void __launch_bounds__(kWideThreads)
    k_wide_nodes(const uint2 *__restrict__ kd, WideSets T, int l, WideCounters *C, WideTask *task,
                 uint32_t max_nodes, uint32_t *__restrict__ out, int32_t *__restrict__ dst) {
  uint32_t const b = C->level[l], e = C->level[l + 1];
  for (uint32_t i = b + blockIdx.x * blockDim.x + threadIdx.x; i < e; i += gridDim.x * blockDim.x) {
    uint32_t w[kWideWords];
    wide_make_node(
        kd, T, task[i], 0.0f, w, [&](int k) { return atomicAdd(&C->nodes, static_cast<uint32_t>(k)); },
        [&](int k) { return atomicAdd(&C->tris, static_cast<uint32_t>(k)); },
        [&](uint32_t at, WideTask t) {
          if (at < max_nodes) task[at] = t;
        },
        [&](int32_t at, uint32_t rec) { dst[at] = static_cast<int32_t>(rec); });
    uint4 *const o = reinterpret_cast<uint4 *>(out + static_cast<size_t>(i) * kWideWords);
#pragma unroll
    for (int q = 0; q < kWideWords / 4; ++q) o[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&C->done[l], 1u) == gridDim.x - 1) C->level[l + 2] = min(atomicAdd(&C->nodes, 0u), max_nodes);
  }
}

// Triangle records in the order the nodes name them (within a kd leaf of
// several triangles in arrival order: the closest hit does not depend on it).
__global__ void k_wide_tris(const float4 *__restrict__ tri, int n, WideSets T, const int32_t *__restrict__ owner,
                            const int32_t *__restrict__ dst, float4 *__restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int32_t const leaf = owner[i];
    // w counts up from the 0xffffffff it was filled with
    uint32_t const k = atomicAdd(reinterpret_cast<uint32_t *>(T.lo + leaf) + 3, 1u) + 1u;
    size_t const rec = static_cast<size_t>(dst[T.first[leaf] + static_cast<int32_t>(k)]) * kWideTriVec;
    float4 const a = tri[3 * i], b = tri[3 * i + 1], c = tri[3 * i + 2];
    out[rec] = a;
    out[rec + 1] = b;
    out[rec + 2] = c;
    WideTri const w = wide_triangle(xyz3(a), xyz3(b), xyz3(c), mk3(a.w, b.w, c.w));
    out[rec + 3] = make_float4(__int_as_float(i), w.e, w.n, w.parallel);
  }
}

}  // namespace

#define XYZ_BUILD_TRY(call)                                                                       \
  do {                                                                                            \
    cudaError_t const e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                        \
      return set_error(e_ == cudaErrorMemoryAllocation ? XYZGPU_E_NOMEM : XYZGPU_E_CUDA,          \
                       "kd-tree build: %s failed: %s", #call, cudaGetErrorString(e_));            \
  } while (0)

int kd_build_device(SceneImpl &s, const float4 *d_tri, int n, const BuildConfig &cfg, cudaStream_t st) {
  if (cfg.bins < 2 || cfg.bins > kKdMaxBins)
    return set_error(XYZGPU_E_INVALID, "kd-tree build: bins must be in [2, 64]");
  if (cfg.max_refs >= (int64_t{1} << 31))
    return set_error(XYZGPU_E_LIMIT, "kd-tree build: the reference budget exceeds 2^31 - 1 "
                                     "(lower max_refs_factor or the triangle count)");
  BuildArgs A;
  A.leaf_max = cfg.leaf_max_tris;
  A.max_depth = cfg.max_depth;
  A.bins = cfg.bins;
  A.ct = cfg.cost_traversal;
  A.ci = cfg.cost_intersect;
  A.eb = cfg.empty_bonus;
  int const dev = s.device;

  RefBufs refs[2];
  LevelBufs lv[2];
  DevBuf<uint2> nodes;
  DevBuf<int32_t> leaf_refs;
  DevBuf<int32_t> big_list, big_count;
  DevBuf<int2> big_cnt;
  DevBuf<uint32_t> big_hist;
  DevBuf<uint4> block_sums;
  DevBuf<LevelTotals> totals;
  for (int q = 0; q < 2; ++q) {
    refs[q].tri.st = st;
    for (auto &c : refs[q].c) c.st = st;
    for (auto *b : {&lv[q].begin, &lv[q].count, &lv[q].axis, &lv[q].nl, &lv[q].nr}) b->st = st;
    lv[q].blo.st = lv[q].bhi.st = st;
    lv[q].plane.st = st;
    lv[q].scan.st = st;
  }
  nodes.st = st;
  leaf_refs.st = st;
  big_list.st = big_count.st = st;
  big_cnt.st = big_hist.st = st;
  block_sums.st = totals.st = st;
  XYZ_BUILD_TRY(refs[0].reserve(std::max(1, n)));
  // (a level may hold twice the nodes of the one before: not from one node up)
  for (auto &l : lv) XYZ_BUILD_TRY(l.reserve(std::min(std::max(1, n), kFirstLevelNodes)));
  XYZ_BUILD_TRY(nodes.reserve(std::max<int64_t>(64, 2 * static_cast<int64_t>(n) / std::max(1, cfg.leaf_max_tris))));
  XYZ_BUILD_TRY(leaf_refs.reserve(std::max<int64_t>(64, 2 * static_cast<int64_t>(n))));
  XYZ_BUILD_TRY(big_count.reserve(1));
  XYZ_BUILD_TRY(totals.reserve(1));

  if (n > 0) {
    k_init_refs<<<grid_for(n, 256, dev), 256, 0, st>>>(d_tri, n, refs[0].view());
    XYZ_BUILD_TRY(cudaGetLastError());
  }
  float4 const rlo = make_float4(s.dev.bmin.x, s.dev.bmin.y, s.dev.bmin.z, 0.0f);
  float4 const rhi = make_float4(s.dev.bmax.x, s.dev.bmax.y, s.dev.bmax.z, 0.0f);
  k_init_root<<<1, 1, 0, st>>>(lv[0].view(), rlo, rhi, n, big_count.p);
  XYZ_BUILD_TRY(cudaGetLastError());

  int64_t level_base = 0, leaf_total = 0, leaves = 0, empty = 0;
  int m = 1, depth = 0, cur = 0;
  A.depth = 0;
  int n_big = n >= kBigRefs && eligible(A, n) ? 1 : 0;
  std::vector<int64_t> level_start;
  for (depth = 0;; ++depth) {
    level_start.push_back(level_base);
    A.depth = depth;
    LevelArrays L = lv[cur].view();
    if (n_big > 0) {
      XYZ_BUILD_TRY(big_list.reserve(n_big));
      k_classify<<<grid_for(m, 256, dev), 256, 0, st>>>(L, m, A, big_list.p, big_count.p);
    }
    RefArrays const R = refs[cur].view();
    k_decide_small<<<grid_for(int64_t{m} * 32, 32 * kWarpsPerBlock, dev), 32 * kWarpsPerBlock, 0, st>>>(
        L, m, R, A, totals.p, big_count.p);
    // big nodes: sliced histograms, one CTA per node for the decision, sliced
    // left / right counts (kept for the emit) and their per-node totals;
    // slices per node: up to 128, about 1,024 CTAs per launch in all
    int const slices = n_big > 0 ? std::max(1, std::min(kBigSlicesMax, kBigSliceBudget / n_big)) : 1;
    if (n_big > 0) {
      XYZ_BUILD_TRY(big_hist.reserve(int64_t{n_big} * kHistWords));
      XYZ_BUILD_TRY(big_cnt.reserve(int64_t{n_big} * slices));
      XYZ_BUILD_TRY(cudaMemsetAsync(big_hist.p, 0, sizeof(uint32_t) * n_big * kHistWords, st));
      k_decide_big_hist<<<n_big * slices, kBigThreads, 0, st>>>(L, big_list.p, R, A, slices, big_hist.p);
      k_decide_big<<<n_big, kBigThreads, 0, st>>>(L, big_list.p, A, big_hist.p);
      k_emit_big_count<<<n_big * slices, kBigThreads, 0, st>>>(L, R, big_list.p, slices, big_cnt.p);
      k_big_totals<<<n_big, 32, 0, st>>>(L, big_list.p, slices, big_cnt.p);
    }
    XYZ_BUILD_TRY(cudaGetLastError());
    // flags + scan (twice if the reference budget is exceeded)
    BuildArgs next = A;
    next.depth = depth + 1;
    LevelTotals level{};
    uint4 &tot = level.scan;
    for (int pass = 0; pass < 2; ++pass) {
      k_flags<<<grid_for(m, 256, dev), 256, 0, st>>>(L, m, pass, next, totals.p);
      int const nb = static_cast<int>((m + kScanPerBlock - 1) / kScanPerBlock);
      XYZ_BUILD_TRY(block_sums.reserve(nb));
      // one block: its sums are the level's
      k_scan_blocks<<<nb, kScanThreads, 0, st>>>(L.scan, m, nb == 1 ? &totals.p->scan : block_sums.p);
      if (nb > 1) {
        k_scan_totals<<<1, kScanThreads, 0, st>>>(block_sums.p, nb, &totals.p->scan);
        k_scan_add<<<(m + 255) / 256, 256, 0, st>>>(L.scan, m, block_sums.p);
      }
      XYZ_BUILD_TRY(cudaGetLastError());
      XYZ_BUILD_TRY(cudaMemcpyAsync(&level, totals.p, sizeof(level), cudaMemcpyDeviceToHost, st));
      XYZ_BUILD_TRY(cudaStreamSynchronize(st));
      if (static_cast<int64_t>(tot.z) <= cfg.max_refs) break;
    }
    int64_t const splits = tot.x;
    int64_t const next_m = 2 * splits;
    int64_t const next_base = level_base + m;
    if (next_base + next_m >= (int64_t{1} << 30))
      return set_error(XYZGPU_E_LIMIT, "kd-tree build: node count exceeds 2^30");
    XYZ_BUILD_TRY(nodes.reserve(next_base + std::max<int64_t>(next_m, 1), level_base));
    XYZ_BUILD_TRY(leaf_refs.reserve(leaf_total + std::max<int64_t>(tot.y, 1), leaf_total));
    XYZ_BUILD_TRY(lv[cur ^ 1].reserve(std::max<int64_t>(next_m, 1)));
    XYZ_BUILD_TRY(refs[cur ^ 1].reserve(std::max<int64_t>(tot.z, 1)));
    EmitArgs E;
    E.L = lv[cur].view();
    E.N = lv[cur ^ 1].view();
    E.R = refs[cur].view();
    E.RN = refs[cur ^ 1].view();
    E.nodes = nodes.p;
    E.leaf_refs = leaf_refs.p;
    E.level_base = level_base;
    E.next_base = next_base;
    E.leaf_base = leaf_total;
    E.m = m;
    k_emit_small<<<grid_for(int64_t{m} * 32, 32 * kWarpsPerBlock, dev), 32 * kWarpsPerBlock, 0, st>>>(E, A);
    // big_cnt was written by k_emit_big_count at decision time, before the
    // flag / scan passes, and holds valid per-slice counts only for nodes that
    // decided to split (axis >= 0); leaves never have theirs written.  The
    // second k_flags pass (reference budget exceeded) only turns nodes into
    // leaves (axis = -1), and k_emit_big takes its leaf branch for those
    // without reading cnt, so the counts stay valid for every node that reads
    // them here.
    if (n_big > 0) k_emit_big<<<n_big * slices, kBigThreads, 0, st>>>(E, big_list.p, slices, big_cnt.p);
    XYZ_BUILD_TRY(cudaGetLastError());
    leaves += m - splits;
    empty += tot.w;
    leaf_total += tot.y;
    level_base = next_base;
    if (next_m == 0) break;
    m = static_cast<int>(next_m);
    n_big = level.next_big;
    cur ^= 1;
  }
  XYZ_BUILD_TRY(cudaStreamSynchronize(st));
  level_start.push_back(level_base);
  s.n_nodes = level_base;
  s.n_refs = leaf_total;
  s.n_leaves = leaves;
  s.n_empty = empty;
  s.depth = depth;
  s.d_nodes = nodes.release();
  s.d_refs = leaf_refs.release();
  return kd_layout_depth_first(s, level_start, st);
}

namespace {

// Nodes a wide tree over n triangles may need: a node either has eight
// children or only leaf children and then at least four triangles, so there
// are at most n / 4 of the second kind and (n + n / 4) / 7 of the first.
int64_t wide_max_nodes(int64_t n) { return n / 4 + (n + n / 4) / 7 + 64; }

struct WideBufs {
  DevBuf<uint4> lo, hi;
  DevBuf<int32_t> first, owner, dst;
  DevBuf<uint32_t> nodes;
  DevBuf<WideTask> task;
  DevBuf<WideCounters> counters;
  DevBuf<float4> tris;
};

// Fills the wide tree from the sets of the breadth-first kd nodes.  A tree
// deeper than the traversal's stack is dropped (the kd-tree serves alone).
int wide_build(SceneImpl &s, WideBufs &B, const WideSets &T, float largest, cudaStream_t st) {
  int const dev = s.device, n = s.n_tris;
  uint32_t const max_nodes = static_cast<uint32_t>(wide_max_nodes(n));
  WideCounters h{};
  h.nodes = 1;
  h.level[1] = 1;
  WideTask const root{0, 0, n};
  XYZ_BUILD_TRY(cudaMemcpyAsync(B.counters.p, &h, offsetof(WideCounters, extents), cudaMemcpyHostToDevice, st));
  XYZ_BUILD_TRY(cudaMemcpyAsync(B.task.p, &root, sizeof(root), cudaMemcpyHostToDevice, st));
  int const grid = grid_for(n / 8 + 1, kWideThreads, dev);
  int done = 0;
  bool more = true;
  // about log8(n) levels, a few more where the tree is uneven: their launches
  // are issued ahead and the host looks at the ranges after each group
  for (int group = n > 4096 ? 10 : 4; more && done < kWideStack; group = 4) {
    int const upto = std::min(kWideStack, done + group);
    for (; done < upto; ++done)
      k_wide_nodes<<<grid, kWideThreads, 0, st>>>(s.d_nodes, T, done, B.counters.p, B.task.p, max_nodes,
                                                  B.nodes.p, B.dst.p);
    XYZ_BUILD_TRY(cudaGetLastError());
    XYZ_BUILD_TRY(cudaMemcpyAsync(&h, B.counters.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    XYZ_BUILD_TRY(cudaStreamSynchronize(st));
    more = h.level[done] < h.level[done + 1];
  }
  if (more || h.nodes > max_nodes || h.tris != static_cast<uint32_t>(n)) return XYZGPU_OK;
  k_wide_tris<<<grid_for(n, 256, dev), 256, 0, st>>>(s.d_tri, n, T, B.owner.p, B.dst.p, B.tris.p);
  XYZ_BUILD_TRY(cudaGetLastError());
  DevBuf<uint32_t> out;
  out.st = st;
  size_t const words = static_cast<size_t>(h.nodes) * kWideWords;
  if (out.reserve(static_cast<int64_t>(words)) != cudaSuccess) {
    cudaGetLastError();
    return XYZGPU_OK;
  }
  XYZ_BUILD_TRY(cudaMemcpyAsync(out.p, B.nodes.p, words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  s.n_wide = h.nodes;
  s.d_wide = out.release();
  s.d_wide_tri = B.tris.release();
  f3 const half = scl3(sub3(s.dev.bmax, s.dev.bmin), 0.5f);
  s.dev.wide_mid = add3(s.dev.bmin, half);
  s.dev.wide_reach = wide_reach_of(std::max({half.x, half.y, half.z}), largest, h.extents, static_cast<uint32_t>(n));
  return XYZGPU_OK;
}

}  // namespace

int kd_layout_depth_first(SceneImpl &s, const std::vector<int64_t> &level_start, cudaStream_t st) {
  int64_t const n = s.n_nodes;
  if (n < 1 || s.n_tris < 1) return XYZGPU_OK;
  if (level_start.size() < 2 || level_start.front() != 0 || level_start.back() != n)
    return set_error(XYZGPU_E_INVALID, "kd-tree layout: level ranges do not cover the nodes");
  int const dev = s.device, nt = s.n_tris;
  DevBuf<int32_t> desc, pos, base;
  DevBuf<uint2> out;
  desc.st = pos.st = base.st = out.st = st;
  XYZ_BUILD_TRY(desc.reserve(n));
  XYZ_BUILD_TRY(pos.reserve(n));
  XYZ_BUILD_TRY(base.reserve(n));
  XYZ_BUILD_TRY(out.reserve(n));
  // the wide tree: without room for it (or with coordinates its grid
  // arithmetic cannot hold) the scene keeps the kd-tree alone
  float const reach = std::max({std::fabs(s.dev.bmin.x), std::fabs(s.dev.bmin.y), std::fabs(s.dev.bmin.z),
                                std::fabs(s.dev.bmax.x), std::fabs(s.dev.bmax.y), std::fabs(s.dev.bmax.z)});
  WideBufs B;
  B.lo.st = B.hi.st = B.first.st = B.owner.st = B.dst.st = B.nodes.st = B.task.st = B.counters.st = B.tris.st = st;
  WideSets T;
  int64_t const max_wide = wide_max_nodes(nt);
  bool const wide = reach < 1e12f && B.lo.reserve(n) == cudaSuccess && B.hi.reserve(n) == cudaSuccess &&
                    B.first.reserve(n) == cudaSuccess && B.owner.reserve(nt) == cudaSuccess &&
                    B.dst.reserve(nt) == cudaSuccess && B.nodes.reserve(max_wide * kWideWords) == cudaSuccess &&
                    B.task.reserve(max_wide) == cudaSuccess && B.counters.reserve(1) == cudaSuccess &&
                    B.tris.reserve(int64_t{kWideTriVec} * nt) == cudaSuccess;
  if (!wide) cudaGetLastError();
  if (wide) {
    T = WideSets{B.lo.p, B.hi.p, B.first.p};
    XYZ_BUILD_TRY(cudaMemsetAsync(B.lo.p, 0xff, n * sizeof(uint4), st));
    XYZ_BUILD_TRY(cudaMemsetAsync(B.hi.p, 0, n * sizeof(uint4), st));
    XYZ_BUILD_TRY(cudaMemsetAsync(B.counters.p, 0, sizeof(WideCounters), st));
    k_wide_assign<<<grid_for(nt, 256, dev), 256, 0, st>>>(s.d_tri, nt, s.d_nodes, T, B.owner.p, B.counters.p->extents);
  }
  int const levels = static_cast<int>(level_start.size()) - 1;
  TopLevels V{};
  while (V.n < kTopLevels && V.n < levels && level_start[V.n + 1] - level_start[V.n] <= kTopNodes) ++V.n;
  for (int l = 0; l <= V.n; ++l) V.start[l] = level_start[l];
  for (int l = levels; l-- > V.n;) {
    int64_t const b = level_start[l], e = level_start[l + 1];
    if (e > b) k_layout_desc<<<grid_for(e - b, 256, dev), 256, 0, st>>>(s.d_nodes, b, e, desc.p, T);
  }
  k_layout_top<<<1, 1024, 0, st>>>(s.d_nodes, V, desc.p, pos.p, base.p, T);
  for (int l = V.n; l < levels; ++l) {
    int64_t const b = level_start[l], e = level_start[l + 1];
    if (e > b) k_layout_place<<<grid_for(e - b, 256, dev), 256, 0, st>>>(s.d_nodes, b, e, desc.p, pos.p, base.p, T);
  }
  k_layout_scatter<<<grid_for(n, 256, dev), 256, 0, st>>>(s.d_nodes, n, pos.p, base.p, out.p);
  XYZ_BUILD_TRY(cudaGetLastError());
  if (wide) {
    int const rc = wide_build(s, B, T, reach, st);
    if (rc) return rc;
  }
  XYZ_BUILD_TRY(cudaFreeAsync(s.d_nodes, st));
  s.d_nodes = out.release();
  XYZ_BUILD_TRY(cudaStreamSynchronize(st));
  return XYZGPU_OK;
}

}  // namespace xyzgpu
