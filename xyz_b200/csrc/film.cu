// Film output on the device and the file formats around it:
//  * the Radiance RGBE pixel encoding of ImageFilm::SaveAsHdr
//    (xyz/core/imagefilm_hdr.cpp:14-31, 124-183) as a kernel, and the file
//    (header and run-length scanlines, :46-114) written on the host;
//  * the float2bmp tone operators (float2bmp/main.cpp:69-118, 209-214) as a
//    kernel producing 24-bit BMP pixel rows, and the BMP file;
//  * a resumable render checkpoint: film sums, the number of samples done
//    and the render parameters, so a render continues where it stopped (the
//    reference's periodic .pfm dump, xyz/integrator/integrator.cpp:140-160,
//    keeps the image but not a way to continue it).
// All three read the film as xyzgpu_render leaves it: W * H XYZ sums, row 0
// at the bottom.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "scene.h"

namespace xyzgpu {
namespace {

constexpr int kFilmThreads = 256;

bool aligned(const void *p, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

int device_sms() {
  int dev = 0;
  cudaGetDevice(&dev);
  return sm_count(dev);
}

// One thread per item (a grid-stride loop takes what lies beyond the limit).
int film_grid(int64_t n) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + kFilmThreads - 1) / kFilmThreads, 1 << 20)));
}

// static_cast<unsigned char>(float) as the reference's build performs it: the
// value truncated towards zero to a 32-bit integer, whose low byte is kept
// (negative colour components of saturated XYZ wrap around rather than
// saturate).
__device__ __forceinline__ uint8_t byte_of(float v) { return static_cast<uint8_t>(static_cast<uint32_t>(__float2int_rz(v))); }

// hdr_encode (imagefilm_hdr.cpp:14-31): the scale frexp(d) * 255.9999 / d,
// in double, rounded to float, times each component.  frexp(d) / d is the power
// of two 2^-e, so the scale is 255.9999 2^-e up to the two roundings in double
// (2^-52), and 255.9999 lies far from a float rounding border: the rounded
// scale is the float nearest 255.9999 with its exponent lowered by e (d is
// above 1e-32, so e and the scale stay in the normal range).
__host__ __device__ __forceinline__ float rgbe_scale(int e) {
  uint32_t const bits = 0x437ffff9u - (static_cast<uint32_t>(e) << 23);  // 255.9999f
#ifdef __CUDA_ARCH__
  return __uint_as_float(bits);
#else
  float f;
  std::memcpy(&f, &bits, 4);
  return f;
#endif
}

__device__ __forceinline__ uchar4 rgbe_of(float r, float g, float b) {
  float const d = fmaxf(fmaxf(r, g), b);
  if (static_cast<double>(d) <= 1e-32) return make_uchar4(0, 0, 0, 0);
  int e = (static_cast<int>(__float_as_uint(d) >> 23) & 0xff) - 126;
  float f = rgbe_scale(e);
  if (!isfinite(d)) {  // XYZE keeps such pixels
    e = 0;
    float const m = frexpf(d, &e);
    f = static_cast<float>(static_cast<double>(m) * 255.9999 / static_cast<double>(d));
  }
  return make_uchar4(byte_of(r * f), byte_of(g * f), byte_of(b * f), static_cast<uint8_t>(e + 128));
}

// Four film pixels of a row from pixel p (n of them inside the row): 16-byte
// loads where the film's rows allow it.
__device__ __forceinline__ void load_pixels(const float *__restrict__ film, int64_t p, int n, bool vec, float v[12]) {
  if (vec) {
    const float4 *q = reinterpret_cast<const float4 *>(film + 3 * p);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float4 const x = __ldcs(q + k);
      v[4 * k] = x.x, v[4 * k + 1] = x.y, v[4 * k + 2] = x.z, v[4 * k + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = k < 3 * n ? film[3 * p + k] : 0.0f;
  }
}

// Four pixels of a row per thread; output in file order.  RGBE: scanlines from
// the top image row down ("-Y H +X W"), the film's XYZ / spp converted to CCIR
// 601-1 RGB (CCIR601_1_XYZ2RGB, libhi/hi/image/color_space.hpp:69-79) and a
// non-finite pixel written as 0.  XYZE (the reference's CONFIG_HDR_STRICT
// build): XYZ / spp, scanlines from the bottom row up ("+Y H +X W").
// Measured at 1920 x 1080: one pixel per thread with the scale in double 13.4
// us, this form 9.2 (33 MB; 5.1 us at the copy rate).
__global__ void __launch_bounds__(kFilmThreads)
    k_film_rgbe(const float *__restrict__ film, int W, int H, float scale, int xyze, int vec, uchar4 *__restrict__ out) {
  int const quads = (W + 3) >> 2;
  int64_t const n = static_cast<int64_t>(quads) * H;
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < n;
       q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t const row = q / quads;
    int const x = static_cast<int>(q - row * quads) * 4, m = min(4, W - x);
    float v[12];
    load_pixels(film, (xyze ? row : (H - 1 - row)) * W + x, m, vec != 0, v);
    uchar4 px[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float const X = v[3 * k] * scale, Y = v[3 * k + 1] * scale, Z = v[3 * k + 2] * scale;
      if (xyze) {
        px[k] = rgbe_of(X, Y, Z);
        continue;
      }
      float r = 1.9104f * X - 0.5338f * Y - 0.2891f * Z;
      float g = -0.9844f * X + 1.9985f * Y - 0.0279f * Z;
      float b = 0.0585f * X - 0.1187f * Y + 0.9017f * Z;
      if (!isfinite(r) || !isfinite(g) || !isfinite(b)) r = g = b = 0.0f;
      px[k] = rgbe_of(r, g, b);
    }
    uchar4 *const o = out + row * W + x;
    if (vec) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = *reinterpret_cast<const uint32_t *>(&px[k]);
      *reinterpret_cast<uint4 *>(o) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < m) o[k] = px[k];
    }
  }
}

// float2bmp's luminance for the white point of the Reinhard operator: the
// maximum over pixels of 0.6069 c0 + 0.1735 c1 + 0.2003 c2 of the values
// tone-mapped (float2bmp/main.cpp:186-196; the maximum starts at 0, so the
// non-negative float bits order as integers).
// Four pixels per thread and step; one atomic per CTA (a CTA of every eighth
// of an SM's threads would otherwise send 9,472 to one word).
__global__ void __launch_bounds__(kFilmThreads)
    k_film_max_luminance(const float *__restrict__ film, int64_t n, float scale, int rgb, int vec, unsigned int *out) {
  __shared__ float s_best[kFilmThreads / 32];
  float best = 0.0f;
  int64_t const quads = (n + 3) >> 2;
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < quads;
       q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int const m = static_cast<int>(min(int64_t{4}, n - 4 * q));
    float v[12];
    load_pixels(film, 4 * q, m, vec != 0 && m == 4, v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= m) break;
      float c[3] = {v[3 * k] * scale, v[3 * k + 1] * scale, v[3 * k + 2] * scale};
      if (rgb) {
        float const X = c[0], Y = c[1], Z = c[2];
        c[0] = 1.9104f * X - 0.5338f * Y - 0.2891f * Z;
        c[1] = -0.9844f * X + 1.9985f * Y - 0.0279f * Z;
        c[2] = 0.0585f * X - 0.1187f * Y + 0.9017f * Z;
      }
      float const l = 0.6069f * c[0] + 0.1735f * c[1] + 0.2003f * c[2];
      if (best < l) best = l;
    }
  }
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_down_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < kFilmThreads / 32) {
    best = s_best[threadIdx.x];
    for (int o = kFilmThreads / 64; o > 0; o >>= 1) best = fmaxf(best, __shfl_down_sync(0xffu, best, o));
    if (threadIdx.x == 0 && best > 0.0f) atomicMax(out, __float_as_uint(best));
  }
}

struct ToneArgs {
  float scale, exposure, white, gamma;
  int op, rgb;
  const unsigned int *white_bits;  // device maximum luminance (white <= 0), else null
};

// tonemap() of float2bmp/main.cpp:80-118: operator, gamma src / dst, then the
// 8-bit quantisation of clamp() (:69-77), in the tool's float arithmetic.
__device__ __noinline__ uint8_t tone_exact(float light, const ToneArgs &T, float white) {
  if (light <= 0.0f) return 0;
  float v;
  switch (T.op) {
    case XYZGPU_TONEMAP_LINEAR: v = T.exposure * light; break;
    case XYZGPU_TONEMAP_REINHARD: v = T.exposure * light / (1.0f + light); break;
    case XYZGPU_TONEMAP_REINHARD_WHITE: v = T.exposure * light * (1.0f + light / (white * white)) / (1.0f + light); break;
    default: v = 1.0f - expf(-T.exposure * light); break;
  }
  v = powf(v, T.gamma);
  if (v <= 0.0f) return 0;
  if (v >= 1.0f) return 255;
  return static_cast<uint8_t>(v * 256.0f);
}

__device__ __forceinline__ float exp2_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float log2_fast(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float clamp_nan(float x, float lo, float hi) {
  float r;
  asm("{ .reg .f32 t; max.NaN.f32 t, %1, %2; min.NaN.f32 %0, t, %3; }" : "=f"(r) : "f"(x), "f"(lo), "f"(hi));
  return r;
}

// The same byte by the fast reciprocal, exponential and logarithm where their
// result p (in 256ths) lies clear of an integer, or -1 where tone_exact has to be
// asked.  p = 256 v^g up to 257 errs, with L = log2 v, by p (1.7e-7 (1 + |L|) g +
// 2.4e-7) from the logarithm (2^-22, relative below 1/2) and the power, by 1e-6 p g
// from the operator (6 roundings and a reciprocal of 1 ulp) and tone_exact by 2.4e-7 p
// from its power: 1.5e-4 + 3e-4 g, so 2e-4 + 3.5e-4 g is clear.  Of the film
// operator's v = 1 - e^-x either side may be off by 2.1e-7 (the cancellation; below
// 1/4 the series x - x^2/2 + ... is used here, tone_exact stays off): p by
// 5e-7 g p / v.  Below half and above 255.5 no integer can matter (bytes 0 and 255),
// except that a v too small for the fast logarithm may still be seen by exponents
// below 0.1.  Where a rounding could take the Reinhard operators out of range (light
// of 1e37 on, a white point whose square is not within 1e-30 .. 1e30; inv_white2 is
// NaN then), for exponents above 16 and for NaN, tone_exact is asked.
template <int kOp>
__device__ __forceinline__ int tone_fast(float light, const ToneArgs &T, float inv_white2) {
  float v = T.exposure * light;
  float clear = T.gamma <= 16.0f ? 2e-4f + 3.5e-4f * T.gamma : 1.0f;
  if (kOp == XYZGPU_TONEMAP_REINHARD) {
    v = v * rcp_fast(1.0f + light);
  } else if (kOp == XYZGPU_TONEMAP_REINHARD_WHITE) {
    v = v * (1.0f + light * inv_white2) * rcp_fast(1.0f + light);
  } else if (kOp == XYZGPU_TONEMAP_FILM) {
    float s = __fmaf_rn(v, -1.0f / 720.0f, 1.0f / 120.0f);
    s = __fmaf_rn(v, s, -1.0f / 24.0f);
    s = __fmaf_rn(v, s, 1.0f / 6.0f);
    s = __fmaf_rn(v, s, -0.5f);
    s = __fmaf_rn(v, s, 1.0f);
    v = fabsf(v) < 0.25f ? v * s : 1.0f - exp2_fast(-1.44269504f * v);
  }
  // (a NaN stays one)
  float const p = clamp_nan(exp2_fast(T.gamma * log2_fast(v)) * 256.0f, T.gamma >= 0.1f ? 0.5f : 0.0f, 255.5f);
  if (kOp == XYZGPU_TONEMAP_FILM) clear += 5e-7f * T.gamma * p * rcp_fast(fabsf(v));
  // nearest integer in the low bits of p + 2^23
  float const q = p + 8388608.0f, r = q - 8388608.0f;
  int const byte = (__float_as_int(q) & 0x7fffff) - (p < r ? 1 : 0);
  bool const sure = fabsf(p - r) > clear && (kOp == XYZGPU_TONEMAP_LINEAR || kOp == XYZGPU_TONEMAP_FILM || light < 1e37f);
  return light <= 0.0f ? 0 : (sure ? byte : -1);
}

__device__ __forceinline__ void tone_channels(const ToneArgs &T, float X, float Y, float Z, float c[3]) {
  c[0] = X * T.scale;
  c[1] = Y * T.scale;
  c[2] = Z * T.scale;
  if (T.rgb) {
    float const x = c[0], y = c[1], z = c[2];
    c[0] = 1.9104f * x - 0.5338f * y - 0.2891f * z;
    c[1] = -0.9844f * x + 1.9985f * y - 0.0279f * z;
    c[2] = 0.0585f * x - 0.1187f * y + 0.9017f * z;
  }
}

// Four pixels of a row per thread: twelve bytes, which are three aligned words
// of the row (rows are padded to 4 bytes).  BMP order (rows from the bottom, as
// the film) and byte order (blue, green, red = channel 2, 1, 0); the row's
// padding bytes are zero (the caller's buffer may hold anything).
// Measured at 1920 x 1080 (Reinhard with the image's white): a pixel per
// thread with powf and byte stores 37.0 us, this form 16.4 (issue-bound: 76 % of
// cycles); the maximum before it 9.5 -> 5.1.  The film operator 18.8, on a film a
// hundredth as bright too: whole calls 68 us with powf, 77 (89 if dark) with the
// fast form for exposures from 0.05 and exponents up to 1 only, 52 now.
template <int kOp>
__global__ void __launch_bounds__(kFilmThreads)
    k_film_tonemap(const float *__restrict__ film, int W, int H, ToneArgs T, int vec, int words,
                   uint8_t *__restrict__ out) {
  float const white = T.white_bits ? __uint_as_float(*T.white_bits) : T.white;
  float const white2 = white * white;
  float const inv_white2 = white2 > 1e-30f && white2 < 1e30f ? 1.0f / white2 : __int_as_float(0x7fffffff);
  int64_t const stride_b = (3 * static_cast<int64_t>(W) + 3) & ~int64_t{3};
  int const quads = (W + 3) >> 2;
  int64_t const n = static_cast<int64_t>(quads) * H;
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < n;
       q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t const y = q / quads;
    int const x = static_cast<int>(q - y * quads) * 4, m = min(4, W - x);
    float v[12];
    load_pixels(film, y * W + x, m, vec != 0, v);
    uint32_t w[3] = {0u, 0u, 0u}, ask = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float c[3];
      tone_channels(T, v[3 * k], v[3 * k + 1], v[3 * k + 2], c);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        int const at = 3 * k + j, byte = tone_fast<kOp>(c[2 - j], T, inv_white2);
        w[at >> 2] |= static_cast<uint32_t>(byte & 0xff) << (8 * (at & 3));
        if (byte < 0 && k < m) ask |= 1u << at;
        if (k >= m) w[at >> 2] &= ~(0xffu << (8 * (at & 3)));
      }
    }
    // one copy of the exact form, in a loop: unrolled into the twelve channels
    // it overflows the instruction cache (22 us)
    for (; ask; ask &= ask - 1) {
      int const at = __ffs(static_cast<int>(ask)) - 1, k = at / 3, j = at - 3 * k;
      const float *f = film + 3 * (y * W + x + k);
      float c[3];
      tone_channels(T, f[0], f[1], f[2], c);
      uint32_t const byte = tone_exact(j == 0 ? c[2] : (j == 1 ? c[1] : c[0]), T, white);
      uint32_t const shift = 8 * (at & 3);
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (q == at >> 2) w[q] = (w[q] & ~(0xffu << shift)) | (byte << shift);
    }
    // the group's words: all three, or (the row's end) those that hold its
    // 3 m bytes, whose rest is the padding
    uint8_t *const o = out + y * stride_b + 3 * x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (4 * k >= 3 * m) break;
      if (words) {
        reinterpret_cast<uint32_t *>(o)[k] = w[k];
      } else {
        for (int j = 0; j < 4; ++j) o[4 * k + j] = static_cast<uint8_t>(w[k] >> (8 * j));
      }
    }
  }
}

// ---- Radiance run-length scanline (the format of imagefilm_hdr.cpp:46-114):
// lines of 8..32767 pixels start with 2, 2, width (16 bits, big-endian) and
// hold each of the four byte planes as packets: a run (128 + n, value) of
// n = 4..127 equal bytes or a literal (n, then n bytes) of n = 1..128 bytes;
// shorter runs stay inside literals.  Other widths are written flat.
void write_rle_line(const uint8_t *px, int W, std::vector<uint8_t> &o) {
  if (W < 8 || W > 0x7fff) {
    o.insert(o.end(), px, px + 4 * static_cast<size_t>(W));
    return;
  }
  o.push_back(2);
  o.push_back(2);
  o.push_back(static_cast<uint8_t>((W >> 8) & 0xff));
  o.push_back(static_cast<uint8_t>(W & 0xff));
  for (int c = 0; c < 4; ++c) {
    auto at = [&](int i) { return px[4 * i + c]; };
    int lit = 0;  // start of the pending literal bytes
    int i = 0;
    auto flush = [&](int end) {
      while (lit < end) {
        int const n = std::min(128, end - lit);
        o.push_back(static_cast<uint8_t>(n));
        for (int k = 0; k < n; ++k) o.push_back(at(lit + k));
        lit += n;
      }
    };
    while (i < W) {
      int run = 1;
      while (run < 127 && i + run < W && at(i + run) == at(i)) ++run;
      if (run >= 4) {
        flush(i);
        o.push_back(static_cast<uint8_t>(128 + run));
        o.push_back(at(i));
        i += run;
        lit = i;
      } else {
        i += run;
      }
    }
    flush(W);
  }
}

uint64_t fnv1a(const void *p, size_t n, uint64_t h = 1469598103934665603ull) {
  const uint8_t *b = static_cast<const uint8_t *>(p);
  for (size_t i = 0; i < n; ++i) {
    h ^= b[i];
    h *= 1099511628211ull;
  }
  return h;
}

constexpr char kCkptMagic[8] = {'X', 'Y', 'Z', 'G', 'P', 'U', 'C', 'K'};
constexpr uint32_t kCkptVersion = 1;

}  // namespace
}  // namespace xyzgpu

using namespace xyzgpu;

extern "C" {

int xyzgpu_film_encode_rgbe(const float *film, int width, int height, float scale, int xyze, uint8_t *out,
                            void *stream) {
  clear_error();
  if (!film || !out || width <= 0 || height <= 0 || !std::isfinite(scale))
    return set_error(XYZGPU_E_INVALID, "film_encode_rgbe: bad argument");
  int64_t const n = (static_cast<int64_t>(width) + 3) / 4 * height;
  k_film_rgbe<<<film_grid(n), kFilmThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      film, width, height, scale, xyze != 0, aligned(film, 16) && aligned(out, 16) && width % 4 == 0,
      reinterpret_cast<uchar4 *>(out));
  XYZ_CUDA_TRY(cudaGetLastError());
  return XYZGPU_OK;
}

int xyzgpu_hdr_write(const char *path, const uint8_t *rgbe, int width, int height, int xyze) {
  clear_error();
  if (!path || !rgbe || width <= 0 || height <= 0) return set_error(XYZGPU_E_INVALID, "hdr_write: bad argument");
  std::vector<uint8_t> o;
  char head[256];
  int const hn = std::snprintf(head, sizeof(head),
                               "#?RADIANCE\n# Made with xyzgpu\nFORMAT=32-bit_rle_%s\nEXPOSURE=1.0000000000000\n\n"
                               "%cY %d +X %d\n",
                               xyze ? "xyze" : "rgbe", xyze ? '+' : '-', height, width);
  o.insert(o.end(), head, head + hn);
  for (int r = 0; r < height; ++r) write_rle_line(rgbe + 4 * static_cast<size_t>(r) * width, width, o);
  FILE *f = std::fopen(path, "wb");
  if (!f) return set_error(XYZGPU_E_INVALID, "hdr_write: cannot open %s", path);
  size_t const w = std::fwrite(o.data(), 1, o.size(), f);
  if (std::fclose(f) != 0 || w != o.size()) return set_error(XYZGPU_E_INVALID, "hdr_write: writing %s failed", path);
  return XYZGPU_OK;
}

void xyzgpu_tonemap_params_default(xyzgpu_tonemap_params *tp) {
  if (!tp) return;
  tp->scale = 1.0f;
  tp->op = XYZGPU_TONEMAP_FILM;
  tp->exposure = 1.0f;
  tp->white = 0.0f;
  tp->dst_gamma = 2.2f;
  tp->src_gamma = 1.0f;
  tp->rgb = 0;
}

int xyzgpu_film_tonemap(const float *film, int width, int height, const xyzgpu_tonemap_params *tp, uint8_t *out,
                        unsigned int *scratch_white, void *stream) {
  clear_error();
  if (!film || !out || !tp || width <= 0 || height <= 0 || !std::isfinite(tp->scale) ||
      !std::isfinite(tp->exposure) || !(tp->dst_gamma > 0.0f) || !(tp->src_gamma > 0.0f) || tp->op < 0 ||
      tp->op > XYZGPU_TONEMAP_REINHARD_WHITE)
    return set_error(XYZGPU_E_INVALID, "film_tonemap: bad argument");
  bool const need_white = tp->op == XYZGPU_TONEMAP_REINHARD_WHITE && !(tp->white > 0.0f);
  if (need_white && !scratch_white)
    return set_error(XYZGPU_E_INVALID, "film_tonemap: the image's white point needs a device word (scratch_white)");
  cudaStream_t const st = static_cast<cudaStream_t>(stream);
  int64_t const n = static_cast<int64_t>(width) * height;
  ToneArgs T{tp->scale, tp->exposure, tp->white, tp->src_gamma / tp->dst_gamma, tp->op, tp->rgb != 0, nullptr};
  if (need_white) {
    XYZ_CUDA_TRY(cudaMemsetAsync(scratch_white, 0, sizeof(unsigned int), st));
    k_film_max_luminance<<<std::min(film_grid((n + 3) / 4), 8 * device_sms()), kFilmThreads, 0, st>>>(film, n, tp->scale, tp->rgb != 0,
                                                                          aligned(film, 16), scratch_white);
    T.white_bits = scratch_white;
  }
  auto const kernel = tp->op == XYZGPU_TONEMAP_LINEAR           ? k_film_tonemap<XYZGPU_TONEMAP_LINEAR>
                      : tp->op == XYZGPU_TONEMAP_REINHARD       ? k_film_tonemap<XYZGPU_TONEMAP_REINHARD>
                      : tp->op == XYZGPU_TONEMAP_REINHARD_WHITE ? k_film_tonemap<XYZGPU_TONEMAP_REINHARD_WHITE>
                                                                : k_film_tonemap<XYZGPU_TONEMAP_FILM>;
  kernel<<<film_grid((static_cast<int64_t>(width) + 3) / 4 * height), kFilmThreads, 0, st>>>(
      film, width, height, T, aligned(film, 16) && width % 4 == 0, aligned(out, 4), out);
  XYZ_CUDA_TRY(cudaGetLastError());
  return XYZGPU_OK;
}

int xyzgpu_bmp_write(const char *path, const uint8_t *bgr, int width, int height) {
  clear_error();
  if (!path || !bgr || width <= 0 || height <= 0) return set_error(XYZGPU_E_INVALID, "bmp_write: bad argument");
  uint32_t const stride = (3u * static_cast<uint32_t>(width) + 3u) & ~3u;
  uint32_t const data = stride * static_cast<uint32_t>(height);
  uint8_t h[54] = {0};
  auto put32 = [&](int at, uint32_t v) {
    for (int k = 0; k < 4; ++k) h[at + k] = static_cast<uint8_t>(v >> (8 * k));
  };
  h[0] = 'B';
  h[1] = 'M';
  put32(2, 54 + data);                        // file size
  put32(10, 54);                              // pixel data offset
  put32(14, 40);                              // BITMAPINFOHEADER size
  put32(18, static_cast<uint32_t>(width));
  put32(22, static_cast<uint32_t>(height));   // positive: rows from the bottom
  h[26] = 1;                                  // planes
  h[28] = 24;                                 // bits per pixel, BI_RGB
  FILE *f = std::fopen(path, "wb");
  if (!f) return set_error(XYZGPU_E_INVALID, "bmp_write: cannot open %s", path);
  bool ok = std::fwrite(h, 1, 54, f) == 54 && std::fwrite(bgr, 1, data, f) == data;
  ok = (std::fclose(f) == 0) && ok;
  return ok ? XYZGPU_OK : set_error(XYZGPU_E_INVALID, "bmp_write: writing %s failed", path);
}

// Host-film conveniences: upload, device encode / tone map, write the file.
int xyzgpu_film_save_hdr(const char *path, const float *film, int width, int height, float spp, int xyze) {
  clear_error();
  if (!path || !film || width <= 0 || height <= 0 || !(spp > 0.0f))
    return set_error(XYZGPU_E_INVALID, "film_save_hdr: bad argument");
  size_t const n = static_cast<size_t>(width) * height;
  float *d_film = nullptr;
  uint8_t *d_px = nullptr;
  struct Free {
    float *&a;
    uint8_t *&b;
    ~Free() {
      cudaFree(a);
      cudaFree(b);
    }
  } guard{d_film, d_px};
  XYZ_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&d_film), 3 * n * sizeof(float)));
  XYZ_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&d_px), 4 * n));
  XYZ_CUDA_TRY(cudaMemcpy(d_film, film, 3 * n * sizeof(float), cudaMemcpyHostToDevice));
  int rc = xyzgpu_film_encode_rgbe(d_film, width, height, 1.0f / spp, xyze, d_px, nullptr);
  if (rc) return rc;
  std::vector<uint8_t> px(4 * n);
  XYZ_CUDA_TRY(cudaMemcpy(px.data(), d_px, 4 * n, cudaMemcpyDeviceToHost));
  return xyzgpu_hdr_write(path, px.data(), width, height, xyze);
}

int xyzgpu_film_save_bmp(const char *path, const float *film, int width, int height,
                         const xyzgpu_tonemap_params *tp) {
  clear_error();
  if (!path || !film || !tp || width <= 0 || height <= 0)
    return set_error(XYZGPU_E_INVALID, "film_save_bmp: bad argument");
  size_t const n = static_cast<size_t>(width) * height;
  size_t const bytes = ((3 * static_cast<size_t>(width) + 3) & ~size_t{3}) * height;
  float *d_film = nullptr;
  uint8_t *d_px = nullptr;
  unsigned int *d_white = nullptr;
  struct Free {
    float *&a;
    uint8_t *&b;
    unsigned int *&c;
    ~Free() {
      cudaFree(a);
      cudaFree(b);
      cudaFree(c);
    }
  } guard{d_film, d_px, d_white};
  XYZ_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&d_film), 3 * n * sizeof(float)));
  XYZ_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&d_px), bytes));
  XYZ_CUDA_TRY(cudaMalloc(reinterpret_cast<void **>(&d_white), sizeof(unsigned int)));
  XYZ_CUDA_TRY(cudaMemcpy(d_film, film, 3 * n * sizeof(float), cudaMemcpyHostToDevice));
  int rc = xyzgpu_film_tonemap(d_film, width, height, tp, d_px, d_white, nullptr);
  if (rc) return rc;
  std::vector<uint8_t> px(bytes);
  XYZ_CUDA_TRY(cudaMemcpy(px.data(), d_px, bytes, cudaMemcpyDeviceToHost));
  return xyzgpu_bmp_write(path, px.data(), width, height);
}

int xyzgpu_checkpoint_save(const char *path, const xyzgpu_render_params *rp, int spp_done, const float *film) {
  clear_error();
  if (!path || !rp || !film || rp->width <= 0 || rp->height <= 0 || spp_done < 0)
    return set_error(XYZGPU_E_INVALID, "checkpoint_save: bad argument");
  size_t const n = 3 * static_cast<size_t>(rp->width) * rp->height;
  std::string const tmp = std::string(path) + ".part";
  FILE *f = std::fopen(tmp.c_str(), "wb");
  if (!f) return set_error(XYZGPU_E_INVALID, "checkpoint_save: cannot open %s", tmp.c_str());
  uint32_t const ver = kCkptVersion, psize = sizeof(xyzgpu_render_params);
  int32_t const done = spp_done;
  uint64_t const sum = fnv1a(film, n * sizeof(float));
  bool ok = std::fwrite(kCkptMagic, 1, 8, f) == 8 && std::fwrite(&ver, 4, 1, f) == 1 &&
            std::fwrite(&psize, 4, 1, f) == 1 && std::fwrite(rp, psize, 1, f) == 1 &&
            std::fwrite(&done, 4, 1, f) == 1 && std::fwrite(&sum, 8, 1, f) == 1 &&
            std::fwrite(film, sizeof(float), n, f) == n;
  ok = (std::fclose(f) == 0) && ok;
  if (!ok || std::rename(tmp.c_str(), path) != 0) {
    std::remove(tmp.c_str());
    return set_error(XYZGPU_E_INVALID, "checkpoint_save: writing %s failed", path);
  }
  return XYZGPU_OK;
}

int xyzgpu_checkpoint_load(const char *path, xyzgpu_render_params *rp, int *spp_done, float *film) {
  clear_error();
  if (!path || !rp || !spp_done) return set_error(XYZGPU_E_INVALID, "checkpoint_load: bad argument");
  FILE *f = std::fopen(path, "rb");
  if (!f) return set_error(XYZGPU_E_INVALID, "checkpoint_load: cannot open %s", path);
  char magic[8];
  uint32_t ver = 0, psize = 0;
  int32_t done = 0;
  uint64_t sum = 0;
  xyzgpu_render_params p;
  bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, kCkptMagic, 8) == 0 &&
            std::fread(&ver, 4, 1, f) == 1 && ver == kCkptVersion && std::fread(&psize, 4, 1, f) == 1 &&
            psize == sizeof(p) && std::fread(&p, psize, 1, f) == 1 && std::fread(&done, 4, 1, f) == 1 &&
            std::fread(&sum, 8, 1, f) == 1 && p.width > 0 && p.height > 0 && done >= 0;
  if (!ok) {
    std::fclose(f);
    return set_error(XYZGPU_E_INVALID, "checkpoint_load: %s is not a checkpoint of this library", path);
  }
  *rp = p;
  *spp_done = done;
  if (film) {
    size_t const n = 3 * static_cast<size_t>(p.width) * p.height;
    ok = std::fread(film, sizeof(float), n, f) == n && fnv1a(film, n * sizeof(float)) == sum;
  }
  std::fclose(f);
  return ok ? XYZGPU_OK : set_error(XYZGPU_E_INVALID, "checkpoint_load: %s is truncated or damaged", path);
}

}  // extern "C"
