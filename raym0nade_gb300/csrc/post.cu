// Post passes over the render buffers: Photo::shade + gammaCorrection
// (src/image.cpp:215-246, 454-468) and Photo::FXAA (src/image.cpp:358-452).
//
// FXAA reads, per output pixel, its 3x3 luminance neighbourhood and up to 12
// samples marching in +x or +y (never negative: the step is
// clamp(edge / range, -2, 2) of two non-negative numbers). The reference's
// step length is 1/width for a horizontal edge but is applied along y, and
// 1/height along x for a vertical one, so the march reaches at most
// 24 * H / W rows or 24 * W / H columns. A block computes luminance for its
// tile plus that halo once into shared memory (luma is the only
// per-sample quantity the march needs) and fetches the colour of the winning
// sample once at the end. Samples outside the staged halo are read from
// global memory, so the result does not depend on the halo size.
#include <algorithm>
#include <cmath>

#include "rmn_host.h"

namespace {

// A block of 32 x 8 threads computes a tile of TX x TY pixels in two passes. The
// first looks at every pixel's four neighbours, copies the pixels below the
// contrast threshold and lists the others; the second takes the list, so that
// the march -- most of the work, on a fraction of the pixels -- runs on full
// warps. Only one coordinate of the samples varies in a march: the other's
// index, bounds and place in the tile are the pixel's.
constexpr int BX = 32, BY = 8, HALO_LO = 1;
constexpr int kTileMost = 64 * 16;

__device__ __forceinline__ float luma3(const float* p) { return p[0] * 0.3f + p[1] * 0.6f + p[2] * 0.1f; }

__global__ void __launch_bounds__(BX* BY) fxaa_kernel(const float* __restrict__ in, float* __restrict__ out, int W,
                                                       int H, int SW, int SH, int TX, int TY) {
  extern __shared__ float lum_s[];
  __shared__ uint16_t list[kTileMost];
  __shared__ int listed;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
  const int tid = threadIdx.y * BX + threadIdx.x;
  if (tid == 0) listed = 0;
  for (int ly = threadIdx.y; ly < SH; ly += BY) {
    const float* row = in + 3 * (size_t)min(max(y0 - HALO_LO + ly, 0), H - 1) * W;
    for (int lx = threadIdx.x; lx < SW; lx += BX)
      lum_s[ly * SW + lx] = luma3(row + 3 * (size_t)min(max(x0 - HALO_LO + lx, 0), W - 1));
  }
  __syncthreads();
  // the neighbours of a pixel are within the halo of one
  auto at = [&](int gx, int gy) { return lum_s[(gy - y0 + HALO_LO) * SW + gx - x0 + HALO_LO]; };
#pragma unroll 1
  for (int ey = threadIdx.y; ey < TY; ey += BY)
#pragma unroll 1
    for (int ex = threadIdx.x; ex < TX; ex += BX) {
      const int x = x0 + ex, y = y0 + ey;
      bool edge = false;
      if (x < W && y < H) {
        const float M = at(x, y);
        const float N = y > 0 ? at(x, y - 1) : M, S = y < H - 1 ? at(x, y + 1) : M;
        const float E = x < W - 1 ? at(x + 1, y) : M, Wl = x > 0 ? at(x - 1, y) : M;
        const float lo = fminf(fminf(N, S), fminf(E, Wl)), hi = fmaxf(fmaxf(N, S), fmaxf(E, Wl));
        edge = !(hi - lo < fmaxf(0.0312f, hi * 0.125f));
        if (!edge) {
          const size_t i = 3 * ((size_t)y * W + x);
          out[i] = in[i];
          out[i + 1] = in[i + 1];
          out[i + 2] = in[i + 2];
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, edge);
      int first = 0;
      if (threadIdx.x == 0 && m) first = atomicAdd(&listed, __popc(m));
      first = __shfl_sync(0xffffffffu, first, 0);
      if (edge) list[first + __popc(m & ((1u << threadIdx.x) - 1u))] = (uint16_t)(ey * TX + ex);
    }
  __syncthreads();
#pragma unroll 1
  for (int k = tid; k < listed; k += BX * BY) {
    const int x = x0 + list[k] % TX, y = y0 + list[k] / TX;
    const float M = at(x, y);
    const float N = y > 0 ? at(x, y - 1) : M, S = y < H - 1 ? at(x, y + 1) : M;
    const float E = x < W - 1 ? at(x + 1, y) : M, Wl = x > 0 ? at(x - 1, y) : M;
    const float NW = (y > 0 && x > 0) ? at(x - 1, y - 1) : M;
    const float NE = (y > 0 && x < W - 1) ? at(x + 1, y - 1) : M;
    const float SW_ = (y < H - 1 && x > 0) ? at(x - 1, y + 1) : M;
    const float SE = (y < H - 1 && x < W - 1) ? at(x + 1, y + 1) : M;
    const float range = fmaxf(fmaxf(N, S), fmaxf(E, Wl)) - fminf(fminf(N, S), fminf(E, Wl));
    const float eh = fabsf((NW + Wl + SW_) - (NE + E + SE)) * (1.0f / 3.0f);
    const float ev = fabsf((NW + N + NE) - (SW_ + S + SE)) * (1.0f / 3.0f);
    const bool horiz = eh >= ev;
    const float step = horiz ? 1.0f / float(W) : 1.0f / float(H);
    float g = (horiz ? eh : ev) / range;
    g = g < -2.0f ? -2.0f : (2.0f < g ? 2.0f : g);
    const float ux = float(x) / float(W), uy = float(y) / float(H);
    // the march's own coordinate u (of n pixels, in units of the image) and the fixed one's index
    const float u = horiz ? uy : ux, fn = horiz ? float(H) : float(W);
    const int n = horiz ? H : W;
    const int fixed = horiz ? min(max((int)(ux * float(W)), 0), W - 1) : min(max((int)(uy * float(H)), 0), H - 1);
    const int start = horiz ? y0 - HALO_LO : x0 - HALO_LO, room = horiz ? SH : SW;
    // (x / W) * W can round to the pixel before: at most one, within the halo
    const float* row = horiz ? lum_s + (fixed - x0 + HALO_LO) : lum_s + (fixed - y0 + HALO_LO) * SW;
    const int stride = horiz ? SW : 1;
    const float gs = g * step;
    float best = 0.0f;
    int found = -1;
#pragma unroll 4
    for (int i = 0; i < 12; ++i) {
      const float s = u + gs * float(i + 1);
      if (s < 0.0f || s > 1.0f) continue;
      const int v = min(max((int)(s * fn), 0), n - 1);
      const int l = v - start;
      float lum;
      if (l >= 0 && l < room) lum = row[l * stride];
      else lum = luma3(in + 3 * (horiz ? (size_t)v * W + fixed : (size_t)fixed * W + v));
      const float d = fabsf(lum - M);
      if (d > best) {
        best = d;
        found = v;
      }
    }
    const size_t i = 3 * ((size_t)y * W + x);
    const size_t j = found < 0 ? i : 3 * (horiz ? (size_t)found * W + fixed : (size_t)fixed * W + found);
    const float sub = fminf((fabsf(N + S - 2.0f * M) * 2.0f + fabsf(E + Wl - 2.0f * M)) * 0.25f, 1.0f);
    const float a = sub * 0.75f;
    out[i] = in[i] * (1.0f - a) + in[j] * a;
    out[i + 1] = in[i + 1] * (1.0f - a) + in[j + 1] * a;
    out[i + 2] = in[i + 2] * (1.0f - a) + in[j + 2] * a;
  }
}

__device__ __forceinline__ float3 ld3(const float* p) { return f3(p[0], p[1], p[2]); }

__global__ void compose_kernel(const float4* __restrict__ dd, const float4* __restrict__ ds,
                               const float4* __restrict__ id, const float4* __restrict__ is,
                               const float* __restrict__ gbuf, int n, float exposure, int opt, float* __restrict__ rgb,
                               float* __restrict__ linear) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* g = gbuf + (size_t)RMN_GBUFFER_FLOATS * i;
  float3 p;
  if (opt & 64) {
    p = (ld3(g + 9) + f3(1.0f)) / 2.0f;
  } else if (opt & 128) {
    p = (ld3(g + 12) + f3(1.0f)) / 2.0f;
  } else {
    float3 rd = f3(0.0f), rs = f3(0.0f);
    if (opt & RMN_SHADE_DIRECT) {
      if (opt & RMN_SHADE_DIFFUSE) rd += f3(dd[i]);
      if (opt & RMN_SHADE_SPECULAR) rs += f3(ds[i]);
    }
    if (opt & RMN_SHADE_INDIRECT) {
      if (opt & RMN_SHADE_DIFFUSE) rd += f3(id[i]);
      if (opt & RMN_SHADE_SPECULAR) rs += f3(is[i]);
    }
    if (!(opt & (RMN_SHADE_DIRECT | RMN_SHADE_INDIRECT))) rd = f3(1.0f);
    float3 dc = (opt & RMN_SHADE_BASECOLOR) ? ld3(g) : f3(1.0f);
    p = dc * rd + rs;
    if (opt & RMN_SHADE_EMISSION) p += ld3(g + 3) * exposure;
  }
  if (linear) {
    linear[3 * (size_t)i] = p.x;
    linear[3 * (size_t)i + 1] = p.y;
    linear[3 * (size_t)i + 2] = p.z;
  }
  if (opt & RMN_SHADE_GAMMA) {
    p = max3(p, f3(0.0f));
    float c = dot3(p, f3(0.3f, 0.6f, 0.1f));
    if (c > 0.75f) p = p / c * (tanhf(3.0f * (c - 0.75f)) / 3.0f + 0.75f);
    p = min3(p, f3(1.0f));
    const float e = 1.0f / 2.2f;
    p = f3(powf(p.x, e), powf(p.y, e), powf(p.z, e));
  }
  rgb[3 * (size_t)i] = p.x;
  rgb[3 * (size_t)i + 1] = p.y;
  rgb[3 * (size_t)i + 2] = p.z;
}

}  // namespace

namespace rmn {

cudaError_t launch_fxaa(const float* in, float* out, int w, int h, cudaStream_t stream) {
  if (w <= 0 || h <= 0) return cudaSuccess;
  int hx = (int)std::ceil(24.0 * w / h) + 2, hy = (int)std::ceil(24.0 * h / w) + 2;
  hx = std::min(hx, 96);
  hy = std::min(hy, 96);
  // the larger tile stages less halo a pixel (16:9: 2.5 luminances beside its
  // own against 6.6) where it leaves four blocks per SM. A noisy 1280x720 image: 41
  // us with 32 x 8 tiles in one pass over the pixels, 23 now; 1920x1080, mean of
  // seven exports, 53 and 37.
  const int tiles[2][2] = {{64, 16}, {32, 8}};
  int tx = 0, ty = 0;
  dim3 grid;
  for (const int* t : tiles) {
    tx = t[0];
    ty = t[1];
    grid = dim3((w + tx - 1) / tx, (h + ty - 1) / ty);
    if ((long long)grid.x * grid.y >= 4LL * device_sms()) break;
  }
  const int sw = tx + HALO_LO + hx, sh = ty + HALO_LO + hy;  // at most 161 x 26 or 74 x 113 floats
  fxaa_kernel<<<grid, dim3(BX, BY), sizeof(float) * sw * sh, stream>>>(in, out, w, h, sw, sh, tx, ty);
  return cudaGetLastError();
}

cudaError_t launch_compose(const float* dd, const float* ds, const float* id, const float* is, const float* gbuf,
                           int w, int h, float exposure, int options, float* rgb, cudaStream_t stream,
                           float* linear) {
  int n = w * h;
  compose_kernel<<<(n + 255) / 256, 256, 0, stream>>>(
      reinterpret_cast<const float4*>(dd), reinterpret_cast<const float4*>(ds), reinterpret_cast<const float4*>(id),
      reinterpret_cast<const float4*>(is), gbuf, n, exposure, options, rgb, linear);
  return cudaGetLastError();
}

}  // namespace rmn
