// Photo's post passes beside compose and FXAA (src/image.cpp:30-356):
// spatialClamp, the a-trous filter, bloom and the depth-of-field blur, on
// the device, each pass restating the reference's float operations in the
// reference's order.
//
//  * spatialClamp: a row kernel (7-tap blur of luminance) and a column kernel
//    (7-tap blur, clamp in place), the four buffers in one grid (z).
//  * filter: filterVar and five a-trous passes, ping-ponging between the
//    caller's buffers and a scratch copy (the sixth write lands back in the
//    caller's); the G-buffer fields the edge-stopping weight reads are packed
//    once into 48 bytes per pixel.
//  * bloom: the bright part, then five a-trous passes, each adding its
//    result to the image (ping-pong scratch).
//  * depth of field: the reference scatters pixels in stable depth order and
//    every receiving pixel stops taking weight at 0.99, so what a pixel
//    receives depends on the order of its senders. That order is per
//    receiver: the blur is a gather in which each receiver folds its
//    senders in the reference's order. The pixels of each tile of T x T
//    pixels (T >= the largest radius) are listed in that order with a sort
//    key; a receiver merges the lists of its 3 x 3 tiles by key, so it meets
//    every sender that can reach it, in order (a block per tile first keeps
//    the senders whose square reaches the tile and merges them once, so a
//    receiver only walks its tile's candidates). Without NaN depths a stable
//    sort by depth is the order by (depth, raster index), whose key is
//    (depth bits, index): each tile ranks its own pixels on the device. A
//    NaN depth (a pixel without a hit) compares false both ways in the
//    reference's comparator, so its place depends on std::stable_sort's
//    algorithm, which stable_order.cu carries out; the key is then the rank.
//    A plan (order, radii, weights) serves every blur of the same G-buffer.
#include <algorithm>
#include <cmath>
#include <vector>

#include "rmn_host.h"

namespace {

constexpr float kLumR = 0.3f, kLumG = 0.6f, kLumB = 0.1f;
__device__ __forceinline__ float lum3(float3 v) { return dot3(v, f3(kLumR, kLumG, kLumB)); }
__device__ __forceinline__ float3 xyz(float4 v) { return f3(v.x, v.y, v.z); }

// ------------------------------------------------------- spatialClamp -----
__constant__ float c_h7[7] = {0.03125f, 0.109375f, 0.21875f, 0.28125f, 0.21875f, 0.109375f, 0.03125f};

struct Bufs {
  float4* b[4];  // Dd, Ds, Id, Is (radiance, Var)
};

__global__ void clamp_rows_kernel(Bufs in, float* __restrict__ b1, int W, int H) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= W) return;
  const float4* r = in.b[z] + (size_t)y * W;
  float sum = 0.0f;
  for (int dx = -3; dx <= 3; ++dx) {
    int nx = x + dx;
    if (nx >= 0 && nx < W) sum += lum3(xyz(r[nx])) * c_h7[dx + 3];
  }
  b1[(size_t)z * W * H + (size_t)y * W + x] = sum;
}

__global__ void clamp_cols_kernel(Bufs io, const float* __restrict__ b1, int W, int H) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= W) return;
  const float* c = b1 + (size_t)z * W * H;
  float sum = 0.0f;
  for (int dy = -3; dy <= 3; ++dy) {
    int ny = y + dy;
    if (ny >= 0 && ny < H) sum += c[(size_t)ny * W + x] * c_h7[dy + 3];
  }
  float4& p = io.b[z][(size_t)y * W + x];
  const float l = lum3(xyz(p));
  const float h3 = c_h7[3];
  const float bl = sum - h3 * h3 * l;
  if (l > 36.0f * bl) {
    const float s = bl / (l + RMN_EPS) / (1.0f - h3 * h3);
    p.x *= s;
    p.y *= s;
    p.z *= s;
  }
}

// ------------------------------------------------------------- filter -----
// Guide record of a pixel for the edge-stopping weight (48 B):
// (position, metallic), (surface normal, opacity), (shape normal, roughness).
__global__ void guide_kernel(const float* __restrict__ gbuf, float4* __restrict__ guide, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* g = gbuf + (size_t)RMN_GBUFFER_FLOATS * i;
  guide[3 * (size_t)i] = make_float4(g[6], g[7], g[8], g[16]);
  guide[3 * (size_t)i + 1] = make_float4(g[12], g[13], g[14], g[17]);
  guide[3 * (size_t)i + 2] = make_float4(g[9], g[10], g[11], g[15]);
}

// filterVar, src/image.cpp:84-108.
__global__ void filter_var_kernel(Bufs in, Bufs out, int W, int H) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= W) return;
  const float h[3] = {0.25f, 0.5f, 0.25f};
  const float4* r = in.b[z];
  float3 E = f3(0.0f);
  float E2 = 0.0f, V = 0.0f;
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) {
      int nx = x + dx, ny = y + dy;
      if (nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
      const float4 q = r[(size_t)ny * W + nx];
      const float wt = h[dx + 1] * h[dy + 1];
      E += xyz(q) * wt;
      E2 += dot3(xyz(q), xyz(q)) * wt;
      V += q.w * wt;
    }
  const size_t i = (size_t)y * W + x;
  const float4 p = r[i];
  out.b[z][i] = make_float4(p.x, p.y, p.z, V + E2 - dot3(E, E));
}

// filterRadiance(..., step), src/image.cpp:160-199, with getWeight
// (:110-158; sigma_z = sigma_l = sigma_m = 1, sigma_n = 1024, eps 1e-2,
// eps_r 4e-2; every pixel's specular is the HitInfo default 0.04, so its
// difference is 0).
//
// A thread filters one pixel of all four buffers: of a tap's weight only the
// radiance term and the specular buffers' roughness factor differ between
// them, while the normal term (powf), the plane distance (a normalisation, a
// square root and three divisions) and the material term are the geometry's.
// The pass is bound by instruction issue; a thread per pixel and buffer
// computed the geometry's part four times. 1920x1080, a pass: 1.09 ms before,
// 0.6 ms with all four; 6 blocks per SM (80 registers) against the 94 it would
// take: another 0.05 ms less.
__constant__ float c_h5[5] = {0.0625f, 0.25f, 0.375f, 0.25f, 0.0625f};

__global__ void __launch_bounds__(128, 6) filter_pass_kernel(Bufs in, Bufs out, const float4* __restrict__ guide, int W,
                                                          int H, int step) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= W || y >= H) return;
  const size_t i = (size_t)y * W + x;
  float3 rb[4];
  float vb[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    rb[b] = f3(0.0f);
    vb[b] = 0.0f;
  }
  const float4 p0 = guide[3 * i];
  if (any_finite3(xyz(p0))) {
    const float4 p1 = guide[3 * i + 1], p2 = guide[3 * i + 2];
    const float rough = p2.w < 4e-2f ? 4e-2f : p2.w;
    float3 Lp[4];
    float ws[4], sl[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float4 v = in.b[b][i];
      Lp[b] = xyz(v);
      sl[b] = 1.0f * sqrtf(v.w) + 1e-2f;
      ws[b] = 0.0f;
    }
#pragma unroll 1
    for (int dy = -2; dy <= 2; ++dy) {
      const int ny = y + dy * step;
      if (ny < 0 || ny >= H) continue;
#pragma unroll 1
      for (int dx = -2; dx <= 2; ++dx) {
        const int nx = x + dx * step;
        if (nx < 0 || nx >= W) continue;
        const float hh = c_h5[dx + 2] * c_h5[dy + 2];
        const size_t j = (size_t)ny * W + nx;
        const bool centre = dx == 0 && dy == 0;
        float4 Lq[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) Lq[b] = in.b[b][j];
        // the geometry's part: w, and k before and after the radiance term
        float w = 0.0f, tt = 0.0f, md = 0.0f;
        if (!centre) {
          const float4 q0 = guide[3 * j], q1 = guide[3 * j + 1];
          if (any_finite3(xyz(q0))) {
            const float d = dot3(xyz(p1), xyz(q1));
            w = powf(0.0f < d ? d : 0.0f, 1024.0f);
            if (w < 1e-6f) {
              w = 0.0f;
            } else {
              const float3 dir = norm3(xyz(q0) - xyz(p0));
              const float st = fabsf(dot3(xyz(p2), dir));
              tt = st / (sqrtf(1.0f - st * st) + RMN_EPS);
              md = len3(f3(p0.w - q0.w, 0.04f - 0.04f, p1.w - q1.w));
            }
          }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          float wt = hh;
          if (!centre) {
            float e = 0.0f;
            if (w != 0.0f) {  // a NaN goes on and is dropped below
              float k = 0.0f;
              k += -tt / 1.0f;
              k += -(len3(Lp[b] - xyz(Lq[b])) / sl[b]);
              k += -md / 1.0f;
              if (!(k < -7.5f)) {
                e = w * expf(k);
                if (b & 1) e *= rough;  // Ds, Is
                if (!isfinite(e)) e = 0.0f;
              }
            }
            wt *= e;
          }
          ws[b] += wt;
          rb[b] += xyz(Lq[b]) * wt;
          vb[b] += Lq[b].w * wt * wt;
        }
      }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      rb[b] = rb[b] / ws[b];
      vb[b] /= ws[b] * ws[b];
    }
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) out.b[b][i] = make_float4(rb[b].x, rb[b].y, rb[b].z, vb[b]);
}

// --------------------------------------------------------------- bloom ----
__global__ void bloom_init_kernel(const float* __restrict__ rgb, float3* __restrict__ bc, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 p = f3(rgb[3 * (size_t)i], rgb[3 * (size_t)i + 1], rgb[3 * (size_t)i + 2]);
  const float c = lum3(p);
  float3 b = f3(0.0f);
  if (!(c < 1.0f)) {
    b = p / powf(c, 0.65f);
    b.x = b.x - 1.0f < 0.0f ? 0.0f : b.x - 1.0f;  // std::max(v - 1, 0)
    b.y = b.y - 1.0f < 0.0f ? 0.0f : b.y - 1.0f;
    b.z = b.z - 1.0f < 0.0f ? 0.0f : b.z - 1.0f;
  }
  bc[i] = b;
}

__device__ __forceinline__ float3 gamma3(float3 p) {  // Photo::gammaCorrection, src/image.cpp:454-468
  p = max3(p, f3(0.0f));
  const float c = lum3(p);
  if (c > 0.75f) p = p / c * (tanhf(3.0f * (c - 0.75f)) / 3.0f + 0.75f);
  p = min3(p, f3(1.0f));
  const float e = 1.0f / 2.2f;
  return f3(powf(p.x, e), powf(p.y, e), powf(p.z, e));
}

// One bloom pass: out = blur(in, step) (not kept by the LAST); rgb = base +
// out / 6, gamma-corrected when the last pass is asked for it. base: the
// image before bloom in the first pass, then rgb itself.
template <bool LAST>
__global__ void bloom_pass_kernel(const float3* __restrict__ in, float3* __restrict__ out, const float* base,
                                  float* rgb, int W, int H, int step, bool gamma) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= W) return;
  const float h[5] = {0.0625f, 0.25f, 0.375f, 0.25f, 0.0625f};
  float3 col = f3(0.0f);
  for (int ky = -2; ky <= 2; ++ky)
    for (int kx = -2; kx <= 2; ++kx) {
      int nx = x + kx * step, ny = y + ky * step;
      if (nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
      col += in[(size_t)ny * W + nx] * h[ky + 2] * h[kx + 2];
    }
  const size_t i = (size_t)y * W + x;
  if (!LAST) out[i] = col;
  float3 p = f3(base[3 * i], base[3 * i + 1], base[3 * i + 2]) + col / 6.0f;
  if (LAST && gamma) p = gamma3(p);
  rgb[3 * i] = p.x;
  rgb[3 * i + 1] = p.y;
  rgb[3 * i + 2] = p.z;
}

// ----------------------------------------------------- depth of field -----
// float -> int of the radii: truncation, 0 for NaN (CUDA's and aarch64's
// conversion; in C++ the conversion of NaN is undefined).
__host__ __device__ __forceinline__ int dof_int(float v) {
  if (v != v) return 0;
  if (v >= 2147483647.0f) return 2147483647;
  if (v <= -2147483648.0f) return (-2147483647 - 1);
  return (int)v;
}
__host__ __device__ __forceinline__ float dof_coc(float coc, float focus, float depth) {
  const float c = coc * fabsf(1.0f - focus / depth) + RMN_EPS;
  return 96.0f < c ? 96.0f : c;  // std::min(..., MaxCoC)
}

// depth = length(position - camera); flags[0] |= a NaN depth.
__global__ void depth_kernel(const float* __restrict__ gbuf, float3 cam, float* __restrict__ depth, int n,
                             int* __restrict__ flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* g = gbuf + (size_t)RMN_GBUFFER_FLOATS * i;
  const float d = len3(f3(g[6], g[7], g[8]) - cam);
  depth[i] = d;
  if (d != d) atomicOr(&flags[0], 1);
}

// Per sending pixel: CoC0, its total weight (the reference's two loops per
// row, inwards from the disc's edge until a weight reaches 1), radius.
// flags[1] = max radius.
__global__ void dof_source_kernel(const float* __restrict__ depth, float coc, float focus, float4* __restrict__ src,
                                  int n, int* __restrict__ flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float c0 = dof_coc(coc, focus, depth[i]);
  const int radius = dof_int(c0);
  atomicMax(&flags[1], radius);
  float tw = 0.0f;
  for (int dy = -radius; dy <= radius; ++dy) {
    const int xlen = dof_int(sqrtf(c0 * c0 - (float)(dy * dy)));
    int xl, xr;
    for (xl = -xlen; xl <= 0; xl++) {
      float w = c0 - sqrtf((float)(xl * xl + dy * dy));
      w = 1.0f < w ? 1.0f : w;
      if (w == 1.0f) break;
      tw += w;
    }
    for (xr = xlen; xr > 0; xr--) {
      float w = c0 - sqrtf((float)(xr * xr + dy * dy));
      w = 1.0f < w ? 1.0f : w;
      if (w == 1.0f) break;
      tw += w;
    }
    tw += (float)(xr - xl + 1);
  }
  src[i] = make_float4(c0, tw, __int_as_float(radius), 0.0f);
}

// Tile t = (tx, ty) of a T-grid covers x in [tx T, min(W, tx T + T)) and
// likewise y; its list occupies [tile_start[t], tile_start[t + 1]).
// `order`: the high word of a pixel's key -- its depth's bits, or (NaN depths)
// its rank in the sorted order.
__global__ void dof_rank_kernel(const unsigned* __restrict__ order, const int* __restrict__ tile_start, int W, int H,
                                int T, int TW, unsigned long long* __restrict__ key, int* __restrict__ pix) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= W) return;
  const int tx = x / T, ty = y / T;
  const int x0 = tx * T, y0 = ty * T, x1 = min(W, x0 + T), y1 = min(H, y0 + T);
  const int p = y * W + x;
  const unsigned long long kp = ((unsigned long long)order[p] << 32) | (unsigned)p;
  int rank = 0;
  for (int qy = y0; qy < y1; ++qy)
    for (int qx = x0; qx < x1; ++qx) {
      const int q = qy * W + qx;
      const unsigned long long kq = ((unsigned long long)order[q] << 32) | (unsigned)q;
      rank += kq < kp ? 1 : 0;
    }
  const int slot = tile_start[ty * TW + tx] + rank;
  key[slot] = kp;
  pix[slot] = p;
}

// Per receiving tile: the senders of its 3 x 3 tiles whose square of
// half-width radius touches the tile, in the reference's order. A block per
// tile compacts each neighbour list (order kept) into `tmp`, then places every
// survivor at its rank in the merged order: its index in its own list plus,
// for every other list, the number of survivors with a smaller key.
constexpr int kCandThreads = 256;

__device__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int w = lane < kCandThreads / 32 ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kCandThreads / 32) warp_sums[lane] = w;  // inclusive
  }
  __syncthreads();
  const int before = (wid > 0 ? warp_sums[wid - 1] : 0) + x - v;
  total = warp_sums[kCandThreads / 32 - 1];
  __syncthreads();
  return before;
}

__global__ void __launch_bounds__(kCandThreads) dof_candidates_kernel(
    const float4* __restrict__ src, const int* __restrict__ tile_start, const unsigned long long* __restrict__ key,
    const int* __restrict__ pix, const long long* __restrict__ cand_off, int W, int H, int T, int TW, int TH,
    unsigned long long* __restrict__ tmp_key, int* __restrict__ tmp_pix, int* __restrict__ cand,
    int* __restrict__ cand_count) {
  __shared__ int warp_sums[kCandThreads / 32];
  __shared__ int lst_begin[9], lst_len[9];
  const int t = blockIdx.x, tx = t % TW, ty = t / TW;
  const int x0 = tx * T, y0 = ty * T, x1 = min(W, x0 + T) - 1, y1 = min(H, y0 + T) - 1;
  const long long base = cand_off[t];
  int nl = 0, filled = 0;
  for (int j = ty - 1; j <= ty + 1; ++j)
    for (int i = tx - 1; i <= tx + 1; ++i) {
      if (i < 0 || i >= TW || j < 0 || j >= TH) continue;
      const int u = j * TW + i, b = tile_start[u], len = tile_start[u + 1] - b;
      int kept = 0;
      for (int c0 = 0; c0 < len; c0 += kCandThreads) {
        const int c = c0 + threadIdx.x;
        bool keep = false;
        int s = 0;
        if (c < len) {
          s = pix[b + c];
          const int sx = s % W, sy = s / W, r = __float_as_int(src[s].z);
          keep = sx - r <= x1 && sx + r >= x0 && sy - r <= y1 && sy + r >= y0;
        }
        int total;
        const int at = block_exclusive_scan(keep ? 1 : 0, warp_sums, total);
        if (keep) {
          tmp_key[base + filled + kept + at] = key[b + c];
          tmp_pix[base + filled + kept + at] = s;
        }
        kept += total;
      }
      if (threadIdx.x == 0) {
        lst_begin[nl] = filled;
        lst_len[nl] = kept;
      }
      filled += kept;
      ++nl;
    }
  __syncthreads();
  for (int c = threadIdx.x; c < filled; c += kCandThreads) {
    const unsigned long long k = tmp_key[base + c];
    int rank = 0;
    for (int l = 0; l < nl; ++l) {
      const int b = lst_begin[l], len = lst_len[l];
      if (c >= b && c < b + len) {
        rank += c - b;
        continue;
      }
      int lo = 0, hi = len;  // survivors of list l with a smaller key
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tmp_key[base + b + mid] < k) lo = mid + 1;
        else hi = mid;
      }
      rank += lo;
    }
    cand[base + rank] = tmp_pix[base + c];
  }
  if (threadIdx.x == 0) cand_count[t] = filled;
}

// The receivers of a tile: its candidates folded in order, for one image or
// two at once (the weights are the plan's alone). A warp has 8 x 4 receivers;
// a block stages the tile's candidates in shared memory, kFoldChunk at a time,
// and each warp goes through those whose square of half-width radius touches
// its 32 receivers: a lane tests one candidate, a vote makes the list, in
// order. Positions are relative to the tile (at most 3 x 96 a side: exact in
// float, as are their squares).
//
// The reference's tests of a pair, |dx| <= int(sqrt(c0^2 - dy^2)) and the
// weight min(1, c0 - sqrt(dx^2 + dy^2)) / total, need neither root nor division
// where the pair lies clearly inside: dx^2 <= c0^2 - dy^2 as floats makes the
// root at least |dx| (the integer's square is exact and the root's rounding
// monotone), and dx^2 + dy^2 < (c0 - 1)^2 (1 - 1e-6) makes c0 less the root at
// least 1 (the margin is above the three roundings), so that the weight is
// 1 / total, found once per candidate. What lies below 1 - 1e-6 times the
// square is outside; the rest takes the reference's operations.
//
// A receiver that has gained so much that no weight of at least eps can be
// added any more (0.99 - gained below eps / 2; a candidate's weight is at least
// eps or skipped, and what is left of it after the cap is below eps, so it is
// skipped) is done, and a block whose receivers are all done stops. Not so a
// receiver whose own weight is NaN (a pixel without a hit): that weight is not
// skipped and reaches itself alone, so it waits for its own turn.
constexpr int kFoldThreads = 256;
constexpr int kFoldChunk = 128;

template <int NI>
__global__ void __launch_bounds__(kFoldThreads) dof_fold_kernel(
    const float* __restrict__ in0, const float* __restrict__ in1, const float4* __restrict__ src,
    const long long* __restrict__ cand_off, const int* __restrict__ cand, const int* __restrict__ cand_count, int W,
    int H, int T, int TW, float* __restrict__ out0, float* __restrict__ out1) {
  __shared__ float4 place[kFoldChunk];       // x, y, radius, c0
  __shared__ float2 weight[kFoldChunk];      // the sender's total weight, (c0 - 1)^2 (1 - 1e-6) or 0
  __shared__ float4 colour[NI][kFoldChunk];  // rgb, 1 / the total weight
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  const int rect = (blockIdx.y * blockDim.x + threadIdx.x) >> 5, across = (T + 7) / 8;
  const int x0 = (t % TW) * T, y0 = (t / TW) * T;
  const int ex = (rect % across) * 8, ey = (rect / across) * 4;  // the warp's receivers in the tile
  const int rx = ex + (lane & 7), ry = ey + (lane >> 3);
  const bool receiver = rx < T && ry < T && x0 + rx < W && y0 + ry < H;
  const float wx = (float)ex, wy = (float)ey, x = (float)rx, y = (float)ry;
  const int* c = cand + cand_off[t];
  const int n = cand_count[t];
  float3 blur[NI];
  float gained = 0.0f;
#pragma unroll
  for (int m = 0; m < NI; ++m) blur[m] = f3(0.0f);
  bool done = !receiver, fills = false;
  if (receiver) {
    const float4 own = src[(size_t)(y0 + ry) * W + x0 + rx];
    const float w = (1.0f < own.x ? 1.0f : own.x) / own.y;
    fills = w == w;
  }
  for (int k0 = 0; k0 < n; k0 += kFoldChunk) {
    if (__syncthreads_and(done)) break;
    const int len = min(kFoldChunk, n - k0);
    for (int k = threadIdx.x; k < len; k += blockDim.x) {
      const int s = c[k0 + k];
      const float4 sv = src[s];
      place[k] = make_float4((float)(s % W - x0), (float)(s / W - y0), (float)__float_as_int(sv.z), sv.x);
      weight[k] = make_float2(sv.y, sv.x > 1.0f ? (sv.x - 1.0f) * (sv.x - 1.0f) * (1.0f - 1e-6f) : 0.0f);
      const float inv = 1.0f / sv.y;
      const size_t s3 = 3 * (size_t)s;
      colour[0][k] = make_float4(in0[s3], in0[s3 + 1], in0[s3 + 2], inv);
      if (NI > 1) colour[NI - 1][k] = make_float4(in1[s3], in1[s3 + 1], in1[s3 + 2], inv);
    }
    __syncthreads();
    for (int kk = 0; kk < len; kk += 32) {
      bool touches = false;
      if (kk + lane < len) {
        const float4 pl = place[kk + lane];
        touches = pl.x + pl.z >= wx && pl.x - pl.z <= wx + 7.0f && pl.y + pl.z >= wy && pl.y - pl.z <= wy + 3.0f;
      }
      unsigned list = __ballot_sync(0xffffffffu, touches);
      if (done) continue;
      while (list) {
        const int k = kk + __ffs(list) - 1;
        list &= list - 1;
        const float4 pl = place[k];
        const float dx = x - pl.x, dy = y - pl.y, c0 = pl.w;
        if (fabsf(dy) > pl.z || fabsf(dx) > pl.z) continue;  // the disc's half width is at most the radius
        const float dx2 = dx * dx, dy2 = dy * dy, half2 = c0 * c0 - dy2;
        if (!(dx2 <= half2)) {
          if (half2 < dx2 * (1.0f - 1e-6f)) continue;
          const float xlen = (float)dof_int(sqrtf(half2));
          if (fabsf(dx) > xlen) continue;
        }
        float w;
        if (dx2 + dy2 < weight[k].y) {
          w = colour[0][k].w;
        } else {
          w = c0 - sqrtf(dx2 + dy2);
          w = (1.0f < w ? 1.0f : w) / weight[k].x;
        }
        if (w < RMN_EPS) continue;
        if (gained + w > 0.99f) w = 0.99f - gained;
        if (w < RMN_EPS) continue;
#pragma unroll
        for (int m = 0; m < NI; ++m) {
          const float4 v = colour[m][k];
          blur[m] += f3(v.x, v.y, v.z) * w;
        }
        gained += w;
      }
      done = done || (fills && 0.99f - gained < 0.5f * RMN_EPS);
    }
  }
  if (!receiver) return;
  const size_t i = (size_t)(y0 + ry) * W + x0 + rx;
#pragma unroll
  for (int m = 0; m < NI; ++m) {
    const float3 o = blur[m] / gained;
    float* out = m == 0 ? out0 : out1;
    out[3 * i] = o.x;
    out[3 * i + 1] = o.y;
    out[3 * i + 2] = o.z;
  }
}

__global__ void gamma_kernel(const float* in, float* out, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float3 p = gamma3(f3(in[3 * (size_t)i], in[3 * (size_t)i + 1], in[3 * (size_t)i + 2]));
  out[3 * (size_t)i] = p.x;
  out[3 * (size_t)i + 1] = p.y;
  out[3 * (size_t)i + 2] = p.z;
}

struct DevScratch {
  std::vector<void*> ptrs;
  cudaStream_t st;
  cudaError_t err = cudaSuccess;
  template <class T>
  T* get(size_t count) {
    void* p = nullptr;
    if (err != cudaSuccess) return nullptr;
    err = rmn::staging_malloc(&p, count * sizeof(T) + 16, st);
    if (err != cudaSuccess) return nullptr;
    ptrs.push_back(p);
    return static_cast<T*>(p);
  }
  ~DevScratch() {
    for (void* p : ptrs) cudaFreeAsync(p, st);
  }
};

dim3 row_grid(int W, int H, int z = 1) { return dim3((W + 127) / 128, H, z); }

}  // namespace

namespace rmn {

cudaError_t launch_spatial_clamp(float* const bufs[4], int W, int H, cudaStream_t st) {
  DevScratch sc{{}, st};
  float* b1 = sc.get<float>((size_t)4 * W * H);
  if (sc.err != cudaSuccess) return sc.err;
  Bufs b;
  for (int k = 0; k < 4; ++k) b.b[k] = reinterpret_cast<float4*>(bufs[k]);
  clamp_rows_kernel<<<row_grid(W, H, 4), 128, 0, st>>>(b, b1, W, H);
  clamp_cols_kernel<<<row_grid(W, H, 4), 128, 0, st>>>(b, b1, W, H);
  return cudaGetLastError();
}

cudaError_t launch_filter(float* const bufs[4], const float* gbuf, int W, int H, cudaStream_t st) {
  const size_t n = (size_t)W * H;
  DevScratch sc{{}, st};
  float4* guide = sc.get<float4>(3 * n);
  float4* tmp = sc.get<float4>(4 * n);
  if (sc.err != cudaSuccess) return sc.err;
  Bufs A, B;
  for (int k = 0; k < 4; ++k) {
    A.b[k] = reinterpret_cast<float4*>(bufs[k]);
    B.b[k] = tmp + k * n;
  }
  guide_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(gbuf, guide, (int)n);
  filter_var_kernel<<<row_grid(W, H, 4), 128, 0, st>>>(A, B, W, H);
  // passes of step 1, 2, 4, 8, 16: B -> A -> B -> A -> B -> A
  bool toA = true;
  for (int step = 1; step <= 16; step *= 2) {
    const dim3 grid((W + 31) / 32, (H + 3) / 4), block(32, 4);
    if (toA) filter_pass_kernel<<<grid, block, 0, st>>>(B, A, guide, W, H, step);
    else filter_pass_kernel<<<grid, block, 0, st>>>(A, B, guide, W, H, step);
    toA = !toA;
  }
  return cudaGetLastError();
}

// Photo::bloom of `in` into rgb (which may be `in`), then gammaCorrection when
// asked for.
cudaError_t launch_bloom(const float* in, float* rgb, int W, int H, bool gamma, cudaStream_t st) {
  const size_t n = (size_t)W * H;
  DevScratch sc{{}, st};
  float3* a = sc.get<float3>(n);
  float3* b = sc.get<float3>(n);
  if (sc.err != cudaSuccess) return sc.err;
  bloom_init_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, a, (int)n);
  for (int step = 1; step <= 8; step *= 2) {
    bloom_pass_kernel<false><<<row_grid(W, H), 128, 0, st>>>(a, b, step == 1 ? in : rgb, rgb, W, H, step, false);
    std::swap(a, b);
  }
  bloom_pass_kernel<true><<<row_grid(W, H), 128, 0, st>>>(a, b, rgb, rgb, W, H, 16, gamma);
  return cudaGetLastError();
}

struct DofPlan {
  int W = 0, H = 0, T = 0, TW = 0, TH = 0;
  float4* src = nullptr;
  int* tile_start = nullptr;
  unsigned long long* key = nullptr;
  int* pix = nullptr;
  // per receiving tile: its candidate senders in order
  long long* cand_off = nullptr;
  int* cand = nullptr;
  int* cand_count = nullptr;
  float* out = nullptr;
  std::vector<void*> allocs;
};

void dof_plan_destroy(DofPlan* p, cudaStream_t st) {
  if (!p) return;
  for (void* a : p->allocs) cudaFreeAsync(a, st);
  delete p;
}

// Order, radii and weights of the depth-of-field blur of one G-buffer and
// camera. Synchronises `st` (the tile size depends on the largest radius).
cudaError_t dof_plan_create(const float* gbuf, int W, int H, float focus, float coc, const float cam[3],
                            cudaStream_t st, DofPlan** out) {
  *out = nullptr;
  const int n = W * H;
  DofPlan* p = new DofPlan();
  p->W = W;
  p->H = H;
  cudaError_t e = cudaSuccess;
  auto alloc = [&](size_t bytes) -> void* {
    void* q = nullptr;
    if (e == cudaSuccess) e = rmn::staging_malloc(&q, bytes + 16, st);
    if (e == cudaSuccess) p->allocs.push_back(q);
    return e == cudaSuccess ? q : nullptr;
  };
  float* depth = static_cast<float*>(alloc(sizeof(float) * n));
  int* flags = static_cast<int*>(alloc(2 * sizeof(int)));
  p->src = static_cast<float4*>(alloc(sizeof(float4) * n));
  p->key = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * n));
  p->pix = static_cast<int*>(alloc(sizeof(int) * n));
  p->out = static_cast<float*>(alloc(sizeof(float) * 3 * n));
  int hflags[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0, 2 * sizeof(int), st);
  if (e == cudaSuccess) {
    depth_kernel<<<(n + 255) / 256, 256, 0, st>>>(gbuf, f3(cam[0], cam[1], cam[2]), depth, n, flags);
    dof_source_kernel<<<(n + 255) / 256, 256, 0, st>>>(depth, coc, focus, p->src, n, flags);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(hflags, flags, sizeof hflags, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    dof_plan_destroy(p, st);
    return e;
  }
  p->T = std::max(hflags[1], 8);
  p->TW = (W + p->T - 1) / p->T;
  p->TH = (H + p->T - 1) / p->T;
  std::vector<int> tile_start((size_t)p->TW * p->TH + 1, 0);
  for (int ty = 0; ty < p->TH; ++ty)
    for (int tx = 0; tx < p->TW; ++tx) {
      const int w = std::min(W, tx * p->T + p->T) - tx * p->T, h = std::min(H, ty * p->T + p->T) - ty * p->T;
      tile_start[(size_t)ty * p->TW + tx + 1] = w * h;
    }
  for (size_t t = 0; t + 1 < tile_start.size(); ++t) tile_start[t + 1] += tile_start[t];
  p->tile_start = static_cast<int*>(alloc(sizeof(int) * tile_start.size()));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(p->tile_start, tile_start.data(), sizeof(int) * tile_start.size(), cudaMemcpyHostToDevice, st);
  const unsigned* order = reinterpret_cast<const unsigned*>(depth);  // non-negative: their bits ascend with them
  if (e == cudaSuccess && hflags[0]) {
    // NaN depths: the order the reference's std::stable_sort gives them
    unsigned* rank = static_cast<unsigned*>(alloc(sizeof(unsigned) * n));
    if (e == cudaSuccess) e = rmn::launch_stable_order(depth, n, rank, st);
    order = rank;
  }
  if (e == cudaSuccess) {
    dof_rank_kernel<<<row_grid(W, H), 128, 0, st>>>(order, p->tile_start, W, H, p->T, p->TW, p->key, p->pix);
    e = cudaGetLastError();
  }
  // candidate lists: capacity of tile t = the pixels of its 3 x 3 tiles
  const size_t ntiles = (size_t)p->TW * p->TH;
  std::vector<long long> cand_off(ntiles + 1, 0);
  for (int ty = 0; ty < p->TH; ++ty)
    for (int tx = 0; tx < p->TW; ++tx) {
      long long cap = 0;
      for (int j = ty - 1; j <= ty + 1; ++j)
        for (int i = tx - 1; i <= tx + 1; ++i)
          if (i >= 0 && i < p->TW && j >= 0 && j < p->TH) {
            const size_t u = (size_t)j * p->TW + i;
            cap += tile_start[u + 1] - tile_start[u];
          }
      cand_off[(size_t)ty * p->TW + tx + 1] = cap;
    }
  for (size_t t = 0; t < ntiles; ++t) cand_off[t + 1] += cand_off[t];
  const size_t total = (size_t)cand_off[ntiles];
  p->cand_off = static_cast<long long*>(alloc(sizeof(long long) * (ntiles + 1)));
  p->cand = static_cast<int*>(alloc(sizeof(int) * total));
  p->cand_count = static_cast<int*>(alloc(sizeof(int) * ntiles));
  unsigned long long* tmp_key = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * total));
  int* tmp_pix = static_cast<int*>(alloc(sizeof(int) * total));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(p->cand_off, cand_off.data(), sizeof(long long) * (ntiles + 1), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    dof_candidates_kernel<<<(unsigned)ntiles, kCandThreads, 0, st>>>(p->src, p->tile_start, p->key, p->pix,
                                                                     p->cand_off, W, H, p->T, p->TW, p->TH, tmp_key,
                                                                     tmp_pix, p->cand, p->cand_count);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // host arrays were copied from
  if (e != cudaSuccess) {
    dof_plan_destroy(p, st);
    return e;
  }
  *out = p;
  return cudaSuccess;
}

// Photo::depthFeildBlur of in0 into out0 and, unless null, of in1 into out1,
// with a plan of their G-buffer.
cudaError_t dof_apply(const DofPlan* p, const float* in0, float* out0, const float* in1, float* out1,
                      cudaStream_t st) {
  const int per_tile = 32 * ((p->T + 7) / 8) * ((p->T + 3) / 4);  // 8 x 4 receivers a warp
  const int threads = std::min(kFoldThreads, per_tile);
  const dim3 grid((unsigned)(p->TW * p->TH), (per_tile + threads - 1) / threads);
  if (in1)
    dof_fold_kernel<2><<<grid, threads, 0, st>>>(in0, in1, p->src, p->cand_off, p->cand, p->cand_count, p->W, p->H,
                                                 p->T, p->TW, out0, out1);
  else
    dof_fold_kernel<1><<<grid, threads, 0, st>>>(in0, nullptr, p->src, p->cand_off, p->cand, p->cand_count, p->W,
                                                 p->H, p->T, p->TW, out0, nullptr);
  return cudaGetLastError();
}

// The same in place on rgb.
cudaError_t dof_apply(const DofPlan* p, float* rgb, cudaStream_t st) {
  cudaError_t e = dof_apply(p, rgb, p->out, nullptr, nullptr, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(rgb, p->out, sizeof(float) * 3 * (size_t)p->W * p->H, cudaMemcpyDeviceToDevice, st);
  return e;
}

cudaError_t launch_dof(float* rgb, const float* gbuf, int W, int H, float focus, float coc, const float cam[3],
                       cudaStream_t st) {
  DofPlan* p = nullptr;
  cudaError_t e = dof_plan_create(gbuf, W, H, focus, coc, cam, st, &p);
  if (e != cudaSuccess) return e;
  e = dof_apply(p, rgb, st);
  dof_plan_destroy(p, st);
  return e;
}

// Photo::gammaCorrection of n pixels; in == out allowed.
cudaError_t launch_gamma(const float* in, float* out, int n, cudaStream_t st) {
  gamma_kernel<<<(n + 255) / 256, 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

}  // namespace rmn
