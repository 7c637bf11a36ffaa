// The order std::stable_sort gives pixels by depth when some depths are NaN.
//
// The reference's depth-of-field blur sorts its pixels with std::stable_sort
// and `a.depth < b.depth` (src/image.cpp:282-356). A NaN depth (a pixel
// without a hit) compares false both ways, so the result is no longer "by
// (depth, index)" but whatever the algorithm makes of it. This file carries
// the algorithm out on the device, comparison for comparison: libstdc++'s
// merge sort with a buffer of half the elements -- the two halves of the
// array sorted on their own (insertion sort of chunks of 7, then merges of
// runs of 7, 14, 28, ...), then merged, forward when the halves are of equal
// length, else from the back.
//
// A merge of runs A and B takes B's head when it is less than A's, else A's.
// With NaNs the runs consist of sorted segments between NaNs, a NaN at B's
// head holds B back until A is used up, and a NaN at A's head is taken at
// once. So only B's elements before its first NaN (f of them, ascending) pass
// elements of A: when A[i] is taken, c_i = max over k <= i of (number of
// those less than A[k]; 0 for a NaN) of B have been, and the merged places
// are i + c_i for A[i], and j + (first i with c_i > j) for B[j]. All places
// of a merge are thus found at once: a binary search, a prefix maximum and a
// second binary search. The merge from the back is the same merge of the
// reversed, negated runs.
//
// The first 8 levels run in shared memory, tiles of 1792 = 7 x 256 elements;
// each further level is four launches of up to 25 us. 1920 x 1080 pixels,
// half of them NaN: 0.7 ms, against about 48 ms for the sort on a host core
// with its copies (the export set with depth of field: 61-63 ms before, 13.4).
#include <algorithm>

#include "rmn_host.h"

namespace {

constexpr int kTileThreads = 256;
constexpr int kTile = 7 * kTileThreads;
constexpr int kRun = 1024;  // elements per block of a merge level: 256 threads x 4

// One part of the array and the runs merged in it: parts of a level are the
// two halves, or (last merge) the whole array.
struct Level {
  int base[2], len[2];  // parts
  int S;                // length of an A run
  int mirror;           // read from the back, keys negated
  int pairs;            // run pairs per part (the larger part's)
  int blocks;           // blocks of kRun elements of a run, ceil(max run / kRun)
};

__device__ __forceinline__ float key_at(const Level& L, int part, const float* key, int t) {
  const float k = key[L.mirror ? L.base[part] + L.len[part] - 1 - t : L.base[part] + t];
  return L.mirror ? -k : k;
}
__device__ __forceinline__ int place(const Level& L, int part, int t) {
  return L.mirror ? L.base[part] + L.len[part] - 1 - t : L.base[part] + t;
}
// Runs of a pair: A = [a, a + la), B = [a + la, a + la + lb) of its part.
__device__ __forceinline__ void pair_runs(const Level& L, int part, int pair, int& a, int& la, int& lb) {
  a = min(2 * L.S * pair, L.len[part]);
  la = min(L.S, L.len[part] - a);
  lb = L.mirror ? L.len[part] - a - la : min(L.S, L.len[part] - a - la);
}

// Chunks of 7 by insertion sort, then every merge inside tiles of kTile
// elements, in shared memory.
__global__ void __launch_bounds__(kTileThreads) order_tiles_kernel(const float* __restrict__ depth, int len1, int n,
                                                                   int tiles1, float* __restrict__ key,
                                                                   int* __restrict__ idx) {
  __shared__ float sk[2][kTile];
  __shared__ int si[2][kTile];
  __shared__ int sc[kTile];
  __shared__ int tm[kTileThreads], fn[kTileThreads / 2];
  const int tid = threadIdx.x;
  const int half = (int)blockIdx.x >= tiles1 ? 1 : 0;
  const int base = half ? len1 : 0, len = half ? n - len1 : len1;
  const int t0 = ((int)blockIdx.x - (half ? tiles1 : 0)) * kTile;
  const int m = min(kTile, len - t0);
  for (int k = tid; k < m; k += kTileThreads) {
    sk[0][k] = depth[base + t0 + k];
    si[0][k] = base + t0 + k;
  }
  __syncthreads();
  const int mine = min(7, max(0, m - 7 * tid));
  {
    float* p = sk[0] + 7 * tid;
    int* q = si[0] + 7 * tid;
    for (int i = 1; i < mine; ++i) {
      const float x = p[i];
      const int xi = q[i];
      int at = i;
      if (x < p[0]) {  // to the front, past NaNs too
        for (; at > 0; --at) {
          p[at] = p[at - 1];
          q[at] = q[at - 1];
        }
      } else {
        for (; x < p[at - 1]; --at) {  // ends at p[0] at the latest
          p[at] = p[at - 1];
          q[at] = q[at - 1];
        }
      }
      p[at] = x;
      q[at] = xi;
    }
  }
  int cur = 0;
  for (int s = 1; s < kTileThreads; s *= 2) {
    const int S = 7 * s;
    const int pair = tid / (2 * s), a = pair * 2 * S;
    const int la = min(S, max(0, m - a)), b = a + la, lb = min(S, max(0, m - b));
    const bool in_a = tid % (2 * s) < s;
    __syncthreads();
    if (tid < kTileThreads / 2) fn[tid] = kTile;
    __syncthreads();
    const float* k = sk[cur];
    if (!in_a)
      for (int i = 0; i < mine; ++i) {
        const float v = k[7 * tid + i];
        if (v != v) {
          atomicMin(&fn[pair], 7 * tid + i - b);
          break;
        }
      }
    __syncthreads();
    int run = 0;
    if (in_a) {
      const int f = min(lb, fn[pair]);
      for (int i = 0; i < mine; ++i) {
        const float v = k[7 * tid + i];
        int lo = 0, hi = f;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (k[b + mid] < v) lo = mid + 1;
          else hi = mid;
        }
        run = max(run, lo);
        sc[7 * tid + i] = run;
      }
    }
    tm[tid] = run;
    __syncthreads();
    for (int off = 1; off < s; off <<= 1) {  // prefix maximum over the threads of the A run
      const int v = tid % s >= off ? tm[tid - off] : 0;
      __syncthreads();
      tm[tid] = max(tm[tid], v);
      __syncthreads();
    }
    const int before = tid % s > 0 ? tm[tid - 1] : 0;
    if (in_a)
      for (int i = 0; i < mine; ++i) sc[7 * tid + i] = max(sc[7 * tid + i], before);
    __syncthreads();
    for (int i = 0; i < mine; ++i) {
      const int e = 7 * tid + i;
      int dst;
      if (in_a) {
        dst = e + sc[e];
      } else {
        const int j = e - b;
        int lo = 0, hi = la;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (sc[a + mid] > j) hi = mid;
          else lo = mid + 1;
        }
        dst = a + j + lo;
      }
      sk[cur ^ 1][dst] = sk[cur][e];
      si[cur ^ 1][dst] = si[cur][e];
    }
    cur ^= 1;
  }
  __syncthreads();
  for (int k = tid; k < m; k += kTileThreads) {
    key[base + t0 + k] = sk[cur][k];
    idx[base + t0 + k] = si[cur][k];
  }
}

// fn[part * pairs + pair] = min over its B run's NaNs (preset to a large value).
__global__ void __launch_bounds__(256) order_nan_kernel(Level L, const float* __restrict__ key, int* __restrict__ fn) {
  const int part = blockIdx.y, pair = blockIdx.x / L.blocks, blk = blockIdx.x % L.blocks;
  int a, la, lb;
  pair_runs(L, part, pair, a, la, lb);
  int first = 0x7fffffff;
  for (int q = 3; q >= 0; --q) {
    const int j = blk * kRun + q * 256 + threadIdx.x;
    if (j < lb) {
      const float v = key_at(L, part, key, a + la + j);
      if (v != v) first = j;
    }
  }
  for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
  __shared__ int w[8];
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = first;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) first = min(first, w[i]);
    if (first != 0x7fffffff) atomicMin(&fn[part * L.pairs + pair], first);
  }
}

// c[place of A[i]] = the running maximum within A[i]'s block of kRun elements;
// bm = every block's maximum.
__global__ void __launch_bounds__(256) order_bound_kernel(Level L, const float* __restrict__ key,
                                                          const int* __restrict__ fn, int* __restrict__ c,
                                                          int* __restrict__ bm) {
  const int part = blockIdx.y, pair = blockIdx.x / L.blocks, blk = blockIdx.x % L.blocks;
  int a, la, lb;
  pair_runs(L, part, pair, a, la, lb);
  const int f = min(lb, fn[part * L.pairs + pair]);
  const int i0 = blk * kRun + 4 * threadIdx.x;
  int run[4], mx = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (i0 + q < la) {
      const float v = key_at(L, part, key, a + i0 + q);
      int lo = 0, hi = f;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (key_at(L, part, key, a + la + mid) < v) lo = mid + 1;
        else hi = mid;
      }
      mx = max(mx, lo);
    }
    run[q] = mx;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = mx;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl = max(incl, v);
  }
  int excl = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) excl = 0;
  __shared__ int w[8];
  if (lane == 31) w[wid] = incl;
  __syncthreads();
  for (int i = 0; i < wid; ++i) excl = max(excl, w[i]);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (i0 + q < la) c[L.base[part] + a + i0 + q] = max(excl, run[q]);
  if (threadIdx.x == 255) bm[(size_t)(part * L.pairs + pair) * (L.blocks + 1) + blk] = max(excl, mx);
}

// Per pair: bm becomes the maximum before each block; entry `blocks` the run's.
__global__ void __launch_bounds__(256) order_scan_kernel(Level L, int* __restrict__ bm) {
  int* p = bm + (size_t)(blockIdx.y * L.pairs + blockIdx.x) * (L.blocks + 1);
  __shared__ int w[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int carry = 0;
  for (int k0 = 0; k0 < L.blocks; k0 += 256) {
    const int k = k0 + threadIdx.x;
    int incl = k < L.blocks ? p[k] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl = max(incl, v);
    }
    int excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 0;
    __syncthreads();
    if (lane == 31) w[wid] = incl;
    __syncthreads();
    for (int i = 0; i < wid; ++i) excl = max(excl, w[i]);
    excl = max(excl, carry);
    if (k < L.blocks) p[k] = excl;
    for (int i = 0; i < 8; ++i) carry = max(carry, w[i]);
  }
  if (threadIdx.x == 0) p[L.blocks] = carry;
}

// Every element to its place in the merged run; the last merge writes each
// pixel's rank instead.
__global__ void __launch_bounds__(256) order_scatter_kernel(Level L, const float* __restrict__ key,
                                                            const int* __restrict__ idx, const int* __restrict__ c,
                                                            const int* __restrict__ bm, float* __restrict__ key_out,
                                                            int* __restrict__ idx_out,
                                                            unsigned* __restrict__ rank) {
  const int part = blockIdx.y, pair = blockIdx.x / (2 * L.blocks), blk2 = blockIdx.x % (2 * L.blocks);
  int a, la, lb;
  pair_runs(L, part, pair, a, la, lb);
  const bool in_a = blk2 < L.blocks;
  const int blk = in_a ? blk2 : blk2 - L.blocks;
  const int* p = bm + (size_t)(part * L.pairs + pair) * (L.blocks + 1);
  const int* cr = c + L.base[part] + a;
  for (int q = 0; q < 4; ++q) {
    const int e = blk * kRun + q * 256 + (int)threadIdx.x;
    if (e >= (in_a ? la : lb)) break;
    int dst;
    if (in_a) {
      dst = a + e + max(p[blk], cr[e]);
    } else {
      // the first A[i] with c_i > e: its block, then its place in it
      const int nb = (la + kRun - 1) / kRun;
      int lo = 0, hi = nb;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (p[mid + 1] > e) hi = mid;
        else lo = mid + 1;
      }
      int i = la;
      if (lo < nb) {
        int u = lo * kRun, v = min(la, u + kRun);
        while (u < v) {
          const int mid = (u + v) >> 1;
          if (cr[mid] > e) v = mid;
          else u = mid + 1;
        }
        i = u;
      }
      dst = a + e + i;
    }
    const int from = place(L, part, in_a ? a + e : a + la + e), to = place(L, part, dst);
    if (rank) {
      rank[idx[from]] = (unsigned)to;
    } else {
      key_out[to] = key[from];
      idx_out[to] = idx[from];
    }
  }
}

}  // namespace

namespace rmn {

cudaError_t launch_stable_order(const float* depth, int n, unsigned* rank, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (n == 1) return cudaMemsetAsync(rank, 0, sizeof(unsigned), st);
  const int len1 = (n + 1) / 2, len2 = n / 2;
  const int tiles1 = (len1 + kTile - 1) / kTile, tiles2 = (len2 + kTile - 1) / kTile;
  // the levels after the tiles: runs of S while some half is longer than S
  Level levels[32];
  int nl = 0;
  for (long long S = kTile; S < len1; S *= 2) {
    const int pairs = (int)((len1 + 2 * S - 1) / (2 * S));
    levels[nl++] = Level{{0, len1}, {len1, len2}, (int)S, 0, pairs, (int)((S + kRun - 1) / kRun)};
  }
  const int parts_last = 1, last = nl++;
  if (len1 == len2) levels[last] = Level{{0, 0}, {n, 0}, len1, 0, 1, (len1 + kRun - 1) / kRun};
  else levels[last] = Level{{0, 0}, {n, 0}, len2, 1, 1, (len1 + kRun - 1) / kRun};
  size_t fn_total = 0, bm_most = 0;
  for (int l = 0; l < nl; ++l) {
    const size_t runs = (size_t)(l == last ? parts_last : 2) * levels[l].pairs;
    fn_total += runs;
    bm_most = std::max(bm_most, runs * (levels[l].blocks + 1));
  }
  // keys and indices (twice), c, first NaNs of every level, block maxima
  const size_t words = 5 * (size_t)n + fn_total + bm_most;
  int* w = nullptr;
  cudaError_t e = staging_malloc(reinterpret_cast<void**>(&w), words * sizeof(int), st);
  if (e != cudaSuccess) return e;
  float* key[2] = {reinterpret_cast<float*>(w), reinterpret_cast<float*>(w + n)};
  int* idx[2] = {w + 2 * (size_t)n, w + 3 * (size_t)n};
  int *c = w + 4 * (size_t)n, *fn = w + 5 * (size_t)n, *bm = fn + fn_total;
  e = cudaMemsetAsync(fn, 0x7f, fn_total * sizeof(int), st);
  if (e == cudaSuccess) {
    order_tiles_kernel<<<tiles1 + tiles2, kTileThreads, 0, st>>>(depth, len1, n, tiles1, key[0], idx[0]);
    int cur = 0;
    for (int l = 0; l < nl; ++l) {
      const Level& L = levels[l];
      const dim3 runs(L.pairs * L.blocks, l == last ? parts_last : 2);
      order_nan_kernel<<<runs, 256, 0, st>>>(L, key[cur], fn);
      order_bound_kernel<<<runs, 256, 0, st>>>(L, key[cur], fn, c, bm);
      order_scan_kernel<<<dim3(L.pairs, runs.y), 256, 0, st>>>(L, bm);
      order_scatter_kernel<<<dim3(2 * L.pairs * L.blocks, runs.y), 256, 0, st>>>(
          L, key[cur], idx[cur], c, bm, key[cur ^ 1], idx[cur ^ 1], l == last ? rank : nullptr);
      fn += (size_t)runs.y * L.pairs;
      cur ^= 1;
    }
    e = cudaGetLastError();
  }
  const cudaError_t f = cudaFreeAsync(w, st);
  return e != cudaSuccess ? e : f;
}

}  // namespace rmn
