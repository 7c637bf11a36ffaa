// Adjoint of the integrator (rmn_adjoint): the gradient of an image loss
// with respect to every material's base colour, roughness and emission
// scale, by path replay. The reference has no counterpart; what is
// differentiated is its estimator, renderPixel (src/render.cpp:448-551) with
// sampleRay (:121-312), composed by Photo::shade(Full) (src/image.cpp:
// 215-246) into I = base (*) (Dd + Id) + Ds + Is + emission * exposure.
//
// Input: the G-buffer and the per-pixel dropped-sample record of a forward
// rmn_render with the same scene and arguments, and dL/dI (3 floats per
// pixel). Every sample slot draws from the counter-based stream keyed
// (seed, pixel, slot), so one thread per slot replays exactly the forward's
// path -- same hits, same branches -- without anything stored per path.
//
// Per sample s of a path (a light sample at the terminating vertex, or the
// emitter or sky the path hits) the contribution S_s = dL/dI . dI_s is
// bilinear in the first-vertex factor w0 and in the sample's light (the
// product of the emitted radiance and every later path factor), so each
// multiplicative factor v of the path adds (A (*) dlog v) with A = dS/dv (*)
// v and sum(A) = S. The replay records, per bounce vertex, the factor's
// log-derivatives (factor_logd) and at the end applies the path's summed
// A to all of them; the first-vertex factor and the demodulation against the
// base colour (demod_adj) are differentiated directly.
//
// Sampling that depends on a parameter is handled by the score function
// (detached sampling): for the roughness, the GGX half vectors drawn and the
// choice between the cosine and the GGX candidate (sample_reflect's
// ReflectAD). Russian roulette and light selection divide by the
// probability of the decision they draw, so their score cancels their
// derivative and neither appears. The base colour and emission change no
// sampling probability except the light selection weights (cancelled the
// same way). Decisions taken by thresholds on the parameters (the
// luminance-clamp boundary, the firefly clamp of :532-547, the NEE switch at
// P_RR < 0.9) are held as the forward took them: the forward's record of
// the sample the firefly clamp dropped is skipped.
#include <algorithm>
#include <vector>

#include "integrator.cuh"

namespace {

constexpr int kGradPerMat = 5;   // base colour r, g, b; roughness; emission scale
constexpr int kSharedMats = 2048;  // per-block gradient table in shared memory up to this many materials
constexpr int kMaxRecords = 16;  // bounce vertices of one path (max depth 16)

struct AdjJob {
  DevScene s;
  Params p;
  const float* gbuf;
  const int* dropped;
  const float* dimg;  // dL/dI, 3 per pixel
};

// Gradient accumulation: a block-wide table in shared memory, flushed to the
// double-precision global table when the block ends.
struct GradSink {
  float* sh;
  double* gl;
  bool use_sh;
  __device__ __forceinline__ void add(int m, int k, float v) {
    if (v == 0.0f || !finite1(v)) return;
    if (use_sh) atomicAdd(sh + m * kGradPerMat + k, v);
    else atomicAdd(gl + m * kGradPerMat + k, (double)v);
  }
  __device__ __forceinline__ void add_base(int m, float3 v) {
    add(m, 0, v.x);
    add(m, 1, v.y);
    add(m, 2, v.z);
  }
};

// S = dL/dI . (contribution of one sample to I) and its derivatives, for
// accumulateInwardRadiance (src/image.cpp:627-659) against the tweaked base
// colour bt, composed with the G-buffer's base colour sav, times calcVar's
// exposure E. f = the sample's bsdfPdf (the first-vertex factor), light =
// its light, w = its weight, g = dL/dI of the pixel. dbase is the
// derivative through bt and sav together (both move with the material's
// base colour; the tweak only shifts it).
struct DemodAdj {
  float S;
  float3 df, dlight, dbase;
};
__device__ __noinline__ DemodAdj demod_adj(float3 bt, float3 sav, float3 f, float3 light, float w, float3 g,
                                           float E) {
  DemodAdj r;
  r.S = 0.0f;
  r.df = r.dlight = r.dbase = f3(0.0f);
  if (len3(light) < RMN_EPS || !finite1(w)) return r;
  const float Ew = E * w;
  const float n = len3(bt);
  const float3 gl = g * light;
  if (n < RMN_EPS) {  // all specular
    if (!all_finite3(light * f)) return r;
    r.S = Ew * dot3(gl, f);
    r.df = Ew * gl;
    r.dlight = Ew * (g * f);
    return r;
  }
  const float3 b0 = norm3(bt);
  const float3 white = norm3(f3(1.0f));
  const float xy = dot3(b0, white);
  if (xy > 0.99f) {  // all diffuse: d = light f / bt
    float3 d = light * f / bt;
    if (!all_finite3(d)) return r;
    r.S = Ew * dot3(g * sav, d);
    r.df = Ew * (g * sav * light / bt);
    r.dlight = Ew * (g * sav * f / bt);
    r.dbase = Ew * (g * light * f / bt - g * sav * d / bt);
    return r;
  }
  // B = beta . f with beta = ((white + b0) / (1 + xy) - (white - b0) / (1 - xy)) / 2
  const float a = dot3(white, f), c = dot3(b0, f);
  const float ip = 1.0f / (1.0f + xy), im = 1.0f / (1.0f - xy);
  const float B = 0.5f * ((a + c) * ip - (a - c) * im);
  const float3 dpart = light * B / n, spart = light * (f - B * b0);
  const bool dok = all_finite3(dpart), sok = all_finite3(spart);
  const float Q = dot3(g * sav, light);
  const float kappa = (dok ? Q / n : 0.0f) - (sok ? dot3(gl, b0) : 0.0f);
  const float3 beta = 0.5f * ((white + b0) * ip - (white - b0) * im);
  r.S = Ew * ((dok ? B * Q / n : 0.0f) + (sok ? dot3(gl, f) - B * dot3(gl, b0) : 0.0f));
  r.df = Ew * (kappa * beta + (sok ? gl : f3(0.0f)));
  r.dlight = Ew * ((dok ? (B / n) * (g * sav) : f3(0.0f)) + (sok ? g * f - B * (g * b0) : f3(0.0f)));
  // through b0 (B and the projection), |bt| and sav
  const float dB_dc = 0.5f * (ip + im);
  const float dB_dxy = 0.5f * (-(a + c) * ip * ip - (a - c) * im * im);
  const float3 dB_db0 = dB_dc * f + dB_dxy * white;
  const float3 dS_db0 = Ew * (kappa * dB_db0 - (sok ? B * gl : f3(0.0f)));
  const float dS_dn = dok ? -Ew * B * Q / (n * n) : 0.0f;
  const float3 dS_dbt = (dS_db0 - b0 * dot3(b0, dS_db0)) / n + b0 * dS_dn;
  const float3 dS_dsav = dok ? Ew * (B / n) * gl : f3(0.0f);
  r.dbase = dS_dbt + dS_dsav;
  return r;
}

// Sums over the samples of one path.
struct PathAdj {
  float S;
  float3 A_light, A_w0, dbase;
};

// One warp's share of the traversals' shared memory: the ordered search's
// stack and leaf keys, or occlusion's stack of references and leaf exchange.
union AdjTrav {
  struct {
    int2 stack[RMN_STACK * 32];
    unsigned long long keys[32];
  } closest;
  struct {
    int stack[RMN_STACK * 32];
    OccExchangeT<32> x;
  } occ;
};

// The warp's shadow rays (all 32 lanes; `go`: the lane has one): whether each
// is occluded, as Model::rayHit_test (no alpha-tested scenes here). A real
// call, as are brdf_logd and demod_adj: inlined at each of their call sites
// they multiplied the replay's code, and its warps stalled on instruction
// fetch.
__device__ __noinline__ bool occluded(const DevScene& s, float3 pos, float3 dir, float aim, bool go, AdjTrav& sh,
                                      int* status) {
  OccT<SharedStackRefN<RMN_STACK, 32>> t;
  t.stack.base = sh.occ.stack + (threadIdx.x & 31);
  occ_begin(s.root, t);
  TRay r;
  if (go) r = make_tray(pos, dir);
  bool active = go, answer = false;
  while (__ballot_sync(0xffffffffu, active) != 0) {
    const int st = occ_nodes<false>(s.nodes, r, RMN_EPS, aim + RMN_EPS, t, active, kOccSteps, nullptr);
    const bool o = occ_leaves<true>(s.tri, r, RMN_EPS, aim, t, sh.occ.x);
    if (!active || (st == 0 && !o)) continue;
    if (st == -2) atomicExch(status, 1);
    answer = o && st != -2;
    active = false;
  }
  return answer;
}

// The warp's closest-hit rays likewise: the leaf-order triangle or -1 (-2 on
// stack overflow), and its distance in tmax.
__device__ __noinline__ int closest(const DevScene& s, float3 pos, float3 dir, float& tmax, bool go, AdjTrav& sh) {
  TravT<SharedStackN<RMN_STACK, 32>> t;
  t.stack.base = sh.closest.stack + (threadIdx.x & 31);
  trav_begin(s, t, INFINITY);
  TRay r;
  if (go) r = make_tray(pos, dir);
  bool active = go;
  int hit = -1;
  while (__ballot_sync(0xffffffffu, active) != 0) {
    int st = coop_nodes<false>(s.nodes, r, RMN_EPS, t, active, kCoopSteps, nullptr);
    coop_leaves<false, true>(s.tri, r, RMN_EPS, 0.0f, t, true, sh.closest.keys);
    if (!active || st == 0) continue;
    hit = st == -2 ? -2 : t.hit;
    active = false;
  }
  tmax = t.tmax;
  return hit;
}

// Log-derivatives of a factor clamp64(brdf(V, L)) * k of surface sf.
__device__ __noinline__ void brdf_logd(const Surf& sf, float3 V, float3 L, int clamp_mode, float3& l, float3& q,
                                          float3& lr) {
  float3 db, dr;
  float3 f = brdf_d(sf, V, L, db, dr);
  bool clamped = clamp_mode == 2 ? dot3(f, RMN_LUM) > 64.0f : clamp_mode == 1;
  factor_logd(f, db, dr, clamped, l, q, lr);
}

struct Record {
  int m, a;  // material of the vertex; material whose roughness the vertex used
  float3 l, q, lr;
};

// The first vertex of a pixel as the forward shades it: the material's base
// colour with renderPixel's tweak (the G-buffer's copy is the composed one).
__device__ __forceinline__ Surf first_vertex(const AdjJob& J, const float* gb) {
  Surf g = default_surf();
  g.id = (int)gb[19];
  g.base = tweak_base(f3(__ldg(&J.s.mats[g.id].base)));
  g.emis = f3(gb[3], gb[4], gb[5]);
  g.pos = f3(gb[6], gb[7], gb[8]);
  g.shapeN = f3(gb[9], gb[10], gb[11]);
  g.surfN = f3(gb[12], gb[13], gb[14]);
  g.roughness = gb[15];
  g.metallic = gb[16];
  g.opacity = gb[17];
  g.eta = gb[18];
  return g;
}
__device__ __forceinline__ const float* gbuf_at(const AdjJob& J, int pixel) {
  return J.gbuf + (size_t)RMN_GBUFFER_FLOATS * pixel;
}
__device__ __forceinline__ float3 dimg_at(const AdjJob& J, int pixel) {
  return f3(J.dimg[3 * (size_t)pixel], J.dimg[3 * (size_t)pixel + 1], J.dimg[3 * (size_t)pixel + 2]);
}

// Both kernels: dynamic shared memory holds the block's gradient table (when
// it fits), flushed to the double-precision sums at the end.
__device__ __forceinline__ GradSink grad_begin(float* sg, double* gout, int nmats) {
  const bool use_sh = nmats <= kSharedMats;
  if (use_sh)
    for (int i = threadIdx.x; i < nmats * kGradPerMat; i += blockDim.x) sg[i] = 0.0f;
  __syncthreads();
  return GradSink{sg, gout, use_sh};
}
__device__ __forceinline__ void grad_end(const GradSink& G, int nmats) {
  __syncthreads();
  if (!G.use_sh) return;
  for (int i = threadIdx.x; i < nmats * kGradPerMat; i += blockDim.x)
    if (G.sh[i] != 0.0f) atomicAdd(G.gl + i, (double)G.sh[i]);
}

// Both kernels run in one block per SM whose warps go through the phases of a
// round together (barriers between them): the code of a round is far larger
// than an SM's instruction caches, so warps in different phases each wait for
// their own instructions (20 cycles of 25 a warp waited between two issues
// while every warp went its own way: 6.9 ms a pass over the paths below;
// 2.9 ms with the phases in step).
constexpr int kPathThreads = 512;

// The light-sample slots of the first vertices, slot-major: a warp replays one
// slot of 32 neighbouring pixels.
__global__ void __launch_bounds__(kPathThreads, 1)
    adjoint_light_kernel(AdjJob J, long long total, int nmats, double* gout, int* status) {
  extern __shared__ __align__(16) unsigned char path_shared[];
  AdjTrav& sh = reinterpret_cast<AdjTrav*>(path_shared)[threadIdx.x >> 5];
  GradSink G = grad_begin(reinterpret_cast<float*>(path_shared + sizeof(AdjTrav) * (kPathThreads / 32)), gout, nmats);
  const Params& p = J.p;
  const DevScene& s = J.s;
  const long long npx = (long long)p.W * p.H;
  for (long long t0 = (long long)blockIdx.x * kPathThreads; t0 < total; t0 += (long long)gridDim.x * kPathThreads) {
    const long long t = t0 + threadIdx.x;
    const int pixel = (int)(t % npx), j = (int)(t / npx);
    const float* gb = gbuf_at(J, pixel);
    bool go = t < total && any_finite3(f3(gb[6], gb[7], gb[8]));  // else a miss: sky only, no material
    Surf g;
    float3 Vd, dir;
    float aim = 0.0f;
    LSample ls;
    int li = -1;
    if (go) {
      g = first_vertex(J, gb);
      if (j == 0) G.add(g.id, 4, p.exposure * dot3(dimg_at(J, pixel), g.emis));  // Photo::shade's emission * exposure
      go = !(len3(g.emis) > 0.0f);
    }
    if (go) {
      RmnRng rng = rmn_rng(p.seed, (uint32_t)pixel, (uint32_t)j);
      Vd = -norm3(g.pos - p.pos);
      float lwt[8];
      float tot = 0.0f;
      go = (s.sky_w != 0 || light_weights(s, g, Vd, lwt, tot)) &&
           light_gen(s, g, Vd, lwt, tot, p.spp_d, rng, dir, aim, ls, &li);
    }
    __syncthreads();
    const bool occ = occluded(s, g.pos, dir, aim, go, sh, status);
    __syncthreads();
    if (occ || !go) continue;
    DemodAdj d = demod_adj(g.base, f3(gb[0], gb[1], gb[2]), ls.bsdf, ls.light, ls.weight, dimg_at(J, pixel),
                           p.exposure);
    if (!finite1(d.S) || d.S == 0.0f) continue;
    float3 l, q, lr;
    brdf_logd(g, Vd, dir, 2, l, q, lr);
    const float3 A = d.df * ls.bsdf;
    G.add_base(g.id, A * l - d.S * q + d.dbase);
    G.add(g.id, 3, dot3(A, lr));
    if (li >= 0) G.add(__ldg(&s.lights[li].material), 4, d.S);
  }
  grad_end(G, nmats);
}

// The indirect paths. A lane replays one path at a time and takes the next
// slot when it is done (slot-major, from one counter, once kRefill lanes of
// the warp are free), so a warp does not wait for its longest path; each round
// takes every lane's path over one vertex -- the bounce from the vertex it
// stands at, first or later, the closest hit, its shading, and where the path
// ends there its light samples -- so that lanes at different depths share every
// call. The rays of a warp are traced together (coop_nodes / coop_leaves,
// occ_nodes / occ_leaves).
//
// 512 threads of 128 registers: 256, 384, 768 and 1024 threads took 4.85, 4.13,
// 4.01 and 4.48 ms a call where 512 took 3.88 (256x256, 32 spp, 16 materials;
// the replay of one path per thread, without refill or cooperation, 6.40).
constexpr int kRefill = 8;

__global__ void __launch_bounds__(kPathThreads, 1)
    adjoint_path_kernel(AdjJob J, long long total, int nmats, double* gout, unsigned long long* next, int* status) {
  extern __shared__ __align__(16) unsigned char path_shared[];
  const unsigned FULL = 0xffffffffu;
  AdjTrav& sh = reinterpret_cast<AdjTrav*>(path_shared)[threadIdx.x >> 5];
  float* sg = reinterpret_cast<float*>(path_shared + sizeof(AdjTrav) * (kPathThreads / 32));
  const int lane = threadIdx.x & 31;
  GradSink G = grad_begin(sg, gout, nmats);
  const Params& p = J.p;
  const DevScene& s = J.s;
  const long long npx = (long long)p.W * p.H;
  bool active = false, more = true;  // more: slots may be left (the same in every lane)
  // the lane's path: rec[0] is its first vertex, rec[i] its i-th bounce
  int pixel = 0, j = 0, depth = 0, rfm = 0, nrec = 0;
  RmnRng rng;
  Surf sf;  // the vertex the path stands at
  float3 V, thr, w0;
  float paw = 1.0f, rf = 0.0f, p_rr = 1.0f;
  bool nee = false, exclude = true;
  PathAdj acc;
  Record rec[kMaxRecords + 1];
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, !active);
    if (more && (__popc(idle) >= kRefill)) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(next, (unsigned long long)__popc(idle));
      base = __shfl_sync(FULL, base, 0);
      more = (long long)base + __popc(idle) < total;
      const long long t = (long long)base + __popc(idle & ((1u << lane) - 1u));
      if (!active && t < total) {
        pixel = (int)(t % npx);
        j = p.spp_d + (int)(t / npx);
        const float* gb = gbuf_at(J, pixel);
        if (any_finite3(f3(gb[6], gb[7], gb[8]))) {  // else a miss: sky only, no material
          sf = first_vertex(J, gb);
          if (j == 0)  // Photo::shade's emission * exposure
            G.add(sf.id, 4, p.exposure * dot3(dimg_at(J, pixel), sf.emis));
          rng = rmn_rng(p.seed, (uint32_t)pixel, (uint32_t)j);
          active = !(len3(sf.emis) > 0.0f) && rng.next() < 1.0f;
          V = -norm3(sf.pos - p.pos);
          rf = sf.roughness;
          rfm = sf.id;
          sf.eta = 1.0f / sf.eta;
          depth = 0;
          nrec = 0;
          paw = 1.0f;
          thr = f3(1.0f);
          acc.S = 0.0f;
          acc.A_light = acc.A_w0 = acc.dbase = f3(0.0f);
        }
      }
    }
    if (!__syncthreads_or(active || more)) break;
    // the bounce from the vertex
    float3 o = f3(0.0f), dir = f3(0.0f);
    bool done = false;  // the path ends in this round
    if (active) {
      float3 wv;
      int nf = 0;
      ReflectAD ad;
      sample_reflect(sf, V, rng, dir, wv, nf, &ad);
      if (!any_finite3(dir) || (depth > 0 && depth == p.maxd)) {
        active = false;  // nothing was added yet: a path's samples come at its end
      } else {
        Record& r = rec[nrec++];
        r.m = sf.id;
        r.a = rfm;
        brdf_logd(sf, V, dir, ad.clamped, r.l, r.q, r.lr);
        r.lr = r.lr + f3(ad.score);
        if (depth == 0) {
          w0 = wv;
          paw = nf > 0 ? 1.0f / (float)(1 + nf) : 1.0f;
        } else {
          wv = wv / 1.0f;
          if (nee) wv = wv / p_rr;
          thr = thr * wv;
          if (nf > 0) paw = paw * (1.0f / (float)(1 + nf));
        }
        exclude = depth == 0 || nee;
        o = sf.pos;
        depth++;
      }
    }
    __syncthreads();
    float tm;
    const int h = closest(s, o, dir, tm, active, sh);
    __syncthreads();
    // one sample of the path: light, weight, into the path's sums
    auto add_sample = [&](float3 light, float w) {
      const float* gb = gbuf_at(J, pixel);
      DemodAdj d = demod_adj(tweak_base(f3(__ldg(&s.mats[rec[0].m].base))), f3(gb[0], gb[1], gb[2]), w0, light, w,
                             dimg_at(J, pixel), p.exposure);
      if (!finite1(d.S) || d.S == 0.0f) {
        d.S = 0.0f;
        d.dlight = f3(0.0f);
        return d;
      }
      acc.S += d.S;
      acc.A_light += d.dlight * light;
      acc.A_w0 += d.df * w0;
      acc.dbase += d.dbase;
      return d;
    };
    int cnt = 0;  // light samples of the vertex, where the path ends there
    float kf = 1.0f;
    if (active) {
      const int drop = J.dropped ? J.dropped[pixel] : -1;
      if (h == -2) {
        atomicExch(status, 1);
        active = false;
      } else if (h < 0) {
        if (!exclude && s.sky_w && drop != j * 8) add_sample(sky_get(s, dir) * thr, paw * p.inv_spp);
        done = true;
      } else {
        sf = default_surf();
        sf.pos = o + dir * tm;
        hit_info(s, h, dir, sf);
        const float own = sf.roughness;
        const float rfn = fmaxf(rf, 1.0f * own);
        if (own >= rf) rfm = sf.id;
        sf.roughness = fmaxf(sf.roughness, rfn);
        rf = rfn;
        p_rr = 1.0f + (0.5f - 1.0f) * sqrtf(sf.roughness);
        nee = p_rr < 0.9f;
        V = -dir;
        if (len3(sf.emis) > RMN_EPS) {
          if (!exclude && drop != j * 8) {
            DemodAdj d = add_sample(sf.emis * thr, paw * p.inv_spp);
            G.add(sf.id, 4, d.S);
          }
          done = true;
        } else if (!(rng.next() <= 1.0f)) {
          done = true;
        } else {
          nee = nee && sf.entering;
          if (nee && (depth >= p.maxd || rng.next() > p_rr)) {
            cnt = c_sample_count[depth < 16 ? depth : 16];
            if (depth < p.maxd) kf /= (1.0f - p_rr);
            done = true;
          }
        }
      }
    }
    // the light samples of the vertices where paths end
    if (__syncthreads_or(cnt > 0)) {
      float lwt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      float tot = 0.0f;
      if (cnt > 0 && s.sky_w == 0 && !light_weights(s, sf, V, lwt, tot)) cnt = 0;
      for (int n = 0; __syncthreads_or(n < cnt); ++n) {
        float3 ld = f3(0.0f);
        float aim = 0.0f;
        LSample ls;
        int li = -1;
        const bool go = n < cnt && light_gen(s, sf, V, lwt, tot, cnt, rng, ld, aim, ls, &li);
        __syncthreads();
        const bool occ = occluded(s, sf.pos, ld, aim, go, sh, status);
        __syncthreads();
        if (occ || !go) continue;
        if ((J.dropped ? J.dropped[pixel] : -1) == j * 8 + n) continue;
        ls.bsdf *= kf;
        const float3 light = (ls.light * ls.bsdf) * thr;
        DemodAdj d = add_sample(light, ls.weight * paw * p.inv_spp);
        if (d.S == 0.0f) continue;
        float3 l, q, lr;
        brdf_logd(sf, V, ld, 2, l, q, lr);
        const float3 A = d.dlight * light;
        G.add_base(sf.id, A * l - d.S * q);
        G.add(rfm, 3, dot3(A, lr));
        if (li >= 0) G.add(__ldg(&s.lights[li].material), 4, d.S);
      }
    }
    if (done) {
      active = false;
      if (acc.S != 0.0f) {
        for (int i = 1; i < nrec; ++i) {
          const Record& r = rec[i];
          G.add_base(r.m, acc.A_light * r.l - acc.S * r.q);
          G.add(r.a, 3, dot3(acc.A_light, r.lr));
        }
        const Record& r = rec[0];
        G.add_base(r.m, acc.A_w0 * r.l - acc.S * r.q + acc.dbase);
        G.add(r.m, 3, dot3(acc.A_w0, r.lr));
      }
    }
  }
  grad_end(G, nmats);
}

__global__ void to_float_kernel(const double* in, float* out, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)in[i];
}

}  // namespace

namespace rmn {

rmn_status launch_adjoint(const rmn_scene* scene, const rmn_render_args& args, const float* gbuf,
                          const int* dropped, const float* dimg, float* dmat, cudaStream_t st) {
  AdjJob J;
  J.s = scene->dev;
  J.p = make_params(args);
  J.gbuf = gbuf;
  J.dropped = dropped;
  J.dimg = dimg;
  const int nmats = scene->dev.num_mats;
  const int ng = nmats * kGradPerMat;
  double* acc = nullptr;
  cudaError_t e = rmn::staging_malloc(reinterpret_cast<void**>(&acc), (size_t)ng * sizeof(double) + 16, st);
  if (e != cudaSuccess) return cuda_fail(e, "staging allocation (adjoint)");
  unsigned long long* next = reinterpret_cast<unsigned long long*>(acc + ng);
  int* status = reinterpret_cast<int*>(next + 1);
  e = cudaMemsetAsync(acc, 0, (size_t)ng * sizeof(double) + 16, st);
  const long long npx = (long long)J.p.W * J.p.H;
  const long long lights = npx * J.p.spp_d, paths = npx * (J.p.slots - J.p.spp_d);
  const size_t shared =
      sizeof(AdjTrav) * (kPathThreads / 32) + (nmats <= kSharedMats ? (size_t)ng * sizeof(float) : 0);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // as many blocks as the device holds, or as the slots need
  auto blocks = [&](const void* kernel, int threads, size_t shared, long long slots) {
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, shared);
    return (unsigned)std::min<long long>((slots + threads - 1) / threads, (long long)sms * std::max(per_sm, 1));
  };
  if (e == cudaSuccess && lights > 0) {
    const unsigned g = blocks((const void*)adjoint_light_kernel, kPathThreads, shared, lights);
    if (e == cudaSuccess) adjoint_light_kernel<<<g, kPathThreads, shared, st>>>(J, lights, nmats, acc, status);
  }
  if (e == cudaSuccess && paths > 0) {
    const unsigned g = blocks((const void*)adjoint_path_kernel, kPathThreads, shared, paths);
    if (e == cudaSuccess) adjoint_path_kernel<<<g, kPathThreads, shared, st>>>(J, paths, nmats, acc, next, status);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) {
    to_float_kernel<<<(ng + 127) / 128, 128, 0, st>>>(acc, dmat, ng);
    e = cudaGetLastError();
  }
  int h_status = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h_status, status, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(acc, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "adjoint launch");
  if (h_status) return fail(RMN_ERR_CUDA, "traversal stack overflow in the adjoint");
  return RMN_OK;
}

}  // namespace rmn
