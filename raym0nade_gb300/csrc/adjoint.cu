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
// (seed, pixel, slot), so a lane replays exactly the forward's path of its slot
// -- same hits, same branches -- without anything stored per path.
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

// Gradient accumulation: a block-wide table in shared memory, added to the
// double-precision global table every kFlushRounds rounds and when the block ends.
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

// The replay: two 256-thread blocks per SM. A lane replays one slot at a time
// -- a first-vertex light sample or an indirect path -- and takes the next when
// it is done (slot-major, paths first, from one counter, once kRefill lanes of
// the warp are free), so no warp waits for its longest path. A round takes every
// path over one vertex and every light sample, of a first vertex or of one where
// a path ends, over one shadow ray: bounces, light samples, closest hits, shadow
// rays, the shading of the hits, the samples' gradients, finished paths. Lanes
// at different depths thus share every call, and a warp's rays are traced
// together (coop_nodes / coop_leaves, occ_nodes / occ_leaves).
//
// A block's warps go through these phases together: the code of a round is far
// larger than an SM's instruction caches, and warps in different phases each wait
// for their own instructions (with every warp going its own way 20 of the 25
// cycles between two issues, and 6.9 ms for the paths alone; 2.9 in step).
// 128 registers a thread. 256x256, 32 spp, 16 materials: one block of 512 threads
// 3.20 ms, two of 256 3.02, four of 128 3.44; one thread per slot, without refill or
// cooperation, 6.40. 64x64, 8 spp: 0.61, 0.55, 0.57 and 0.58.
constexpr int kPathThreads = 256;
constexpr int kPathBlocks = 2;  // per SM
constexpr int kRefill = 4;
// From this many lanes a warp on the phases are in step; with fewer the warps'
// instructions fit side by side and a barrier only makes the short wait for the
// long (24x24, 4 spp: 202 us without barriers, 230 with).
constexpr int kInStep = 4;
// Slots a lane takes one after the other before a warp uses more lanes: most
// slots end long before the longest, so a lane that refills fills the time its
// warp runs anyway, and fewer lanes diverge less. 64x64, 16 spp: 622, 584 and 594 us
// with 1, 3 and 4 (6: 684); 96x96, 16 spp: 628, 603 and 635; 256x256, 32 spp the same.
constexpr int kTurns = 3;
// Rounds after which a block adds its table, in 32 bits, to the double-precision
// sums: a part then holds some 170 slots however large the render (with fewer than
// kInStep lanes a warp a block has some two dozen slots in all, and its table is added
// once, at the end). At 512x512, 256 spp, 220,000 slots a block, one part a block put
// the gradient up to 4.3e-6 of it from the sum of its bands'; parts of 1, 2, 4 and 8
// rounds leave the rounding of the result alone (5e-8). 256x256, 32 spp, 16
// materials: 2986 us with one part, 2978, 2989, 2989 and 3002; 2048 materials 3064,
// 3109, 3092, 3084 and 3069.
constexpr int kFlushRounds = 2;
enum AdjMode { AM_IDLE = 0, AM_BOUNCE, AM_SAMPLE, AM_FIRST };

// total: all slots of all pixels; use: lanes of a warp that take slots, fewer
// than 32 where there are not enough slots for every lane of the device.
__global__ void __launch_bounds__(kPathThreads, kPathBlocks)
    adjoint_kernel(AdjJob J, long long total, int use, int nmats, double* gout, unsigned long long* next,
                   int* status) {
  extern __shared__ __align__(16) unsigned char adj_shared[];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  AdjTrav& sh = reinterpret_cast<AdjTrav*>(adj_shared)[threadIdx.x >> 5];
  // the block's gradient table, where it fits
  float* sg = reinterpret_cast<float*>(adj_shared + sizeof(AdjTrav) * (kPathThreads / 32));
  const bool use_sh = nmats <= kSharedMats;
  if (use_sh)
    for (int i = threadIdx.x; i < nmats * kGradPerMat; i += kPathThreads) sg[i] = 0.0f;
  __syncthreads();
  GradSink G{sg, gout, use_sh};
  auto flush = [&] {
    for (int i = threadIdx.x; i < nmats * kGradPerMat; i += kPathThreads)
      if (sg[i] != 0.0f) {
        atomicAdd(gout + i, (double)sg[i]);
        sg[i] = 0.0f;
      }
  };
  int rounds = 0;
  const Params& p = J.p;
  const DevScene& s = J.s;
  const long long npx = (long long)p.W * p.H;
  const bool in_step = use >= kInStep;
  bool more = true;  // slots may be left (the same in every lane of the warp)
  int mode = AM_IDLE;
  // the lane's slot; of a path, rec[0] is its first vertex, rec[i] its i-th bounce
  int pixel = 0, j = 0, m0 = 0, depth = 0, rfm = 0, nrec = 0;
  RmnRng rng;
  Surf sf;  // the vertex the slot stands at
  float3 V, thr, w0;
  float paw = 1.0f, rf = 0.0f, p_rr = 1.0f;
  bool nee = false, exclude = true;
  int n = 0, cnt = 0;  // light samples taken and to take at the vertex
  float kf = 1.0f, tot = 0.0f, lwt[8];
  PathAdj acc;
  Record rec[kMaxRecords + 1];
  for (;;) {
    const unsigned idle = __ballot_sync(FULL, mode == AM_IDLE && lane < use);
    if (more && __popc(idle) >= min(kRefill, use)) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(next, (unsigned long long)__popc(idle));
      base = __shfl_sync(FULL, base, 0);
      more = (long long)base + __popc(idle) < total;
      const long long t = (long long)base + __popc(idle & ((1u << lane) - 1u));
      if (((idle >> lane) & 1u) && t < total) {
        pixel = (int)(t % npx);
        j = p.slots - 1 - (int)(t / npx);
        const float* gb = gbuf_at(J, pixel);
        if (any_finite3(f3(gb[6], gb[7], gb[8]))) {  // else a miss: sky only, no material
          sf = first_vertex(J, gb);
          m0 = sf.id;
          if (j == 0) G.add(m0, 4, p.exposure * dot3(dimg_at(J, pixel), sf.emis));  // Photo::shade's emission * exposure
          if (!(len3(sf.emis) > 0.0f)) {
            V = -norm3(sf.pos - p.pos);
            rng = rmn_rng(p.seed, (uint32_t)pixel, (uint32_t)j);
            if (j < p.spp_d) {
              mode = AM_FIRST;
              n = 0;
              cnt = 1;
            } else if (rng.next() < 1.0f) {
              mode = AM_BOUNCE;
              rf = sf.roughness;
              rfm = m0;
              sf.eta = 1.0f / sf.eta;
              depth = 0;
              nrec = 0;
              thr = f3(1.0f);
              acc.S = 0.0f;
              acc.A_light = acc.A_w0 = acc.dbase = f3(0.0f);
            }
          }
        }
      }
    }
    if (in_step ? !__syncthreads_or(mode != AM_IDLE || more) : !__any_sync(FULL, mode != AM_IDLE || more)) break;
    // here every add of the rounds before is done, and the next follows a barrier
    if (in_step && use_sh && ++rounds % kFlushRounds == 0) flush();
    // the bounce from the vertex
    float3 o = f3(0.0f), dir = f3(0.0f);
    bool done = false;  // the path ends in this round
    if (mode == AM_BOUNCE) {
      float3 wv;
      int nf = 0;
      ReflectAD ad;
      sample_reflect(sf, V, rng, dir, wv, nf, &ad);
      if (!any_finite3(dir) || (depth > 0 && depth == p.maxd)) {
        mode = AM_IDLE;  // nothing was added yet: a path's samples come at its end
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
          if (nee) wv = wv / p_rr;
          thr = thr * wv;
          if (nf > 0) paw = paw * (1.0f / (float)(1 + nf));
        }
        exclude = depth == 0 || nee;
        o = sf.pos;
        depth++;
      }
    }
    if (in_step) __syncthreads();
    // the vertex's next light sample
    const bool sampled = mode == AM_SAMPLE || mode == AM_FIRST;
    bool go = false;  // it needs a shadow ray
    float3 ld = f3(0.0f);
    float aim = 0.0f;
    LSample ls;
    int li = -1;
    if (sampled) {
      if (n == 0 && s.sky_w == 0 && !light_weights(s, sf, V, lwt, tot)) cnt = 0;
      if (cnt > 0)
        go = light_gen(s, sf, V, lwt, tot, mode == AM_FIRST ? p.spp_d : cnt, rng, ld, aim, ls, &li);
    }
    if (in_step) __syncthreads();
    float tm;
    const int h = closest(s, o, dir, tm, mode == AM_BOUNCE, sh);
    if (in_step) __syncthreads();
    const bool occ = occluded(s, sf.pos, ld, aim, go, sh, status);
    if (in_step) __syncthreads();
    const int drop = J.dropped && mode != AM_IDLE ? J.dropped[pixel] : -1;
    // a sample's contribution and the path's sums
    const float* gb = gbuf_at(J, pixel);
    auto demod = [&](float3 f, float3 light, float w) {
      DemodAdj d = demod_adj(tweak_base(f3(__ldg(&s.mats[m0].base))), f3(gb[0], gb[1], gb[2]), f, light, w,
                             dimg_at(J, pixel), p.exposure);
      if (!finite1(d.S) || d.S == 0.0f) {
        d.S = 0.0f;
        d.dlight = f3(0.0f);
      }
      return d;
    };
    auto add_path = [&](const DemodAdj& d, float3 light) {
      if (d.S == 0.0f) return;
      acc.S += d.S;
      acc.A_light += d.dlight * light;
      acc.A_w0 += d.df * w0;
      acc.dbase += d.dbase;
    };
    if (mode == AM_BOUNCE) {
      if (h == -2) {
        atomicExch(status, 1);
        mode = AM_IDLE;
      } else if (h < 0) {
        if (!exclude && s.sky_w && drop != j * 8) {
          const float3 light = sky_get(s, dir) * thr;
          add_path(demod(w0, light, paw * p.inv_spp), light);
        }
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
            const float3 light = sf.emis * thr;
            const DemodAdj d = demod(w0, light, paw * p.inv_spp);
            add_path(d, light);
            G.add(sf.id, 4, d.S);
          }
          done = true;
        } else if (!(rng.next() <= 1.0f)) {
          done = true;
        } else {
          nee = nee && sf.entering;
          if (nee && (depth >= p.maxd || rng.next() > p_rr)) {
            mode = AM_SAMPLE;
            n = 0;
            cnt = c_sample_count[depth < 16 ? depth : 16];
            kf = 1.0f;
            if (depth < p.maxd) kf /= (1.0f - p_rr);
          }
        }
      }
    }
    if (in_step) __syncthreads();
    if (sampled) {
      const bool first = mode == AM_FIRST;
      if (go && !occ && (first || drop != j * 8 + n)) {
        if (!first) ls.bsdf *= kf;
        const float3 light = first ? ls.light : (ls.light * ls.bsdf) * thr;
        const DemodAdj d = demod(first ? ls.bsdf : w0, light, first ? ls.weight : ls.weight * paw * p.inv_spp);
        if (d.S != 0.0f) {
          if (!first) add_path(d, light);
          float3 l, q, lr;
          brdf_logd(sf, V, ld, 2, l, q, lr);
          const float3 A = first ? d.df * ls.bsdf : d.dlight * light;
          float3 gbase = A * l - d.S * q;
          if (first) gbase += d.dbase;
          G.add_base(sf.id, gbase);
          G.add(first ? sf.id : rfm, 3, dot3(A, lr));
          if (li >= 0) G.add(__ldg(&s.lights[li].material), 4, d.S);
        }
      }
      if (++n >= cnt) {
        done = !first;
        mode = AM_IDLE;
      }
    }
    if (done) {
      mode = AM_IDLE;
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
  __syncthreads();
  if (use_sh) flush();
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
  const long long total = (long long)J.p.W * J.p.H * J.p.slots;
  const size_t fixed = sizeof(AdjTrav) * (kPathThreads / 32);
  const size_t shared = fixed + (nmats <= kSharedMats ? (size_t)ng * sizeof(float) : 0);
  // the limit belongs to the kernel, not to the call: every call sets the same, so
  // none lowers it between another thread's call and its launch
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(fixed + sizeof(float) * kSharedMats * kGradPerMat));
  if (e == cudaSuccess && total > 0) {
    // the slots over all warps first (kInStep lanes), then over their lanes, kTurns to
    // a lane before it takes more lanes
    const long long blocks = (long long)kPathBlocks * device_sms(), warps = blocks * (kPathThreads / 32);
    const long long each = (total + warps - 1) / warps;
    const int use = (int)std::min<long long>(
        32, std::max(std::min<long long>(each, kInStep), (each + kTurns - 1) / kTurns));
    const long long per_block = (long long)use * (kPathThreads / 32);
    const unsigned grid = (unsigned)std::min<long long>(blocks, (total + per_block - 1) / per_block);
    adjoint_kernel<<<grid, kPathThreads, shared, st>>>(J, total, use, nmats, acc, next, status);
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
