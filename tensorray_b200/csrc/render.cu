// Integrator kernels: the interior path tracer (forward and replaying
// adjoint) and the primary / direct / indirect / pixel boundary terms.
//
// The reference builds a tensor expression per stage and compacts surviving rays
// between stages (Integrator.cpp:178-303, Ray.cpp:65-116). Here the interior
// paths and the boundary set-ups run as a wavefront of a few kernels per bounce
// (wavefront.cuh); the paths of boundary samples, the late bounces of few paths and
// the calls that may not allocate run one path per thread, which keeps its state
// in registers and simply stops. The per-slot sample layout replaces the
// reference's per-call RandomFloat tensors (see SampleSource).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <string>
#include <vector>
#include <cub/cub.cuh>
#include "../../include/trn.h"
#include "scene_impl.cuh"
#include "shading.cuh"
#include "cdf.cuh"

namespace trn {

struct Params {
  DeviceScene s;
  const ViewDesc* views;     // [nviews] cameras, slot ranges, pixel offsets
  const long long* vbegin;   // [nviews] first path slot of each view
  int nviews;
  long long total;           // path slots of this launch (all views)
  unsigned long long* work;  // work-distribution counter (zeroed before launch)
  int chunk;                 // slots per lane per work fetch
  const float* table;        // sample table [dim][total-slot] or nullptr (hash)
  long long stride;
  uint32_t term;             // integrator id (hash stream)
  uint32_t seed;             // RenderOptions::mRndSeed
  float* image;              // call image buffer (views without their own)
  const float* dLdI;         // call dL/dI buffer (views without their own)
  int D;                     // max bounces
  float* g_pos;              // [V*3]
  float* g_vn;               // [V*3]
  float* g_tex;              // [texels*3]
  int diff_tex;              // accumulate texture gradients
  // secondary edge sampling table (per scene); primary tables live in the views
  const int* edges;
  const float* ecdf;
  const float* efunc;
  const float* eint;
  int ne;
  int* err;
  unsigned long long* stats;  // optional work counters (see Cnt), nullptr = off
  // AQ guiding of the direct boundary term (nullptr = unguided)
  const float* aq_poly;       // [leaves] leaf weights
  const float* aq_cdf;        // [leaves] leaf distribution
  const float* aq_int;        // [2] integral, sum of weight x volume
  const float* aq_box;        // [6][aq_cap] leaf boxes (x0, y0, z0, x1, y1, z1)
  const int* aq_edge;         // [leaves] the secondary edge a leaf lies on
  const int* aq_n;            // leaf count
  long long aq_cap;
  // samples of a boundary term's round that passed its set-up (items), or the
  // interior term's path records, and their count
  void* queue;
  unsigned long long* q_count;
  long long q_cap;
  // run order of a split set-up round (nullptr = slot order): the i-th slot
  // of the round [order_first, total) is order_first + order[i - order_first]
  const unsigned* order;
  long long order_first;
};

// The wavefront kernels are launched with programmatic stream serialisation:
// a kernel's blocks may become resident while the last blocks of the kernel
// before it still run. Each kernel starts with this: it lets its own successor
// come in as early, and waits until its predecessor has ended and its writes
// are visible. (Nothing a wavefront kernel writes is read through the
// non-coherent path, which may serve a line from before the wait.) A stage of a
// small call takes a few us, about as long as the launch it then hides.
TRN_D void stage_begin() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// Slot that runs at position i of the current round.
TRN_D long long slot_at(const Params& P, long long i) {
  if (!P.order || i >= P.total) return i;
  return P.order_first + (long long)__ldg(P.order + (i - P.order_first));
}

constexpr int kMaxDepth = 16;

// The integrator kernels' parameter block. Its members (the scene above all)
// are passed by reference into non-inlined functions; a plain by-value
// kernel parameter whose address is taken is first copied into every
// thread's local memory, a __grid_constant__ one is addressed in place.
#ifndef TRN_GRID_CONSTANT
#define TRN_GRID_CONSTANT 1
#endif
#if TRN_GRID_CONSTANT
#define TRN_KPARAMS const __grid_constant__ Params P
#else
#define TRN_KPARAMS Params P
#endif

// Minimum resident 256-thread blocks per SM the integrator kernels are
// compiled for (caps registers per thread at 65536 / (256 * minimum)); the
// values below are the measured best per kernel family.
#ifndef TRN_MINB
#define TRN_MINB 4
#endif
#ifndef TRN_MINB_PATHADJ
#define TRN_MINB_PATHADJ 4
#endif
#ifndef TRN_MINB_REVERSE
#define TRN_MINB_REVERSE 2
#endif
// Per-thread work counters behind the roofline's algorithmic-byte model:
// ray queries, shading vertices, light samples, gradient scatters, pixels.
enum { kCntClosest = 0, kCntShadow, kCntShade, kCntSmooth, kCntTex, kCntLight, kCntVScatter, kCntNScatter,
       kCntTScatter, kCntPixel, kCntNum };
struct Cnt {
  unsigned v[kCntNum];
  TRN_D Cnt() {
#pragma unroll
    for (int i = 0; i < kCntNum; i++) v[i] = 0u;
  }
};
TRN_D void flush_cnt(const Cnt& c, unsigned long long* stats) {
  if (!stats) return;
#pragma unroll
  for (int i = 0; i < kCntNum; i++) {
    const unsigned x = __reduce_add_sync(0xffffffffu, c.v[i]);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd(stats + i, (unsigned long long)x);
  }
}
TRN_D void count_shade(Cnt& c, const DeviceScene& s, const SurfF& x) {
  c.v[kCntShade]++;
  if (s.smooth[x.tri]) c.v[kCntSmooth]++;
  if (s.bsdfs[x.bsdf].tex >= 0) c.v[kCntTex]++;
}

TRN_HD F3 F3z() { return F3(0.f, 0.f, 0.f); }
TRN_D F3 scrub(const F3& a) { return finite3(a) ? a : F3z(); }
TRN_D void atomic_add3(float* a, const F3& g) {
  if (g.x != 0.f) atomicAdd(a, g.x);
  if (g.y != 0.f) atomicAdd(a + 1, g.y);
  if (g.z != 0.f) atomicAdd(a + 2, g.z);
}

// Warp-aggregated scatter-add of a float3 into base[3*idx]: the lanes of the
// converged warp that target the same address first sum up by shuffles, in
// log2 rounds (odd ranks of a group drop out after handing over their value),
// then one lane per distinct address issues the global atomics. Replaces the
// plain per-element atomicAdd of IndexedWriteKernel (TensorKernels.cuh:177-209),
// which serialises when many paths hit the same few vertices (quads, lights).
// (Summing in shared memory instead serialised such groups as well: a float
// atomicAdd on shared memory is a compare-and-swap loop.) The rounds are those of
// E. Westphal, "Voting and Shuffling to Optimize Atomic Operations" (2015).
TRN_D void agg_add3(float* base, long long idx, const F3& g) {
  const unsigned active = __activemask();
  const int lane = threadIdx.x & 31;
  // peers share the target address, not just the index: lanes of one warp can
  // scatter into different views' gradient buffers
  float* const target = base + 3 * idx;
  const unsigned peers = __match_any_sync(active, reinterpret_cast<unsigned long long>(target));
  const unsigned lt = (1u << lane) - 1u;
  unsigned rank = __popc(peers & lt);
  const bool leader = rank == 0u;
  unsigned rest = peers & ~lt & ~(1u << lane);
  F3 x = g;
  while (__any_sync(active, rest != 0u)) {
    const int next = rest ? __ffs(rest) - 1 : lane;
    const F3 t(__shfl_sync(active, x.x, next), __shfl_sync(active, x.y, next), __shfl_sync(active, x.z, next));
    if (rest) x = x + t;
    rest &= __ballot_sync(active, !(rank & 1u));
    rank >>= 1;
  }
  if (leader) atomic_add3(target, x);
}
TRN_D F3 g_at(const Params& P, const ViewDesc& V, int pix) {
  if (pix < 0) return F3z();
  const float* d = (V.dLdI ? V.dLdI : P.dLdI + 3 * V.pix_off) + 3 * pix;
  return F3(__ldg(d), __ldg(d + 1), __ldg(d + 2)) * V.inv_spp;
}

// the view owning global slot g (last view whose first slot is <= g)
// View of a launch-global slot. `hint` is the lane's previous view: a lane's
// consecutive slots nearly always fall in the same view, so the range check
// usually replaces the binary search over the view table.
TRN_D const ViewDesc& view_of(const Params& P, long long g, int& hint) {
  const int h = hint;
  if (__ldg(P.vbegin + h) <= g && (h + 1 >= P.nviews || g < __ldg(P.vbegin + h + 1))) return P.views[h];
  int lo = 0, hi = P.nviews - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(P.vbegin + mid) <= g) lo = mid; else hi = mid - 1;
  }
  hint = lo;
  return P.views[lo];
}

// Uniform sample `dim` of one slot: the table is indexed by the launch-global
// slot, the hash by (view seed, term, dim, view-local slot).
struct PathSmp {
  const Params* P;
  uint32_t seed;
  long long gslot, lslot;
  TRN_D float operator()(int dim) const {
    if (P->table) return __ldg(P->table + (long long)dim * P->stride + gslot);
    return hash_uniform(P->seed * 1000003u + seed, P->term, (uint32_t)dim, (uint32_t)lslot);
  }
};

// Persistent work loop: each warp fetches 32*chunk consecutive slots from a
// global counter, so uneven views and path lengths balance across SMs.
template <class F>
TRN_D void for_each_slot(const Params& P, F&& body) {
  const int lane = threadIdx.x & 31;
  const long long step = 32LL * P.chunk;
  for (;;) {
    unsigned long long start = 0;
    if (lane == 0) start = atomicAdd(P.work, (unsigned long long)step);
    start = __shfl_sync(0xffffffffu, start, 0);
    if ((long long)start >= P.total) break;
    for (int j = 0; j < P.chunk; j++) {
      const long long g = (long long)start + 32LL * j + lane;
      if (g < P.total) body(g);
    }
    __syncwarp();
  }
}
TRN_D F3 cam_pos(const CameraDesc& c) { return F3(c.pos[0], c.pos[1], c.pos[2]); }

// AreaLight::Eval (Light.cpp:134-138): radiance when the emitter faces wi
TRN_D F3 emitted(const DeviceScene& s, const SurfF& x, const F3& wi) {
  if (x.emitter < 0) return F3z();
  return dot(wi, x.ng) > 0.f ? light_radiance(s, x.emitter) : F3z();
}

// ---------------------------------------------------------------------------
// templated path factors (differentiated by the adjoint)
// ---------------------------------------------------------------------------
// Next-event estimation factor of EvalRadianceDirect (Integrator.cpp:186-228),
// excluding the incoming throughput and assuming the connection is valid.
template <class S>
TRN_HD V3<S> nee_factor(const BsdfDesc& b, const V3<S>& xprev, const V3<S>& x, const V3<S>& ns, const V3<S>& ng,
                        const V3<S>& kd, const V3<S>& y, const V3<S>& nl, const S& Jl, const F3& Le, float lpdf,
                        float mis) {
  const V3<S> wo = -normalize(x - xprev);
  const Frame<S> fr = make_frame(ns);
  V3<S> wi = y - x;
  const S d2 = dot(wi, wi);
  const S d = sqrt_(d2);
  wi = wi / d;
  const S dotSh = dot(ns, wi);
  const S G = abs_(dot(nl, -wi)) / d2;
  const V3<S> bv = bsdf_eval(b, fr, ng, kd, wo, wi, false) * abs_(dotSh);
  V3<S> out;
  for (int c = 0; c < 3; c++) out[c] = bv[c] * Jl * G * Le[c] / lpdf * mis;
  return out;
}

// BSDF-sampled continuation weight in area measure (Integrator.cpp:252-267).
template <class S>
TRN_HD V3<S> cont_factor(const BsdfDesc& b, const V3<S>& xprev, const V3<S>& x, const V3<S>& ns, const V3<S>& ng,
                         const V3<S>& kd, const V3<S>& xn, const V3<S>& ngn, const S& Jn, float prev_pdf) {
  const V3<S> wo = -normalize(x - xprev);
  const Frame<S> fr = make_frame(ns);
  V3<S> dir = xn - x;
  const S dist2 = dot(dir, dir);
  dir = dir / sqrt_(dist2);
  const S G = abs_(dot(ngn, -dir)) / dist2;
  const V3<S> bv = bsdf_eval(b, fr, ng, kd, wo, dir, false) * abs_(dot(ns, dir));
  V3<S> out;
  for (int c = 0; c < 3; c++) out[c] = bv[c] * G * Jn / prev_pdf;
  return out;
}

// xDotN of the boundary terms: RayIntersectAD (Utils.cpp:288-297) from `org`
// towards `target` against triangle (P0, P1, P2), then n . (w P0 + u P1 + v P2)
// with detached vertices (BoundaryPrimary.cpp:131-145, Edge.cpp:280-291).
template <class S>
TRN_HD S xdotn(const V3<S>& org, const V3<S>& target, const V3<S>& P0, const V3<S>& P1, const V3<S>& P2,
               const F3& n) {
  const V3<S> dir = normalize(target - org);
  const V3<S> e1 = P1 - P0, e2 = P2 - P0;
  const V3<S> h = cross(dir, e2);
  const S f = 1.f / dot(e1, h);
  const V3<S> sv = org - P0;
  const S u = f * dot(sv, h);
  const V3<S> q = cross(sv, e1);
  const S v = f * dot(dir, q);
  const S w = 1.f - u - v;
  const V3<S> u2 = vdetach(P0) * w + vdetach(P1) * u + vdetach(P2) * v;
  return dot(lift<S>(n), u2);
}


// ---------------------------------------------------------------------------
// vertex records -> triangle vertices (the reparameterised PostIntersect)
// ---------------------------------------------------------------------------
struct VAdj { F3 p, ns, ng; float J; };
TRN_D void vadj_zero(VAdj& a) { a.p = F3z(); a.ns = F3z(); a.ng = F3z(); a.J = 0.f; }

// position = w P0 + u P1 + v P2 (detached u, v), face normal c/|c| and
// J = A / Detach(A) with c = cross(P1 - P0, P2 - P0), shading normal
// w n0 + u n1 + v n2 (Scene.cpp:668-730, Primitive.cpp:299-340).
#ifndef TRN_SHARED_SCATTER
#define TRN_SHARED_SCATTER 0
#endif
#if TRN_SHARED_SCATTER
#define TRN_SCATTER_FN __device__ __noinline__
#else
#define TRN_SCATTER_FN TRN_D
#endif
TRN_SCATTER_FN void scatter_vertex(const Params& P, const ViewDesc& V, int tri, float u, float v, const VAdj& a,
                                   Cnt& cnt) {
  const DeviceScene& s = P.s;
  cnt.v[kCntVScatter] += 3;
  int i0, i1, i2; tri_vertices(s, tri, i0, i1, i2);
  const float w = 1.f - u - v;
  F3 g0 = a.p * w, g1 = a.p * u, g2 = a.p * v;
  F3 gng = a.ng;
  if (s.smooth[tri]) {
    cnt.v[kCntNScatter] += 3;
    agg_add3(V.gvn, i0, a.ns * w);
    agg_add3(V.gvn, i1, a.ns * u);
    agg_add3(V.gvn, i2, a.ns * v);
  } else {
    gng = gng + a.ns;
  }
  if (gng.x != 0.f || gng.y != 0.f || gng.z != 0.f || a.J != 0.f) {
    const F3 p0 = load3(s.pos, i0), p1 = load3(s.pos, i1), p2 = load3(s.pos, i2);
    const F3 e1 = p1 - p0, e2 = p2 - p0;
    const F3 c = cross(e1, e2);
    const float len = length(c);
    const F3 n = c / len;
    const float A = 0.5f * len;
    // d|c| from J: dJ/dA = 1/A, dA/d|c| = 1/2
    const float glen = a.J * (0.5f / A);
    const F3 gc = (gng - n * dot(n, gng)) / len + n * glen;
    const F3 ge1 = cross(e2, gc), ge2 = cross(gc, e1);
    g1 = g1 + ge1; g2 = g2 + ge2; g0 = g0 - (ge1 + ge2);
  }
  agg_add3(V.gpos, i0, g0);
  agg_add3(V.gpos, i1, g1);
  agg_add3(V.gpos, i2, g2);
}

TRN_D void scatter_point(const Params& P, const ViewDesc& V, int tri, float u, float v, const F3& gp, Cnt& cnt) {
  cnt.v[kCntVScatter] += 3;
  int i0, i1, i2; tri_vertices(P.s, tri, i0, i1, i2);
  const float w = 1.f - u - v;
  agg_add3(V.gpos, i0, gp * w);
  agg_add3(V.gpos, i1, gp * u);
  agg_add3(V.gpos, i2, gp * v);
}

// ---------------------------------------------------------------------------
// one EvalRadianceDirect step for one ray (Integrator.cpp:178-303)
// ---------------------------------------------------------------------------
struct BounceRec {
  // NEE
  int ltri; float lu, lv, lpdf, lmis; int nee_ok;
  // continuation
  float prev_pdf; float emis; F3 eLe;  // MIS weight and radiance at the next vertex
  int next_ok;
  int scrubbed;                        // contribution was non-finite
};

// One bounce in two halves, so that the wavefront kernels can run the ray
// queries between them: radiance_gen decides the shadow ray and the
// continuation ray of a vertex and evaluates the next-event estimate where
// `visible` says so; radiance_resolve adds what the queries showed. `visible`
// is true for a query that comes later; the fused step answers it at once, and a
// shadowed light is not evaluated (nor kept over the ray's traversal).
struct Shading {  // of a vertex
  BsdfDesc b;
  F3 kd;
  Frame<float> fr;
};
TRN_D Shading shading_at(const DeviceScene& s, const SurfF& x) {
  Shading m;
  m.b = s.bsdfs[x.bsdf];
  long long texel;
  m.kd = bsdf_albedo(s, m.b, x.tu, x.tv, texel);
  m.fr = make_frame(x.ns);
  return m;
}
struct RadianceGen {
  F3 nee;       // contribution of the light sample if it is visible
  F3 sdir;      // shadow ray from the vertex: direction and end
  float stmax;
  bool shadow;  // the light sample needs the shadow ray
  F3 wi;        // continuation ray and its density
  float pdf;
  bool cont;
};

// rec (may be null) takes the light sample's record.
template <class Visible>
TRN_D void radiance_gen(const DeviceScene& s, const SurfF& x, const Shading& m, const F3& rdir, const F3& T, float l0,
                        float l1, float b0, float b1, float b2, RadianceGen& g, BounceRec* rec, Cnt& cnt,
                        Visible&& visible) {
  count_shade(cnt, s, x);
  const F3 wo = -rdir;
  g.shadow = false;
  LightSample ls;
  if (light_sample(s, l0, l1, ls)) {
    cnt.v[kCntLight]++;
    int j0, j1, j2; tri_vertices(s, ls.tri, j0, j1, j2);
    const F3 y = bary3(ls.bu, ls.bv, load3(s.pos, j0), load3(s.pos, j1), load3(s.pos, j2));
    const F3 nl = load3(s.fnormal, ls.tri);
    F3 wi = y - x.p;
    const float d2 = dot(wi, wi);
    const float d = sqrtf(d2);
    wi = wi / d;
    const float dotSh = dot(x.ns, wi), dotGeo = dot(x.ng, wi);
    const bool stable = d > kShadowEps && fabsf(dotSh) > kEdgeEps;
    const bool noleak = dotSh * dotGeo > 0.f;
    if (stable && noleak) cnt.v[kCntShadow]++;
    if (stable && noleak && visible(wi, d - kShadowEps)) {
      const F3 Le = dot(-wi, nl) > 0.f ? light_radiance(s, ls.light) : F3z();
      const float G = fabsf(dot(nl, -wi)) / d2;
      const float bpdf = bsdf_pdf_local(m.b, m.fr.to_local(wo), m.fr.to_local(wi)) * G;
      const float mis = ls.pdf * ls.pdf / (ls.pdf * ls.pdf + bpdf * bpdf);
      const F3 bv = bsdf_eval(m.b, m.fr, x.ng, m.kd, wo, wi, false) * fabsf(dotSh);
      for (int c = 0; c < 3; c++) g.nee[c] = T[c] * (bv[c] * 1.f * G * Le[c] / ls.pdf * mis);
      g.sdir = wi; g.stmax = d - kShadowEps; g.shadow = true;
      if (rec) {
        rec->ltri = ls.tri; rec->lu = ls.bu; rec->lv = ls.bv; rec->lpdf = ls.pdf; rec->lmis = mis;
      }
    }
  }
  // continuation (BSDF sampling)
  bsdf_sample_only(m.b, m.fr, wo, b0, b1, b2, g.wi, g.pdf);
  g.cont = g.pdf > 0.f && out_dir_valid(m.b, x.ns, x.ng, g.wi);
  if (g.cont) cnt.v[kCntClosest]++;
}

// nee_ok: the light sample is visible; hit: the continuation ray's hit (tri <
// 0: none was cast or it missed). Returns the contribution of this bounce
// (already NaN-scrubbed) in contrib; x/rdir/T move to the next vertex, and the
// return value says whether it exists.
template <class ShadingAt>
TRN_D bool radiance_resolve(const DeviceScene& s, SurfF& x, ShadingAt&& shading, F3& rdir, F3& T, bool nee_ok,
                            const F3& nee, float pdf, const Hit& h, F3& contrib, BounceRec* rec) {
  F3 val = F3z();
  if (nee_ok) val = val + nee;
  if (rec) { rec->nee_ok = nee_ok; rec->next_ok = 0; }
  if (h.tri < 0) {
    contrib = scrub(val);
    if (rec) rec->scrubbed = !finite3(val);
    return false;
  }
  const Shading m = shading();
  const F3 wo = -rdir;
  const SurfF xn = post_intersect(s, h.tri, h.u, h.v);
  F3 dir = xn.p - x.p;
  const float dist2 = dot(dir, dir);
  dir = dir / sqrtf(dist2);
  const float G = fabsf(dot(xn.ng, -dir)) / dist2;
  const F3 bv = bsdf_eval(m.b, m.fr, x.ng, m.kd, wo, dir, false) * fabsf(dot(x.ns, dir));
  const float prev_pdf = pdf * G;
  F3 Tn;
  for (int c = 0; c < 3; c++) Tn[c] = T[c] * bv[c] * G * 1.f / prev_pdf;
  if (!(G > 0.f)) Tn = F3z();
  float emis = 0.f;
  F3 eLe = F3z();
  if (xn.emitter >= 0) {
    eLe = emitted(s, xn, -dir);
    const float pn = light_pdf(s, xn.tri);
    emis = prev_pdf * prev_pdf / (prev_pdf * prev_pdf + pn * pn);
    val = val + Tn * eLe * emis;
  }
  contrib = scrub(val);
  if (rec) {
    rec->scrubbed = !finite3(val);
    rec->prev_pdf = prev_pdf; rec->emis = emis; rec->eLe = eLe; rec->next_ok = 1;
  }
  x = xn; rdir = dir; T = Tn;
  return true;
}

// The whole bounce by one thread (the fused kernels).
TRN_D bool radiance_step(const DeviceScene& s, SurfF& x, F3& rdir, F3& T, float l0, float l1, float b0, float b1,
                         float b2, F3& contrib, BounceRec* rec, Cnt& cnt) {
  const Shading m = shading_at(s, x);
  RadianceGen g;
  radiance_gen(s, x, m, rdir, T, l0, l1, b0, b1, b2, g, rec, cnt,
               [&](const F3& wi, float end) { return !occluded(s, x.p, wi, kShadowEps, end); });
  Hit h;
  h.tri = -1;
  if (g.cont && !trace<false>(s, x.p, g.wi, kShadowEps, kRayMax, h)) h.tri = -1;
  return radiance_resolve(s, x, [&] { return m; }, rdir, T, g.shadow, g.nee, g.pdf, h, contrib, rec);
}

// One shared (non-inlined) copy of the step, with the traversal inlined inside
// it, for the fused kernels that run it at more than one place or beside an
// adjoint (they are instruction-fetch bound). Every object it takes by
// reference lives in local memory.
__device__ __noinline__ bool radiance_step_shared(const DeviceScene& s, SurfF& x, F3& rdir, F3& T, float l0, float l1,
                                                  float b0, float b1, float b2, F3& contrib, BounceRec* rec, Cnt& cnt) {
  return radiance_step(s, x, rdir, T, l0, l1, b0, b1, b2, contrib, rec, cnt);
}

// Per-warp compaction of the work queue: lanes keep pulling sample slots (one
// warp-aggregated atomic per round) until each holds a slot that survives the
// cheap `setup` phase (primary hit, valid edge sample, visible, ...); then the
// warp runs the expensive `body` (path tracing + adjoint) together. Rejected
// samples therefore never hold a lane hostage while others trace long paths.
#ifndef TRN_COMPACT
#define TRN_COMPACT 1
#endif
// lanes that must hold a valid sample before the warp runs the body
#ifndef TRN_COMPACT_MIN
#define TRN_COMPACT_MIN 28
#endif

template <class State, class Setup, class Body>
TRN_D void for_each_valid(const Params& P, Setup&& setup, Body&& body) {
#if !TRN_COMPACT
  // lockstep variant: each warp takes 32 consecutive slots per round
  for_each_slot(P, [&](long long g) {
    State st;
    if (setup(g, st)) body(st);
  });
  return;
#endif
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  State st;
  bool have = false, done = false;
  for (;;) {
    for (;;) {
      const unsigned need = __ballot_sync(0xffffffffu, !have && !done);
      if (!need) break;
      // enough lanes are ready: run the body now rather than spend more
      // nearly-empty set-up rounds on the last rejections
      if (__popc(__ballot_sync(0xffffffffu, have)) >= TRN_COMPACT_MIN) break;
      const int leader = __ffs(need) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(P.work, (unsigned long long)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (!have && !done) {
        const long long g = (long long)base + __popc(need & lt);
        if (g >= P.total) done = true;
        else have = setup(g, st);
      }
    }
    if (!__any_sync(0xffffffffu, have)) break;
    if (have) { body(st); have = false; }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// interior term: forward
// ---------------------------------------------------------------------------
struct FwdState {
  const ViewDesc* V;
  long long gslot, p;
  int pix;
  SurfF x;
  F3 T, rdir, L;
};

__global__ void __launch_bounds__(256, TRN_MINB) k_path_fwd(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<FwdState>(P,
    [&](long long gslot, FwdState& st) -> bool {
      const ViewDesc& V = view_of(P, gslot, vhint);
      const long long p = gslot - V.begin;
      const CameraDesc& cam = V.cam;
      const PathSmp S{&P, V.seed, gslot, p + V.slot_off};
      const int W = cam.w, WH = cam.w * cam.h;
      const F3 org = cam_pos(cam);
      const int pix = (int)(p % WH);
      const F3 dir = camera_ray_dir(cam, pix % W, pix / W, S(0), S(1));
      Hit h;
      cnt.v[kCntClosest]++;
      if (!trace<false>(P.s, org, dir, kShadowEps, kRayMax, h, P.err)) return false;
      st.V = &V; st.gslot = gslot; st.p = p; st.pix = pix;
      st.x = post_intersect(P.s, h.tri, h.u, h.v);
      const float t1 = camera_factor<float>(cam, st.x.p, st.x.ng, 1.f);
      st.T = F3(t1, t1, t1);
      st.rdir = normalize(st.x.p - org);
      st.L = scrub(st.T * emitted(P.s, st.x, -st.rdir));
      return true;
    },
    [&](FwdState& st) {
      const ViewDesc& V = *st.V;
      const PathSmp S{&P, V.seed, st.gslot, st.p + V.slot_off};
      SurfF x = st.x;
      F3 T = st.T, rdir = st.rdir, L = st.L;
      for (int b = 0; b < V.D; b++) {
        const int o = 2 + 5 * b;
        F3 c;
        const bool more = radiance_step(P.s, x, rdir, T, S(o), S(o + 1), S(o + 2), S(o + 3), S(o + 4), c, nullptr,
                                        cnt);
        L = L + c;
        if (!more || (T.x == 0.f && T.y == 0.f && T.z == 0.f)) break;
      }
      L = L * V.inv_spp;
      cnt.v[kCntPixel]++;
      atomic_add3((V.image ? V.image : P.image + 3 * V.pix_off) + 3 * st.pix, L);
    });
  flush_cnt(cnt, P.stats);
}

// ---------------------------------------------------------------------------
// interior term: replaying adjoint
// ---------------------------------------------------------------------------
// Gradient of NEE factor w.r.t. (xprev, x, ns, kd, y, nl, Jl).
// ---------------------------------------------------------------------------
// Hand-written reverse mode of the two path factors. Both have the form
//   F_c = B_c(kd, to_local(wo), to_local(wi)) |ns.wi| |nz.wi| / d^2 J K_c
// with wo = -normalize(x - xprev), wi = (z - x) / d, d^2 = |z - x|^2, the
// frame of the (unnormalised, as in the reference) shading normal ns built by
// coordinate_system, and K_c constant (NEE: Le_c mis / lpdf, z = light point,
// nz = light normal; continuation: 1 / prev_pdf, z = next vertex, nz = its
// geometric normal). The derivative conventions are the reference AD's
// (d|x|/dx = +1 for x > 0, else -1, AbsOp::Backward). One backward sweep
// replaces seven forward-mode evaluations per factor.
// ---------------------------------------------------------------------------

// eval_inner in the local frame: returns B and accumulates dB.gB into g_lo,
// g_li (local directions) and g_kd.
TRN_HD F3 eval_inner_vjp(const BsdfDesc& b, const F3& kd, const F3& lo, const F3& li, const F3& gB, F3& g_lo,
                        F3& g_li, F3& g_kd) {
  if (b.type == kDiffuse) {
    const bool reflect = lo.z > 0.f && lo.z * li.z > 0.f;
    if (!reflect) return F3z();
    const float inv_pi = kInvPi;
    g_kd = g_kd + gB * inv_pi;
    return kd * inv_pi;
  }
  const float cv = lo.z, cl = li.z;
  if (!(cv > 0.f && cl > 0.f)) return F3z();
  const F3 hs = lo + li;
  const float Lh = length(hs);
  const F3 wh = hs / Lh;
  const float nh = wh.z, vh = dot(lo, wh);
  const float r = b.roughness;
  const float alpha = r * r;
  const float k = (r + 1.f) * (r + 1.f) * 0.125f;
  const float am1 = alpha * alpha - 1.f;
  const float qd = nh * nh * am1 + 1.f;
  const float tmp = alpha / qd;
  const float ggx = tmp * tmp * kInvPi;
  const float coeff = vh * (vh * -5.55473f - 6.8316f);
  const float e = expf(logf(2.f) * coeff);
  const float q1 = cv * (1.f - k) + k, q2 = cl * (1.f - k) + k;
  const float G1 = cv / q1, G2 = cl / q2;
  const float G = G1 * G2;
  const float den = 4.f * fabsf(cv) * fabsf(cl) + 1e-6f;
  F3 B;
  float g_ggx = 0.f, g_G = 0.f, g_e = 0.f, g_den = 0.f;
  for (int c = 0; c < 3; c++) {
    const float F0 = b.spec[c];
    const float fres = F0 + (1.f - F0) * e;
    const float spec = ggx * G * fres / den;
    B[c] = kd[c] * kInvPi + spec;
    g_ggx += gB[c] * G * fres / den;
    g_G += gB[c] * ggx * fres / den;
    g_e += gB[c] * ggx * G * (1.f - F0) / den;
    g_den -= gB[c] * spec / den;
  }
  g_kd = g_kd + gB * (float)kInvPi;
  const float g_tmp = g_ggx * 2.f * tmp * kInvPi;
  const float g_qd = -g_tmp * tmp / qd;
  const float g_nh = g_qd * 2.f * nh * am1;
  const float g_coeff = g_e * e * logf(2.f);
  const float g_vh = g_coeff * (vh * (2.f * -5.55473f) - 6.8316f);
  float g_cv = g_G * G2 * k / (q1 * q1) + g_den * 4.f * fabsf(cl) * (cv > 0.f ? 1.f : -1.f);
  float g_cl = g_G * G1 * k / (q2 * q2) + g_den * 4.f * fabsf(cv) * (cl > 0.f ? 1.f : -1.f);
  const F3 g_wh = F3(0.f, 0.f, g_nh) + lo * g_vh;
  const F3 g_hs = (g_wh - wh * dot(g_wh, wh)) / Lh;
  g_lo = g_lo + g_hs + wh * g_vh;
  g_li = g_li + g_hs;
  g_lo.z += g_cv;
  g_li.z += g_cl;
  return B;
}

// coordinate_system (Utils.cpp:118-140): t = f(n) on the branch the value took;
// accumulates dt.g_t into g_n.
TRN_HD void tangent_vjp(const F3& n, const F3& g_t, F3& g_n) {
  if (fabsf(n.x) > fabsf(n.y)) {
    const float q = n.x * n.x + n.z * n.z;
    const float inv = 1.f / sqrtf(fmaxf(q, 1e-3f));
    // t = (-n.z inv, 0, n.x inv)
    g_n.z -= g_t.x * inv;
    g_n.x += g_t.z * inv;
    if (q > 1e-3f) {
      const float g_inv = -g_t.x * n.z + g_t.z * n.x;
      const float g_q = -0.5f * g_inv * inv * inv * inv;
      g_n.x += 2.f * g_q * n.x;
      g_n.z += 2.f * g_q * n.z;
    }
  } else {
    const float q = n.y * n.y + n.z * n.z;
    const float inv = 1.f / sqrtf(fmaxf(q, 1e-3f));
    // t = (0, n.z inv, -n.y inv)
    g_n.z += g_t.y * inv;
    g_n.y -= g_t.z * inv;
    if (q > 1e-3f) {
      const float g_inv = g_t.y * n.z - g_t.z * n.y;
      const float g_q = -0.5f * g_inv * inv * inv * inv;
      g_n.y += 2.f * g_q * n.y;
      g_n.z += 2.f * g_q * n.z;
    }
  }
}

// Reverse mode of F above for the output adjoint `adj`; accumulates into the
// gradient outputs (g_prev only if need_prev, g_kd only if need_kd).
#ifndef TRN_SHARED_FACTOR_VJP
#define TRN_SHARED_FACTOR_VJP 2
#endif
// 0: inlined at each call; 1: one shared copy with reference parameters (its
// callers keep every argument in local memory); 2: one shared copy that takes
// its inputs by value and returns its gradient increments
#if TRN_SHARED_FACTOR_VJP == 1
#define TRN_FACTOR_FN __host__ __device__ __noinline__
#else
#define TRN_FACTOR_FN TRN_HD
#endif
TRN_FACTOR_FN F3 factor_vjp_acc(const BsdfDesc& b, bool need_prev, bool need_kd, const F3& xprev, const F3& x,
                                const F3& ns, const F3& kd, const F3& z, const F3& nz, float J, const F3& K,
                                const F3& adj, F3& g_prev, F3& g_x, F3& g_ns, F3& g_kd, F3& g_z, F3& g_nz,
                                float& g_J) {
  const F3 v0 = x - xprev;
  const float L0 = length(v0);
  const F3 n0 = v0 / L0;
  const F3 wo = -n0;
  const F3 vi = z - x;
  const float d2 = dot(vi, vi);
  const float d = sqrtf(d2);
  const F3 wi = vi / d;
  const Frame<float> fr = make_frame(ns);
  const F3 lo = fr.to_local(wo), li = fr.to_local(wi);
  const float cs = dot(ns, wi);
  const float u = dot(nz, -wi);
  const float Q = fabsf(cs) * fabsf(u) / d2 * J;
  const F3 A = adj * K;
  // B(kd, lo, li) with its adjoint gB = A Q
  F3 g_lo = F3z(), g_li = F3z(), gkd = F3z();
  const F3 B = eval_inner_vjp(b, kd, lo, li, A * Q, g_lo, g_li, gkd);
  const F3 F(B.x * Q * K.x, B.y * Q * K.y, B.z * Q * K.z);
  if (need_kd) g_kd = g_kd + gkd;
  const float gQ = dot(A, B);
  if (gQ == 0.f && g_lo.x == 0.f && g_lo.y == 0.f && g_lo.z == 0.f && g_li.x == 0.f && g_li.y == 0.f &&
      g_li.z == 0.f)
    return F;
  // Q = |cs| |u| / d2 J
  const float g_cs = gQ * (cs > 0.f ? 1.f : -1.f) * fabsf(u) / d2 * J;
  const float g_u = gQ * fabsf(cs) * (u > 0.f ? 1.f : -1.f) / d2 * J;
  const float g_d2 = -gQ * Q / d2;
  g_J += gQ * fabsf(cs) * fabsf(u) / d2;
  F3 g_n = wi * g_cs;                    // cs = ns . wi
  F3 g_wi = ns * g_cs - nz * g_u;        // u = -nz . wi
  g_nz = g_nz - wi * g_u;
  // local coordinates (v.t, v.b, v.n)
  const F3 g_wo = fr.t * g_lo.x + fr.b * g_lo.y + fr.n * g_lo.z;
  g_wi = g_wi + fr.t * g_li.x + fr.b * g_li.y + fr.n * g_li.z;
  F3 g_t = wo * g_lo.x + wi * g_li.x;
  const F3 g_b = wo * g_lo.y + wi * g_li.y;
  g_n = g_n + wo * g_lo.z + wi * g_li.z;
  // b = n x t
  g_n = g_n + cross(fr.t, g_b);
  g_t = g_t + cross(g_b, fr.n);
  tangent_vjp(fr.n, g_t, g_n);
  g_ns = g_ns + g_n;
  // wi = vi / |vi|, d2 = vi . vi
  const F3 g_vi = (g_wi - wi * dot(g_wi, wi)) / d + vi * (2.f * g_d2);
  g_z = g_z + g_vi;
  g_x = g_x - g_vi;
  // wo = -v0 / |v0|
  const F3 g_n0 = -g_wo;
  const F3 g_v0 = (g_n0 - n0 * dot(g_n0, n0)) / L0;
  g_x = g_x + g_v0;
  if (need_prev) g_prev = g_prev - g_v0;
  return F;
}

#if TRN_SHARED_FACTOR_VJP == 2
struct FactorGrad {
  F3 F, g_prev, g_x, g_ns, g_kd, g_z, g_nz;
  float g_J;
};
__host__ __device__ __noinline__ FactorGrad factor_vjp_byval(BsdfDesc b, bool need_prev, bool need_kd, F3 xprev, F3 x,
                                                            F3 ns, F3 kd, F3 z, F3 nz, float J, F3 K, F3 adj) {
  FactorGrad r;
  r.g_prev = r.g_x = r.g_ns = r.g_kd = r.g_z = r.g_nz = F3z();
  r.g_J = 0.f;
  r.F = factor_vjp_acc(b, need_prev, need_kd, xprev, x, ns, kd, z, nz, J, K, adj, r.g_prev, r.g_x, r.g_ns, r.g_kd,
                       r.g_z, r.g_nz, r.g_J);
  return r;
}
#endif

TRN_HD F3 factor_vjp(const BsdfDesc& b, bool need_prev, bool need_kd, const F3& xprev, const F3& x, const F3& ns,
                     const F3& kd, const F3& z, const F3& nz, float J, const F3& K, const F3& adj, F3& g_prev,
                     F3& g_x, F3& g_ns, F3& g_kd, F3& g_z, F3& g_nz, float& g_J) {
#if TRN_SHARED_FACTOR_VJP == 2
  const FactorGrad r = factor_vjp_byval(b, need_prev, need_kd, xprev, x, ns, kd, z, nz, J, K, adj);
  g_prev = g_prev + r.g_prev; g_x = g_x + r.g_x; g_ns = g_ns + r.g_ns; g_kd = g_kd + r.g_kd;
  g_z = g_z + r.g_z; g_nz = g_nz + r.g_nz; g_J += r.g_J;
  return r.F;
#else
  return factor_vjp_acc(b, need_prev, need_kd, xprev, x, ns, kd, z, nz, J, K, adj, g_prev, g_x, g_ns, g_kd, g_z,
                        g_nz, g_J);
#endif
}

// Gradient of the NEE factor w.r.t. (xprev, x, ns, kd, y, nl, Jl).
// Reverse mode of camera_factor (Camera::EvalFilter, Camera.cpp:279-303) at
// J = 1: the value G / Detach(G) is 1, so the gradient is W grad(log G) with
// log G = log|cos_x| - 3 log cos_y - 2 log dist, plus W for J.
TRN_HD void camera_factor_grad(const CameraDesc& c, const F3& p, const F3& ng, float W, F3& g_p, F3& g_ng,
                               float& g_J) {
  const F3 v = p - F3(c.pos[0], c.pos[1], c.pos[2]);
  const float dist = length(v);
  const F3 dir = v / dist;
  const F3 cdir(c.dir[0], c.dir[1], c.dir[2]);
  const float cosy = dot(dir, cdir);
  const float cosx = dot(-dir, ng);
  const F3 g_dir = (-ng) * (W / cosx) - cdir * (3.f * W / cosy);
  g_p = (g_dir - dir * dot(g_dir, dir)) / dist - dir * (2.f * W / dist);
  g_ng = (-dir) * (W / cosx);
  g_J = W;
}

// Returns the factor's value.
TRN_HD F3 nee_vjp(const BsdfDesc& b, bool need_prev, bool need_kd, const F3& xprev, const F3& x, const F3& ns,
                  const F3& ng, const F3& kd, const F3& y, const F3& nl, const F3& Le, float lpdf, float mis,
                  const F3& adj, F3& g_prev, F3& g_x, F3& g_ns, F3& g_kd, F3& g_y, F3& g_nl, float& g_Jl) {
  (void)ng;  // the factor evaluates the BSDF without the shading-normal correction
  const F3 K(Le.x / lpdf * mis, Le.y / lpdf * mis, Le.z / lpdf * mis);
  return factor_vjp(b, need_prev, need_kd, xprev, x, ns, kd, y, nl, 1.f, K, adj, g_prev, g_x, g_ns, g_kd, g_y, g_nl,
                    g_Jl);
}

// Gradient of the continuation factor w.r.t. (xprev, x, ns, kd, xn, ngn, Jn).
// Returns the factor's value.
TRN_HD F3 cont_vjp(const BsdfDesc& b, bool need_prev, bool need_kd, const F3& xprev, const F3& x, const F3& ns,
                   const F3& ng, const F3& kd, const F3& xn, const F3& ngn, float prev_pdf, const F3& adj,
                   F3& g_prev, F3& g_x, F3& g_ns, F3& g_kd, F3& g_xn, F3& g_ngn, float& g_Jn) {
  (void)ng;
  const float ip = 1.f / prev_pdf;
  return factor_vjp(b, need_prev, need_kd, xprev, x, ns, kd, xn, ngn, 1.f, F3(ip, ip, ip), adj, g_prev, g_x, g_ns,
                    g_kd, g_xn, g_ngn, g_Jn);
}

struct VRec { int tri; float u, v; };

struct AdjState {
  const ViewDesc* V;
  long long gslot, p;
  int pix;
  F3 g;
  Hit h;
};

// Interior adjoint set-up: the camera ray of the slot (paths whose pixel has a
// zero dL/dI carry no gradient and are skipped).
TRN_D bool path_adj_setup(const Params& P, long long gslot, AdjState& st, int& vhint, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = view_of(P, gslot, vhint);
  const long long p = gslot - V.begin;
  const CameraDesc& cam = V.cam;
  const PathSmp S{&P, V.seed, gslot, p + V.slot_off};
  const int W = cam.w, WH = cam.w * cam.h;
  const int pix = (int)(p % WH);
  cnt.v[kCntPixel]++;
  const F3 g = g_at(P, V, pix);
  if (g.x == 0.f && g.y == 0.f && g.z == 0.f) return false;
  const F3 dir = camera_ray_dir(cam, pix % W, pix / W, S(0), S(1));
  cnt.v[kCntClosest]++;
  if (!trace<false>(s, cam_pos(cam), dir, kShadowEps, kRayMax, st.h, P.err)) return false;
  st.V = &V; st.gslot = gslot; st.p = p; st.pix = pix; st.g = g;
  return true;
}

struct LRec { int ltri; float lu, lv, lpdf, lmis, ppdf; };

// Everything the reverse sweep of one interior path needs from its forward
// replay: vertices (hit records), per-bounce NEE light samples and
// continuation pdfs, throughputs T_k and emission terms M_k.
template <int MAXD>
struct PathRec {
  long long gslot, p;
  int view, K, D;
  unsigned nee_mask;        // bit k: bounce k's NEE contributes
  F3 g;                     // dL/dI of the path's pixel (times 1/spp)
  VRec vr[MAXD + 2];
  LRec br[MAXD + 1];
  F3 Tk[MAXD + 2], Mk[MAXD + 2];
};

// Forward replay of one interior path from its primary hit, recording into r;
// returns the path's radiance (what k_path_fwd adds to its pixel before the
// 1/spp weight).
template <int MAXD, class Rec>
TRN_D F3 path_replay(const Params& P, const AdjState& st, Rec& r, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = *st.V;
  const CameraDesc& cam = V.cam;
  const PathSmp S{&P, V.seed, st.gslot, st.p + V.slot_off};
  const F3 org = cam_pos(cam);
  const Hit h = st.h;
  r.gslot = st.gslot; r.p = st.p; r.view = (int)(st.V - P.views); r.g = st.g;
  SurfF x = post_intersect(s, h.tri, h.u, h.v);
  r.vr[1] = {h.tri, h.u, h.v};
  const float t1 = camera_factor<float>(cam, x.p, x.ng, 1.f);
  F3 T(t1, t1, t1);
  F3 rdir = normalize(x.p - org);
  r.Tk[1] = T;
  F3 m1 = emitted(s, x, -rdir);
  if (!finite3(T * m1)) m1 = F3z();
  r.Mk[1] = m1;
  F3 L = T * m1;
  int K = 1;  // vertices reached
  const int D = min(V.D, MAXD);
  unsigned mask = 0u;
  for (int b = 0; b < D; b++) {
    const int k = b + 1;
    const int o = 2 + 5 * b;
    F3 c;
    BounceRec R;
    const bool more = radiance_step_shared(s, x, rdir, T, S(o), S(o + 1), S(o + 2),
                                    S(o + 3), S(o + 4), c, &R, cnt);
    // a scrubbed (non-finite) bounce contributes nothing and carries no gradient
    if (R.nee_ok && !R.scrubbed) mask |= 1u << k;
    L = L + c;
    r.br[k] = {R.ltri, R.lu, R.lv, R.lpdf, R.lmis, R.prev_pdf};
    if (!more) break;
    r.vr[k + 1] = {x.tri, x.u, x.v};
    r.Tk[k + 1] = T;
    r.Mk[k + 1] = (R.scrubbed || R.emis == 0.f) ? F3z() : R.eLe * R.emis;
    K = k + 1;
    if (T.x == 0.f && T.y == 0.f && T.z == 0.f) break;
  }
  r.K = K;
  r.D = D;
  r.nee_mask = mask;
  return L;
}

// Reverse sweep of one recorded interior path:
// a_k = g*(N_k + M_k) + phi_k * a_{k+1}, one vertex window at a time, then
// the camera factor at vertex 1.
template <int MAXD, class Rec>
TRN_D void path_reverse(const Params& P, const Rec& r, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = P.views[r.view];
  const CameraDesc& cam = V.cam;
  const F3 org = cam_pos(cam);
  const F3 g = r.g;
  const int K = r.K, D = r.D;
  struct VG { F3 p, ns, ng, kd; long long texel; int bsdf; };
  auto load_vg = [&](int k) {
    VG o;
    const SurfF xs = post_intersect(s, r.vr[k].tri, r.vr[k].u, r.vr[k].v);
    o.p = xs.p; o.ns = xs.ns; o.ng = xs.ng; o.bsdf = xs.bsdf;
    o.kd = bsdf_albedo(s, s.bsdfs[xs.bsdf], xs.tu, xs.tv, o.texel);
    return o;
  };
  VG Gk = load_vg(K), Gn = Gk;
  F3 a_next = F3z();
  VAdj acc_next, acc_k, acc_prev;
  vadj_zero(acc_next); vadj_zero(acc_k); vadj_zero(acc_prev);
  for (int k = K; k >= 1; k--) {
    VG Gp;
    if (k >= 2) Gp = load_vg(k - 1);
    else { Gp.p = org; Gp.ns = Gp.ng = Gp.kd = F3z(); Gp.texel = -1; Gp.bsdf = 0; }
    const BsdfDesc b = s.bsdfs[Gk.bsdf];
    const bool need_prev = b.type != kDiffuse;
    const bool need_kd = P.diff_tex && Gk.texel >= 0;
    F3 Nval = F3z(), Phi = F3z();
    F3 gkd = F3z(), gprev = F3z();
    if (k <= D && ((r.nee_mask >> k) & 1u)) {
      // NEE factor value and its reverse mode in one sweep
      const LRec& R = r.br[k];
      int j0, j1, j2; tri_vertices(s, R.ltri, j0, j1, j2);
      const F3 y = bary3(R.lu, R.lv, load3(s.pos, j0), load3(s.pos, j1), load3(s.pos, j2));
      const F3 nl = load3(s.fnormal, R.ltri);
      // the forward step's emitter radiance (one-sided, AreaLight::Eval), same arithmetic
      F3 wl = y - Gk.p;
      wl = wl / sqrtf(dot(wl, wl));
      const F3 Le = dot(-wl, nl) > 0.f ? light_radiance(s, s.emitter_id[R.ltri]) : F3z();
      F3 gy = F3z(), gnl = F3z();
      float gJl = 0.f;
      Nval = nee_vjp(b, need_prev, need_kd, Gp.p, Gk.p, Gk.ns, Gk.ng, Gk.kd, y, nl, Le, R.lpdf, R.lmis,
                     r.Tk[k] * g, gprev, acc_k.p, acc_k.ns, gkd, gy, gnl, gJl);
      VAdj la; la.p = gy; la.ns = F3z(); la.ng = gnl; la.J = gJl;
      scatter_vertex(P, V, R.ltri, R.lu, R.lv, la, cnt);
    }
    if (k < K) {
      // continuation factor value and its reverse mode; a non-finite weight
      // made the forward throughput non-finite: no value, no gradient
      F3 cprev = F3z(), cx = F3z(), cns = F3z(), ckd = F3z(), cxn = F3z(), cngn = F3z();
      float gJn = 0.f;
      Phi = cont_vjp(b, need_prev, need_kd, Gp.p, Gk.p, Gk.ns, Gk.ng, Gk.kd, Gn.p, Gn.ng, r.br[k].ppdf,
                     r.Tk[k] * a_next, cprev, cx, cns, ckd, cxn, cngn, gJn);
      if (finite3(Phi)) {
        gprev = gprev + cprev; acc_k.p = acc_k.p + cx; acc_k.ns = acc_k.ns + cns; gkd = gkd + ckd;
        acc_next.p = acc_next.p + cxn; acc_next.ng = acc_next.ng + cngn; acc_next.J += gJn;
      } else {
        Phi = F3z();
      }
    }
    const F3 a_k = g * (Nval + r.Mk[k]) + Phi * a_next;
    if (k >= 2) acc_prev.p = acc_prev.p + gprev;
    if (need_kd) { cnt.v[kCntTScatter]++; agg_add3(V.gtex, Gk.texel, gkd); }
    // vertex k+1 has received all of its contributions
    if (k < K) scatter_vertex(P, V, r.vr[k + 1].tri, r.vr[k + 1].u, r.vr[k + 1].v, acc_next, cnt);
    acc_next = acc_k; acc_k = acc_prev; vadj_zero(acc_prev);
    a_next = a_k; Gn = Gk; Gk = Gp;
  }
  // primary factor T1 = G / Detach(G) * J at vertex 1 (now in Gn / acc_next)
  {
    const float gam = a_next.x + a_next.y + a_next.z;
    if (gam != 0.f && isfinite(gam)) {
      F3 gp, gn;
      float gJ;
      camera_factor_grad(cam, Gn.p, Gn.ng, gam, gp, gn, gJ);
      acc_next.p = acc_next.p + gp;
      acc_next.ng = acc_next.ng + gn;
      acc_next.J += gJ;
    }
  }
  scatter_vertex(P, V, r.vr[1].tri, r.vr[1].u, r.vr[1].v, acc_next, cnt);
}

template <int MAXD>
__global__ void __launch_bounds__(256, TRN_MINB_PATHADJ) k_path_adj(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<AdjState>(P,
    [&](long long gslot, AdjState& st) -> bool { return path_adj_setup(P, gslot, st, vhint, cnt); },
    [&](AdjState& st) {
      PathRec<MAXD> r;
      path_replay<MAXD>(P, st, r, cnt);
      path_reverse<MAXD>(P, r, cnt);
    });
  flush_cnt(cnt, P.stats);
}

// Path records in structure-of-arrays layout, for up to `cap` paths of up to
// `depth` bounces: field k of path i lives at k * cap + i, so the lanes of a
// warp (consecutive paths) read and write consecutive addresses. (`br` has no
// entry 0, and `vr`, `Tk`, `Mk` start at vertex 1; entry 0 is left out.)
struct PathSoA {
  long long cap;
  long long* p_;
  int *view_, *K_, *D_;
  unsigned* nee_;
  F3* g_;
  VRec* vr_;
  LRec* br_;
  F3 *Tk_, *Mk_;
  unsigned* order;            // [cap] the records in the order their paths ended
  unsigned long long* n_end;  // paths ended so far (nullptr: their order is not kept)
  TRN_D long long& p(long long i) const { return p_[i]; }
  TRN_D int& view(long long i) const { return view_[i]; }
  TRN_D int& K(long long i) const { return K_[i]; }
  TRN_D int& D(long long i) const { return D_[i]; }
  TRN_D unsigned& nee(long long i) const { return nee_[i]; }
  TRN_D F3& g(long long i) const { return g_[i]; }
  TRN_D VRec& vr(long long i, int k) const { return vr_[(k - 1) * cap + i]; }
  TRN_D LRec& br(long long i, int k) const { return br_[(k - 1) * cap + i]; }
  TRN_D F3& Tk(long long i, int k) const { return Tk_[(k - 1) * cap + i]; }
  TRN_D F3& Mk(long long i, int k) const { return Mk_[(k - 1) * cap + i]; }
};

// Places the arrays from `base` on and returns the bytes they take.
inline size_t path_soa(PathSoA& a, void* base, long long cap, int depth) {
  char* c = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) { char* r = c + off; off += (bytes + 255) / 256 * 256; return r; };
  const size_t n = (size_t)cap, v = (size_t)depth + 1;
  a.cap = cap;
  a.p_ = reinterpret_cast<long long*>(take(sizeof(long long) * n));
  a.view_ = reinterpret_cast<int*>(take(sizeof(int) * n));
  a.K_ = reinterpret_cast<int*>(take(sizeof(int) * n));
  a.D_ = reinterpret_cast<int*>(take(sizeof(int) * n));
  a.nee_ = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * n));
  a.g_ = reinterpret_cast<F3*>(take(sizeof(F3) * n));
  a.vr_ = reinterpret_cast<VRec*>(take(sizeof(VRec) * n * v));
  a.br_ = reinterpret_cast<LRec*>(take(sizeof(LRec) * n * std::max(depth, 1)));
  a.Tk_ = reinterpret_cast<F3*>(take(sizeof(F3) * n * v));
  a.Mk_ = reinterpret_cast<F3*>(take(sizeof(F3) * n * v));
  a.order = reinterpret_cast<unsigned*>(take(sizeof(unsigned) * n));
  a.n_end = nullptr;
  return off;
}

// One path's records with the member syntax of PathRec (path_reverse).
struct PathRef {
  const PathSoA& a;
  long long i;
  int view, K, D;
  unsigned nee_mask;
  F3 g;
  struct Vr { const PathSoA& a; long long i; TRN_D const VRec& operator[](int k) const { return a.vr(i, k); } } vr;
  struct Br { const PathSoA& a; long long i; TRN_D const LRec& operator[](int k) const { return a.br(i, k); } } br;
  struct T { const PathSoA& a; long long i; TRN_D const F3& operator[](int k) const { return a.Tk(i, k); } } Tk;
  struct M { const PathSoA& a; long long i; TRN_D const F3& operator[](int k) const { return a.Mk(i, k); } } Mk;
};

// Reverse sweep over the records, in the order in which their paths ended (up to
// kEndOrder paths) or in their own, that of the paths' slots but for the order in
// which warps start. Paths that ended together have the same length, and so have
// their sweeps: 1M paths of depth 3 on 1,284 triangles 0.59 ms, in record order
// 0.94. But the order matters to the sums. A few vertices get millions of 32-bit
// adds, small ones are lost in a large sum, and paths of another length beside it
// make the lanes' adds others. 16.8M paths of depth 5 move the position gradient by
// 6e-5 in ending order, where two runs differ by 1.5e-5; 4M by 7e-6 (two runs 6e-6),
// 1M by no more than the means of four runs differ (2e-6). Bound by instruction
// fetch: the sweep is one long body of inlined scatters, and the few warps that fit
// its registers do not hide the misses. (Its six scatters in a loop, or one shared
// function, take 5 to 10 times as long: lanes then enter them one group at a time.)
constexpr long long kEndOrder = 1 << 20;

// CACHED: the records come from the recording forward render and carry no
// dL/dI yet; each path reads its pixel's now and is skipped when that is zero,
// as the replaying form skips it.
template <bool CACHED>
__global__ void __launch_bounds__(256, TRN_MINB_REVERSE) k_path_reverse(TRN_KPARAMS, const __grid_constant__ PathSoA R) {
  stage_begin();
  Cnt cnt;
  const unsigned long long n = min(*P.q_count, (unsigned long long)P.q_cap);
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const long long i = R.n_end ? (long long)__ldcs(R.order + k) : (long long)k;
    const int view = R.view(i);
    F3 g;
    if (CACHED) {
      const ViewDesc& V = P.views[view];
      g = g_at(P, V, (int)(R.p(i) % ((long long)V.cam.w * V.cam.h)));
      if (g.x == 0.f && g.y == 0.f && g.z == 0.f) continue;
    } else {
      g = R.g(i);
    }
    const PathRef r{R, i, view, R.K(i), R.D(i), R.nee(i), g, {R, i}, {R, i}, {R, i}, {R, i}};
    path_reverse<0>(P, r, cnt);
  }
  flush_cnt(cnt, P.stats);
}

// ---------------------------------------------------------------------------
// EvalImportance for one ray (Integrator.cpp:75-176)
// ---------------------------------------------------------------------------
TRN_D bool importance_step(const DeviceScene& s, const CameraDesc& cam, SurfF& x, F3& rdir, F3& T, float b0,
                           float b1, float b2, F3& contrib, int& pix, Cnt& cnt) {
  contrib = F3z();
  pix = -1;
  const BsdfDesc b = s.bsdfs[x.bsdf];
  count_shade(cnt, s, x);
  long long texel;
  const F3 kd = bsdf_albedo(s, b, x.tu, x.tv, texel);
  const Frame<float> fr = make_frame(x.ns);
  const F3 wo = -rdir;
  const F3 cpos = cam_pos(cam);
  const SensorSample sds = sample_direct(cam, x.p);
  if (sds.valid) {
    const F3 dirc = sensor_ray_dir(cam, sds.qx, sds.qy);
    const float dist2cam = length(x.p - cpos);
    cnt.v[kCntShadow]++;
    if (!occluded(s, cpos, dirc, kShadowEps, dist2cam - kShadowEps)) {
      F3 val = F3z();
      if (out_dir_valid(b, x.ns, x.ng, wo)) {
        const F3 wi = normalize(cpos - x.p);
        if (out_dir_valid(b, x.ns, x.ng, wi))
          val = bsdf_eval(b, fr, x.ng, kd, wo, wi, true) * fabsf(dot(x.ns, wi));
      }
      contrib = scrub(T * sds.sensor_val * val);
      pix = image_pixel(cam, sds.qx, sds.qy);
    }
  }
  if (!out_dir_valid(b, x.ns, x.ng, wo)) return false;
  F3 wi; float pdf;
  bsdf_sample_only(b, fr, wo, b0, b1, b2, wi, pdf);
  const F3 bv = bsdf_eval(b, fr, x.ng, kd, wo, wi, true) * fabsf(dot(x.ns, wi));
  const F3 Tn = T * bv / pdf;
  if (!(pdf > 0.f) || !out_dir_valid(b, x.ns, x.ng, wi)) return false;
  Hit h;
  cnt.v[kCntClosest]++;
  if (!trace<false>(s, x.p, wi, kShadowEps, kRayMax, h)) return false;
  x = post_intersect(s, h.tri, h.u, h.v);
  rdir = wi;
  T = Tn;
  return true;
}

__device__ __noinline__ bool importance_step_shared(const DeviceScene& s, const CameraDesc& cam, SurfF& x, F3& rdir,
                                                    F3& T, float b0, float b1, float b2, F3& contrib, int& pix,
                                                    Cnt& cnt) {
  return importance_step(s, cam, x, rdir, T, b0, b1, b2, contrib, pix, cnt);
}

// scatter W * d xDotN / d(edge vertices, receiver point, far triangle)
// Reverse mode of xdotn (RayIntersectAD + n . (w P0 + u P1 + v P2) with
// detached vertices) for the upstream scalar W; returns the gradients w.r.t.
// org, target and the attached triangle vertices P0, P1, P2.
TRN_HD void xdotn_grad(const F3& org, const F3& target, const F3& P0, const F3& P1, const F3& P2, const F3& n,
                       float W, F3& g_org, F3& g_target, F3& g0, F3& g1, F3& g2) {
  const F3 vd = target - org;
  const float Ld = length(vd);
  const F3 dir = vd / Ld;
  const F3 e1 = P1 - P0, e2 = P2 - P0;
  const F3 h = cross(dir, e2);
  const float f = 1.f / dot(e1, h);
  const F3 sv = org - P0;
  const F3 q = cross(sv, e1);
  const float g_u = W * dot(n, P1 - P0);
  const float g_v = W * dot(n, P2 - P0);
  // v = f (dir . q), u = f (sv . h)
  const float g_f = g_v * dot(dir, q) + g_u * dot(sv, h);
  F3 g_dir = q * (g_v * f);
  const F3 g_q = dir * (g_v * f);
  F3 g_sv = h * (g_u * f);
  F3 g_h = sv * (g_u * f);
  // q = sv x e1
  g_sv = g_sv + cross(e1, g_q);
  F3 g_e1 = cross(g_q, sv);
  // f = 1 / (e1 . h)
  const float g_a = -g_f * f * f;
  g_e1 = g_e1 + h * g_a;
  g_h = g_h + e1 * g_a;
  // h = dir x e2
  g_dir = g_dir + cross(e2, g_h);
  const F3 g_e2 = cross(g_h, dir);
  // sv = org - P0, e1 = P1 - P0, e2 = P2 - P0
  g_org = g_sv;
  g0 = -(g_sv + g_e1 + g_e2);
  g1 = g_e1;
  g2 = g_e2;
  // dir = vd / |vd|
  const F3 g_vd = (g_dir - dir * dot(g_dir, dir)) / Ld;
  g_target = g_vd;
  g_org = g_org - g_vd;
}

// scatter W * d xDotN / d(edge vertices, receiver point, far triangle)
TRN_D void xdotn_vjp(const Params& P, const ViewDesc& V, float W, const F3& org, bool org_attached, int recv_tri, float ru, float rv,
                     int va_, int vb_, float sedge, const F3& target_const, int far_tri, const F3& n, Cnt& cnt) {
  const DeviceScene& s = P.s;
  cnt.v[kCntVScatter] += 3 + (va_ >= 0 ? 2 : 0);
  int i0, i1, i2; tri_vertices(s, far_tri, i0, i1, i2);
  const F3 P0 = load3(s.pos, i0), P1 = load3(s.pos, i1), P2 = load3(s.pos, i2);
  const bool edge_attached = va_ >= 0;
  F3 target = target_const, Pa = F3z(), Pb = F3z();
  if (edge_attached) {
    Pa = load3(s.pos, va_);
    Pb = load3(s.pos, vb_);
    target = Pa + (Pb - Pa) * sedge;
  }
  F3 gorg, gt, g0, g1, g2;
  xdotn_grad(org, target, P0, P1, P2, n, W, gorg, gt, g0, g1, g2);
  // a degenerate sample (the line org -> target parallel to the far
  // triangle, or org == target) has no finite derivative; it contributes
  // nothing instead of turning the whole gradient buffer into NaN
  if (!(finite3(g0) && finite3(g1) && finite3(g2) && (!edge_attached || finite3(gt)) &&
        (!org_attached || finite3(gorg))))
    return;
  agg_add3(V.gpos, i0, g0);
  agg_add3(V.gpos, i1, g1);
  agg_add3(V.gpos, i2, g2);
  if (edge_attached) {
    agg_add3(V.gpos, va_, gt * (1.f - sedge));
    agg_add3(V.gpos, vb_, gt * sedge);
  }
  if (org_attached) scatter_point(P, V, recv_tri, ru, rv, gorg, cnt);
}

// boundary geometry term baseVal (BoundaryPrimary.cpp:115-129, Edge.cpp:258-271)
TRN_D float base_val(float ratio, const F3& edge, const F3& d, const F3& nrm, const F3& edge2, F3& n_out) {
  const F3 e = cross(edge, d);
  const float sinphi = length(e);
  const F3 proj = normalize(cross(e, nrm));
  const float sinphi2 = length(cross(d, proj));
  n_out = normalize(cross(nrm, proj));
  const bool sign0 = dot(e, edge2) > 0.f;
  const bool sign1 = dot(e, n_out) > 0.f;
  float bv = ratio * (sinphi / sinphi2);
  bv = bv * (sinphi > kEps ? 1.f : 0.f) * (sinphi2 > kEps ? 1.f : 0.f);
  return bv * (sign0 == sign1 ? 1.f : -1.f);
}

// ---------------------------------------------------------------------------
// primary boundary (BoundaryPrimary.cpp:36-181, SampleFromPrimEdges Edge.cpp:350-367)
// ---------------------------------------------------------------------------
struct EdgeState {
  const ViewDesc* V;
  long long gslot, p;
  SurfF x;         // receiving surface (sensor side for direct/indirect)
  SurfF xe;        // emitter-side surface (indirect)
  F3 rdir;         // incoming direction at x
  F3 T0;           // start throughput / emitted radiance scale
  F3 p0;           // edge point
  F3 n;            // detached xDotN normal
  float w0;        // Detach(baseVal / pdf) factor
  float sedge;     // edge parameter of p0
  int v0, v1;      // edge vertices (-1: not a scene parameter)
  int far_tri;     // triangle intersected by RayIntersectAD
  int pix;         // primary / pixel: pixel of the sensor point
  F3 g;
};

// Primary boundary set-up (SampleFromPrimEdges, Edge.cpp:350-367;
// BoundaryPrimary.cpp:60-130) in three parts around its two ray queries:
// silhouette edge point and the ray that continues the camera's line behind
// it; the sensor sample of the point hit there, with the ray that tests its
// visibility; boundary geometry. Each returns false for a rejected sample.
struct EdgePoint {
  const ViewDesc* V;
  long long p;
  int v0, v1;
  float s;            // position on the edge
  float pdf;
  F3 p0, edge, edge2;
  F3 dir;             // first set-up ray, from p0
};

TRN_D bool primary_point(const Params& P, long long gslot, EdgePoint& q, int& vhint) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = view_of(P, gslot, vhint);
  q.V = &V;
  q.p = gslot - V.begin;
  const PathSmp S{&P, V.seed, gslot, q.p + V.slot_off};
  const float r0 = S(0), r1 = S(1);
  float reuse;
  const float integral = __ldg(V.pint);
  if (!(integral > 0.f)) return false;
  const int e = sample_discrete(V.pcdf, P.ne, r0, reuse);
  const int v2 = P.edges[5 * e + 4];
  q.v0 = P.edges[5 * e]; q.v1 = P.edges[5 * e + 1];
  const float len_e = V.pfunc[e];
  if (!(len_e > 0.f)) return false;
  const float pmf = len_e / (integral * (float)P.ne);
  q.pdf = pmf / len_e;
  const F3 Pa = load3(s.pos, q.v0), Pb = load3(s.pos, q.v1), Pc = load3(s.pos, v2);
  const F3 e1 = Pb - Pa;
  q.s = r1;
  q.p0 = Pa + e1 * r1;
  q.edge = normalize(e1); q.edge2 = normalize(Pc - Pa);
  q.dir = normalize(q.p0 - cam_pos(V.cam));
  return true;
}

// Sensor sample of the point that the first ray (p0, dir) hit at distance t.
TRN_D bool primary_sensor(const CameraDesc& cam, const F3& p0, const F3& dir, float t, SensorSample& sds, F3& dirc,
                          float& tmax) {
  const F3 hitP = p0 + dir * t;
  sds = sample_direct(cam, hitP);
  if (!sds.valid) return false;
  dirc = sensor_ray_dir(cam, sds.qx, sds.qy);
  tmax = length(p0 - cam_pos(cam)) - kShadowEps;
  return true;
}

TRN_D bool primary_finish(const Params& P, long long gslot, const EdgePoint& q, const Hit& h, const SensorSample& sds,
                          const F3& dirc, EdgeState& st) {
  const ViewDesc& V = *q.V;
  const CameraDesc& cam = V.cam;
  const F3 cpos = cam_pos(cam);
  const SurfF x = post_intersect(P.s, h.tri, h.u, h.v);
  const float dist = length(x.p - cpos);
  const float dist1 = length(q.p0 - cpos);
  const float cos2 = fabsf(dot(x.ng, -dirc));
  F3 n;
  const float bval = base_val((dist / dist1), q.edge, dirc, x.ng, q.edge2, n) * cos2;
  const int pix = image_pixel(cam, sds.qx, sds.qy);
  const F3 g = g_at(P, V, pix);
  if (bval == 0.f || (g.x == 0.f && g.y == 0.f && g.z == 0.f)) return false;
  st.V = &V; st.gslot = gslot; st.p = q.p; st.x = x; st.rdir = dirc;
  st.T0 = F3(sds.sensor_val, sds.sensor_val, sds.sensor_val);
  st.p0 = q.p0; st.n = n; st.w0 = bval / q.pdf; st.sedge = q.s; st.v0 = q.v0; st.v1 = q.v1; st.far_tri = h.tri;
  st.pix = pix; st.g = g;
  return true;
}

// The whole set-up by one thread (the fused kernel).
TRN_D bool primary_setup(const Params& P, long long gslot, EdgeState& st, int& vhint, Cnt& cnt) {
  EdgePoint q;
  if (!primary_point(P, gslot, q, vhint)) return false;
  Hit h;
  cnt.v[kCntClosest]++;
  if (!trace_shared<false>(P.s, q.p0, q.dir, kShadowEps, kRayMax, h, P.err)) return false;
  SensorSample sds;
  F3 dirc;
  float tmax;
  if (!primary_sensor(q.V->cam, q.p0, q.dir, h.t, sds, dirc, tmax)) return false;
  cnt.v[kCntShadow]++;
  Hit hv;
  if (trace_shared<true>(P.s, cam_pos(q.V->cam), dirc, kShadowEps, tmax, hv, nullptr)) return false;
  return primary_finish(P, gslot, q, h, sds, dirc, st);
}

// Primary boundary body: detached radiance along the camera ray through the
// sensor point (BoundaryPrimary.cpp:150-175), then the xDotN scatter.
// (also the pixel boundary's body: its samples start at dimension 1 and its
// edge point is not a scene parameter, v0 = v1 = -1)
TRN_D void primary_body(const Params& P, const ViewDesc& V, long long gslot, long long p, SurfF x, F3 rdir, F3 T,
                        float w0, const F3& g, int v0, int v1, float sedge, const F3& p0, int far_tri, const F3& n,
                        Cnt& cnt, int dim0 = 2) {
  const DeviceScene& s = P.s;
  const PathSmp S{&P, V.seed, gslot, p + V.slot_off};
  F3 L = scrub(T * emitted(s, x, -rdir));
  for (int b = 0; b < V.D; b++) {
    const int o = dim0 + 5 * b;
    F3 c;
    const bool more = radiance_step(s, x, rdir, T, S(o), S(o + 1), S(o + 2), S(o + 3),
                                                                S(o + 4), c, nullptr, cnt);
    L = L + c;
    if (!more || (T.x == 0.f && T.y == 0.f && T.z == 0.f)) break;
  }
  const float W = dot(g, L * w0);
  if (W == 0.f || !isfinite(W)) return;
  xdotn_vjp(P, V, W, cam_pos(V.cam), false, -1, 0.f, 0.f, v0, v1, sedge, p0, far_tri, n, cnt);
}

__global__ void __launch_bounds__(256, TRN_MINB) k_primary_adj(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<EdgeState>(P,
    [&](long long gslot, EdgeState& st) -> bool { return primary_setup(P, gslot, st, vhint, cnt); },
    [&](EdgeState& st) {
      primary_body(P, *st.V, st.gslot, st.p, st.x, st.rdir, st.T0, st.w0, st.g, st.v0, st.v1, st.sedge, st.p0,
                   st.far_tri, st.n, cnt);
    });
  flush_cnt(cnt, P.stats);
}

// A sample that passed the set-up of the primary (or pixel) term; its radiance
// path and scatter follow.
struct PrimaryItem {
  long long p;
  int view, x_tri;
  float x_u, x_v, T0, w0, sedge;
  int v0, v1, far_tri;
  F3 rdir, p0, n, g;
};

// ---------------------------------------------------------------------------
// direct boundary (BoundaryDirect.cpp:38-143, Edge.cpp:90-144, 201-309)
// ---------------------------------------------------------------------------
// coordinate `axis` of a point placed by r in [0, 1) in guiding leaf `leaf`
TRN_D float aq_lerp(const float* box, long long cap, int leaf, int axis, float r) {
  const float lo = __ldg(box + axis * cap + leaf), hi = __ldg(box + (3 + axis) * cap + leaf);
  return __fadd_rn(lo, __fmul_rn(r, __fsub_rn(hi, lo)));
}

// Direct boundary set-up (SampleBoundarySegmentDirect, Edge.cpp:108-144, with
// AQ guiding when enabled; EvalBoundarySegmentDirect's geometry,
// Edge.cpp:201-291): edge and light points with the ray to the light; whether
// that ray met the light point; the receiver behind the edge and the boundary
// geometry. Each part returns false for a rejected sample.
struct DirectPoint {
  EdgePoint e;        // dir: from the edge point to the light
  F3 p2, nL;          // light point and normal
};

TRN_D bool direct_point(const Params& P, long long gslot, DirectPoint& q, int& vhint, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = view_of(P, gslot, vhint);
  q.e.V = &V;
  q.e.p = gslot - V.begin;
  const PathSmp S{&P, V.seed, gslot, q.e.p + V.slot_off};
  float r0 = S(0), r1 = S(1), r2 = S(2);
  float reuse;
  const float integral = __ldg(P.eint);
  if (!(integral > 0.f)) return false;
  float pdf_b = 1.f;
  if (P.aq_cdf) {
    // AdaptiveQuadratureDistribution::sample (AQ_distrb.h:176-195): pick a
    // leaf with the extra uniform, then place the (edge, light) sample point
    // uniformly in its box
    if (!(__ldg(P.aq_int) > 0.f)) return false;
    float unused;
    const int leaf = sample_discrete(P.aq_cdf, __ldg(P.aq_n), S(3 + 3 * V.D), unused);
    r0 = aq_lerp(P.aq_box, P.aq_cap, leaf, 0, r0);
    r1 = aq_lerp(P.aq_box, P.aq_cap, leaf, 1, r1);
    r2 = aq_lerp(P.aq_box, P.aq_cap, leaf, 2, r2);
    pdf_b = __fdiv_rn(__ldg(P.aq_poly + leaf), __ldg(P.aq_int + 1));
  }
  const int e = sample_discrete(P.ecdf, P.ne, r0, reuse);
  const int f0 = P.edges[5 * e + 2], f1 = P.edges[5 * e + 3], v2 = P.edges[5 * e + 4];
  q.e.v0 = P.edges[5 * e]; q.e.v1 = P.edges[5 * e + 1];
  const float len_e = P.efunc[e];
  if (!(len_e > 0.f)) return false;
  const float pdf_e = (len_e / (integral * (float)P.ne)) / len_e;
  const F3 Pa = load3(s.pos, q.e.v0), Pb = load3(s.pos, q.e.v1), Pc = load3(s.pos, v2);
  const F3 e1 = Pb - Pa;
  q.e.s = reuse;
  q.e.p0 = Pa + e1 * reuse;
  q.e.edge = normalize(e1); q.e.edge2 = normalize(Pc - Pa);
  LightSample ls;
  if (!light_sample(s, r1, r2, ls)) return false;
  int j0, j1, j2; tri_vertices(s, ls.tri, j0, j1, j2);
  q.p2 = bary3(ls.bu, ls.bv, load3(s.pos, j0), load3(s.pos, j1), load3(s.pos, j2));
  q.nL = load3(s.fnormal, ls.tri);
  const F3 ev = q.p2 - q.e.p0;
  const float dist_sqr = dot(ev, ev);
  const float dist = sqrtf(dist_sqr);
  const F3 en = ev / dist;
  const float cos_t = dot(q.nL, -en);
  const F3 n0 = load3(s.fnormal, f0);
  const F3 n1 = f1 >= 0 ? load3(s.fnormal, f1) : F3z();
  const bool is_b = f1 < 0;
  const float c0 = dot(en, n0), c1 = dot(en, n1);
  const bool valid0 = fabsf(c0) > kEdgeEps;
  const bool valid1 = (c0 > kEdgeEps && c1 < -kEdgeEps) || (c0 < -kEdgeEps && c1 > kEdgeEps);
  const bool right = (is_b && valid0) || (!is_b && valid1);
  if (!(right && cos_t > kEps && dist > kShadowEps)) return false;
  q.e.pdf = pdf_e * ls.pdf * dist_sqr / cos_t * pdf_b;
  const F3 rdir = normalize(q.e.p0 - q.p2);
  q.e.dir = -rdir;
  cnt.v[kCntClosest] += 2;
  cnt.v[kCntLight]++;
  return true;
}

// The first ray, from the edge point to the light, met the light point.
TRN_D bool direct_lit(const DirectPoint& q, float t) {
  const F3 hp = q.e.p0 + q.e.dir * t;
  return length(hp - q.p2) < kShadowEps;
}

// h0: the light-side hit, h: the receiver behind the edge.
TRN_D bool direct_finish(const Params& P, long long gslot, const DirectPoint& q, const Hit& h0, const Hit& h,
                         EdgeState& st) {
  const DeviceScene& s = P.s;
  const F3 rdir = -q.e.dir;
  const SurfF xl = post_intersect(s, h0.tri, h0.u, h0.v);
  const F3 E = emitted(s, xl, rdir);
  const SurfF x = post_intersect(s, h.tri, h.u, h.v);
  const float dl = length(q.p2 - x.p);
  const float cos2 = fabsf(dot(q.nL, rdir));
  const float its_t = length(x.p - q.e.p0);
  F3 n;
  const float bval = base_val(its_t / dl, q.e.edge, q.e.dir, q.nL, q.e.edge2, n) * cos2;
  if (bval == 0.f || (E.x == 0.f && E.y == 0.f && E.z == 0.f)) return false;
  st.V = q.e.V; st.gslot = gslot; st.p = q.e.p; st.x = x; st.rdir = rdir; st.T0 = E; st.p0 = q.e.p0; st.n = n;
  st.w0 = bval / q.e.pdf; st.sedge = q.e.s; st.v0 = q.e.v0; st.v1 = q.e.v1; st.far_tri = h0.tri;
  return true;
}

TRN_D bool direct_setup(const Params& P, long long gslot, EdgeState& st, int& vhint, Cnt& cnt) {
  DirectPoint q;
  if (!direct_point(P, gslot, q, vhint, cnt)) return false;
  Hit h0, h;
  if (!trace<false>(P.s, q.e.p0, q.e.dir, kShadowEps, kRayMax, h0, P.err)) return false;
  if (!trace<false>(P.s, q.e.p0, -q.e.dir, kShadowEps, kRayMax, h, P.err)) return false;
  if (!direct_lit(q, h0.t)) return false;
  return direct_finish(P, gslot, q, h0, h, st);
}

// Direct boundary body: trace towards the sensor (EvalImportance per bounce,
// Integrator.cpp:75-176), then the xDotN scatter.
TRN_D void direct_body(const Params& P, const ViewDesc& V, long long gslot, long long p, const SurfF& x0, const F3& rdir,
                       const F3& ev0, int v0, int v1, float sedge, const F3& p0, int far_tri, const F3& n, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const PathSmp S{&P, V.seed, gslot, p + V.slot_off};
  F3 T(1.f, 1.f, 1.f);
  F3 dirs = rdir;
  float W = 0.f;
  SurfF xs = x0;
  for (int b = 0; b < V.D; b++) {
    const int o = 3 + 3 * b;
    F3 c; int pix;
    const bool more = importance_step(s, V.cam, xs, dirs, T, S(o), S(o + 1), S(o + 2), c,
                                                                 pix, cnt);
    if (pix >= 0) W += dot(g_at(P, V, pix), ev0 * c);
    if (!more) break;
  }
  if (W == 0.f || !isfinite(W)) return;
  xdotn_vjp(P, V, W, x0.p, true, x0.tri, x0.u, x0.v, v0, v1, sedge, p0, far_tri, n, cnt);
}

__global__ void __launch_bounds__(256, TRN_MINB) k_direct_adj(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<EdgeState>(P,
    [&](long long gslot, EdgeState& st) -> bool { return direct_setup(P, gslot, st, vhint, cnt); },
    [&](EdgeState& st) {
      direct_body(P, *st.V, st.gslot, st.p, st.x, st.rdir, st.T0 * st.w0, st.v0, st.v1, st.sedge, st.p0, st.far_tri,
                  st.n, cnt);
    });
  flush_cnt(cnt, P.stats);
}

// A sample that passed the direct set-up; its importance path and scatter follow.
struct DirectItem {
  long long p;
  int view, x_tri, v0, v1, far_tri, pad_;
  float x_u, x_v, sedge, pad2_;
  F3 rdir, ev0, p0, n;
};

// ---------------------------------------------------------------------------
// AQ guiding of the direct boundary term (AdaptiveQuadratureDistribution::setup,
// AQ_distrb.h:83-173; leaf boxes of NEE.cu:70-89 build_tree at depth 0)
// ---------------------------------------------------------------------------
constexpr uint32_t kGuideTerm = 5;  // hash-sampler term of the set-up samples

// |baseVal| of one (edge, light) sample in guiding mode (Edge.cpp:201-259 with
// guiding_mode=true): only the evaluation mask (same point, both rays hit)
// applies, and neither radiance nor pdf enters. Invalid samples give 0.
// e.dir: from the edge point to the light point.
TRN_D bool guide_point(const Params& P, float x, float y, float z, DirectPoint& q) {
  const DeviceScene& s = P.s;
  float reuse;
  const int e = sample_discrete(P.ecdf, P.ne, x, reuse);
  const int v0 = P.edges[5 * e], v1 = P.edges[5 * e + 1], v2 = P.edges[5 * e + 4];
  const F3 Pa = load3(s.pos, v0), Pb = load3(s.pos, v1), Pc = load3(s.pos, v2);
  const F3 e1 = Pb - Pa;
  q.e.p0 = Pa + e1 * reuse;
  q.e.edge = normalize(e1); q.e.edge2 = normalize(Pc - Pa);
  LightSample ls;
  if (!light_sample(s, y, z, ls)) return false;
  int j0, j1, j2; tri_vertices(s, ls.tri, j0, j1, j2);
  q.p2 = bary3(ls.bu, ls.bv, load3(s.pos, j0), load3(s.pos, j1), load3(s.pos, j2));
  q.nL = load3(s.fnormal, ls.tri);
  q.e.dir = -normalize(q.e.p0 - q.p2);
  return true;
}

// h: the receiver behind the edge; the ray to the light met the light point.
TRN_D float guide_value(const Params& P, const DirectPoint& q, const Hit& h) {
  const SurfF xs = post_intersect(P.s, h.tri, h.u, h.v);
  const float dl = length(q.p2 - xs.p);
  const float cos2 = fabsf(dot(q.nL, -q.e.dir));
  const float its_t = length(xs.p - q.e.p0);
  F3 n;
  const float bv = fabsf(base_val(its_t / dl, q.e.edge, q.e.dir, q.nL, q.e.edge2, n) * cos2);
  return isfinite(bv) ? bv : 0.f;
}

// The whole sample by one thread (the allocation-free entry point).
TRN_D float guide_base_val(const Params& P, float x, float y, float z) {
  DirectPoint q;
  if (!guide_point(P, x, y, z, q)) return 0.f;
  Hit h0, h;
  if (!trace<false>(P.s, q.e.p0, q.e.dir, kShadowEps, kRayMax, h0, P.err)) return 0.f;
  if (!trace<false>(P.s, q.e.p0, -q.e.dir, kShadowEps, kRayMax, h, P.err)) return 0.f;
  if (!direct_lit(q, h0.t)) return 0.f;
  return guide_value(P, q, h);
}

constexpr uint32_t kRefineTerm = 6;  // hash-sampler term of the refinement's random points
constexpr int kAqPoints = 36;        // evaluation points per leaf and refinement pass

// Depth-0 tree (build_tree, NEE.cu:70-89, with one y and one z cell): leaf i
// is edge i's interval of the secondary-edge CDF times [0, 1]^2.
__global__ void k_aq_init(int ne, const float* ecdf, float* box, int* edge, int* count, long long cap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) { count[0] = ne; count[1] = ne; }
  if (i >= ne) return;
  box[i] = i > 0 ? ecdf[i - 1] : 0.f;
  box[cap + i] = 0.f;
  box[2 * cap + i] = 0.f;
  box[3 * cap + i] = ecdf[i];
  box[4 * cap + i] = 1.f;
  box[5 * cap + i] = 1.f;
  edge[i] = i;
}

// Evaluation point k of a leaf for a refinement pass (gen_eval_point,
// NEE.cu:91-240, with the box midpoint m = (p0 + p1) / 2): k < 16 are the
// corners and edge midpoints of the x = p0 and x = p1 faces, 16..19 the
// corners of the x = m section, and 20..35 two random points in each octant
// (octant bits x, y, z = bits 2, 1, 0 of k - 20; the second eight use 1 - r).
TRN_D void aq_point(const float* box, long long cap, int leaf, int k, uint32_t stream, float out[3]) {
  float lo[3], hi[3], mid[3];
  for (int a = 0; a < 3; a++) {
    lo[a] = box[a * cap + leaf];
    hi[a] = box[(3 + a) * cap + leaf];
    mid[a] = __fmul_rn(__fadd_rn(lo[a], hi[a]), 0.5f);
  }
  if (k < 20) {
    // (y, z) of the face points: low, high or middle per axis
    const unsigned char yz16[8][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 0}, {1, 1}, {1, 2}, {2, 0}, {2, 1}};
    const unsigned char yz4[4][2] = {{0, 0}, {0, 1}, {1, 0}, {1, 1}};
    const int sx = k < 8 ? 0 : (k < 16 ? 1 : 2);
    const unsigned char* yz = k < 16 ? yz16[k & 7] : yz4[k - 16];
    auto pick = [&](int a, int c) { return c == 0 ? lo[a] : (c == 1 ? hi[a] : mid[a]); };
    out[0] = pick(0, sx);
    out[1] = pick(1, yz[0]);
    out[2] = pick(2, yz[1]);
    return;
  }
  const int o = (k - 20) & 7;
  for (int a = 0; a < 3; a++) {
    float r = hash_uniform(stream, kRefineTerm, (uint32_t)(3 * (k - 20) + a), (uint32_t)leaf);
    if (k >= 28) r = __fsub_rn(1.f, r);
    const float base = ((o >> (2 - a)) & 1) ? mid[a] : lo[a];
    out[a] = __fadd_rn(base, __fmul_rn(__fsub_rn(mid[a], lo[a]), r));
  }
}

// One thread per (leaf, point): |baseVal| at the refinement's evaluation
// points (GuideDirectBoundary_Helper, AQ_distrb.h:65-79).
__global__ void k_aq_eval(TRN_KPARAMS, uint32_t stream, const float* box, const int* edge, const int* count,
                          long long cap, float* eval) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int leaf = (int)(t / kAqPoints), k = (int)(t % kAqPoints);
  if (leaf >= __ldg(count)) return;
  float v = 0.f;
  if (P.efunc[edge[leaf]] > 0.f && __ldg(P.eint) > 0.f) {
    float x[3];
    aq_point(box, cap, leaf, k, stream, x);
    v = guide_base_val(P, x[0], x[1], x[2]);
  }
  eval[t] = v;
}

// sum of the 8 listed evaluation values of a leaf, added in list order, over 8
TRN_D float aq_avg8(const float* e, int a, int b, int c, int d, int f, int g, int h, int i) {
  float s = __fadd_rn(e[a], e[b]);
  s = __fadd_rn(s, e[c]);
  s = __fadd_rn(s, e[d]);
  s = __fadd_rn(s, e[f]);
  s = __fadd_rn(s, e[g]);
  s = __fadd_rn(s, e[h]);
  s = __fadd_rn(s, e[i]);
  return __fdiv_rn(s, 8.f);
}

// Split decision per leaf (cut_tree, NEE.cu:243-396): the leaf's error is
// |corner average - Monte Carlo average| x volume; above `thold` it splits
// along the axis whose two halves disagree most between their corner and
// Monte Carlo averages (a random axis on ties). flag = 0 (keep) or 1 + axis.
__global__ void k_aq_flag(const float* box, const int* count, long long cap, const float* eval, float thold,
                          uint32_t stream, int* flag) {
  const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  if (leaf >= __ldg(count)) return;
  const float* e = eval + (long long)leaf * kAqPoints;
  const float vol = __fmul_rn(__fmul_rn(__fsub_rn(box[3 * cap + leaf], box[leaf]),
                                        __fsub_rn(box[4 * cap + leaf], box[cap + leaf])),
                              __fsub_rn(box[5 * cap + leaf], box[2 * cap + leaf]));
  const float lag = aq_avg8(e, 0, 1, 3, 4, 8, 9, 11, 12);
  float mc = 0.f;
  for (int k = 20; k < 36; k++) mc = __fadd_rn(mc, e[k]);
  mc = __fdiv_rn(mc, 16.f);
  const float err = __fmul_rn(fabsf(__fsub_rn(lag, mc)), vol);
  int f = 0;
  if (err > thold) {
    const float d1a = aq_avg8(e, 0, 1, 3, 4, 16, 17, 18, 19), d1b = aq_avg8(e, 8, 9, 11, 12, 16, 17, 18, 19);
    const float d2a = aq_avg8(e, 0, 1, 6, 7, 8, 9, 14, 15), d2b = aq_avg8(e, 3, 4, 6, 7, 11, 12, 14, 15);
    const float d3a = aq_avg8(e, 0, 2, 3, 5, 8, 10, 11, 13), d3b = aq_avg8(e, 1, 2, 4, 5, 9, 10, 12, 13);
    const float m1a = aq_avg8(e, 20, 21, 22, 23, 28, 29, 30, 31), m1b = aq_avg8(e, 24, 25, 26, 27, 32, 33, 34, 35);
    const float m2a = aq_avg8(e, 20, 21, 24, 25, 28, 29, 32, 33), m2b = aq_avg8(e, 22, 23, 26, 27, 30, 31, 34, 35);
    const float m3a = aq_avg8(e, 20, 22, 24, 26, 28, 30, 32, 34), m3b = aq_avg8(e, 21, 23, 25, 27, 29, 31, 33, 35);
    const float e0 = fabsf(__fsub_rn(fabsf(__fsub_rn(d1a, m1a)), fabsf(__fsub_rn(d1b, m1b))));
    const float e1 = fabsf(__fsub_rn(fabsf(__fsub_rn(d2a, m2a)), fabsf(__fsub_rn(d2b, m2b))));
    const float e2 = fabsf(__fsub_rn(fabsf(__fsub_rn(d3a, m3a)), fabsf(__fsub_rn(d3b, m3b))));
    int axis;
    if (e0 > e1 && e0 > e2) axis = 0;
    else if (e1 > e0 && e1 > e2) axis = 1;
    else if (e2 > e0 && e2 > e1) axis = 2;
    else {
      const float r = __fmul_rn(hash_uniform(stream, kRefineTerm, 48u, (uint32_t)leaf), 3.f);
      axis = r < 1.f ? 0 : (r < 2.f ? 1 : 2);
    }
    f = 1 + axis;
  }
  flag[leaf] = f;
}

// Exclusive prefix count of the split flags in leaf order (one block), so
// that new leaves are appended in a fixed order; count[1] = leaves after the
// pass, at most `limit`.
__global__ void k_aq_scan(const int* count, const int* flag, int* prefix, int* count_out, int limit) {
  __shared__ int part[1024];
  const int n = __ldg(count);
  const int T = blockDim.x, tid = threadIdx.x;
  const int chunk = (n + T - 1) / T;
  const int a = min(n, tid * chunk), b = min(n, a + chunk);
  int acc = 0;
  for (int i = a; i < b; i++) acc += flag[i] != 0;
  part[tid] = acc;
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int i = 0; i < T; i++) { const int x = part[i]; part[i] = run; run += x; }
    count_out[1] = min(n + run, limit);
  }
  __syncthreads();
  int run = part[tid];
  for (int i = a; i < b; i++) { prefix[i] = run; run += flag[i] != 0; }
}

// Split the flagged leaves: the leaf keeps the lower half along its axis and
// the new leaf n + prefix takes the upper half (cut_tree's split).
__global__ void k_aq_split(const int* count, const int* flag, const int* prefix, float* box, int* edge,
                           long long cap) {
  const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = __ldg(count);
  if (leaf >= n || flag[leaf] == 0) return;
  const int idx = n + prefix[leaf];
  if (idx >= __ldg(count + 1)) return;
  const int axis = flag[leaf] - 1;
  const float lo = box[axis * cap + leaf], hi = box[(3 + axis) * cap + leaf];
  const float mid = __fmul_rn(__fadd_rn(lo, hi), 0.5f);
  for (int c = 0; c < 6; c++) box[c * cap + idx] = box[c * cap + leaf];
  box[axis * cap + idx] = mid;
  box[(3 + axis) * cap + leaf] = mid;
  edge[idx] = edge[leaf];
}

__global__ void k_aq_commit(int* count) { count[0] = count[1]; }

// Leaf weight = mean |baseVal| over gspp uniform samples in the leaf box
// (AQ_distrb.h:150-161). Leaves on non-secondary edges (zero length in the
// edge distribution) do not exist in the reference's compacted edge list and
// get weight 0 here.
__global__ void k_aq_poly(TRN_KPARAMS, uint32_t stream, int gspp, const float* box, const int* edge, const int* count,
                          long long cap, float* poly) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= __ldg(count)) return;
  float acc = 0.f;
  if (P.efunc[edge[i]] > 0.f && __ldg(P.eint) > 0.f) {
    const float fs = (float)gspp;
    for (int k = 0; k < gspp; k++) {
      const uint32_t slot = (uint32_t)i * (uint32_t)gspp + (uint32_t)k;
      const float x = aq_lerp(box, cap, i, 0, hash_uniform(stream, kGuideTerm, 0, slot));
      const float y = aq_lerp(box, cap, i, 1, hash_uniform(stream, kGuideTerm, 1, slot));
      const float z = aq_lerp(box, cap, i, 2, hash_uniform(stream, kGuideTerm, 2, slot));
      acc = __fadd_rn(acc, __fdiv_rn(guide_base_val(P, x, y, z), fs));
    }
  }
  poly[i] = acc;
}

// poly /= sum(poly); poly = eps + (1 - eps) poly; func = poly x leaf volume;
// out[1] = sum(func) (the pdf normaliser of AQ_distrb.h:194). One block of
// 1024 threads.
__global__ void k_aq_mix(const int* count, float* poly, const float* box, long long cap, float eps, float* func,
                         float* out) {
  __shared__ double part[1024];
  const int n = __ldg(count);
  const int tid = threadIdx.x, T = blockDim.x;
  double acc = 0.0;
  for (int i = tid; i < n; i += T) acc += (double)poly[i];
  part[tid] = acc;
  __syncthreads();
  for (int w = T / 2; w > 0; w >>= 1) {
    if (tid < w) part[tid] += part[tid + w];
    __syncthreads();
  }
  const double tot = part[0];
  __syncthreads();
  const float ftot = (float)tot;
  const float one_m = (float)(1.0 - (double)eps);
  acc = 0.0;
  for (int i = tid; i < n; i += T) {
    float p = poly[i];
    if (tot > 0.0) p = __fdiv_rn(p, ftot);
    p = __fadd_rn(eps, __fmul_rn(one_m, p));
    const float vol = __fmul_rn(__fmul_rn(__fsub_rn(box[3 * cap + i], box[i]), __fsub_rn(box[4 * cap + i], box[cap + i])),
                                __fsub_rn(box[5 * cap + i], box[2 * cap + i]));
    const float f = __fmul_rn(p, vol);
    poly[i] = p;
    func[i] = f;
    acc += (double)f;
  }
  part[tid] = acc;
  __syncthreads();
  for (int w = T / 2; w > 0; w >>= 1) {
    if (tid < w) part[tid] += part[tid + w];
    __syncthreads();
  }
  if (tid == 0) out[1] = (float)part[0];
}

// ---------------------------------------------------------------------------
// indirect boundary (BoundaryIndirect.cpp:38-192, Edge.cpp:146-199)
// ---------------------------------------------------------------------------
// Indirect boundary set-up (SampleBoundarySegmentIndirect, Edge.cpp:146-199,
// BoundaryIndirect.cpp:58-130): edge point and direction in the edge wedge;
// with the hits of the two rays that leave the point along -dir (emitter side)
// and dir (sensor side), the boundary geometry. Both return false for a
// rejected sample.
TRN_D bool indirect_point(const Params& P, long long gslot, EdgePoint& q, int& vhint) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = view_of(P, gslot, vhint);
  q.V = &V;
  q.p = gslot - V.begin;
  if (V.D < 2) return false;
  const PathSmp S{&P, V.seed, gslot, q.p + V.slot_off};
  const float r0 = S(0), r1 = S(1), r2 = S(2);
  float reuse;
  const float integral = __ldg(P.eint);
  if (!(integral > 0.f)) return false;
  const int e = sample_discrete(P.ecdf, P.ne, r0, reuse);
  const int f0 = P.edges[5 * e + 2], f1 = P.edges[5 * e + 3], v2 = P.edges[5 * e + 4];
  q.v0 = P.edges[5 * e]; q.v1 = P.edges[5 * e + 1];
  const float len_e = P.efunc[e];
  if (!(len_e > 0.f)) return false;
  const float pdf_e = (len_e / (integral * (float)P.ne)) / len_e;
  const F3 Pa = load3(s.pos, q.v0), Pb = load3(s.pos, q.v1), Pc = load3(s.pos, v2);
  const F3 e1 = Pb - Pa;
  q.s = reuse;
  q.p0 = Pa + e1 * reuse;
  q.edge = normalize(e1); q.edge2 = normalize(Pc - Pa);
  const F3 n0 = load3(s.fnormal, f0);
  float pdf_d;
  if (f1 < 0) {
    const F3 nrm = cross(n0, q.edge);
    F3 tg, bt; coordinate_system(nrm, tg, bt);
    const float z = fminf(1.f - 2.f * r1, 1.f - kEdgeEps);
    const float r = sqrtf(fmaxf(0.f, 1.f - z * z));
    const float phi = 2.f * kPi * r2;
    float sp, cp;
    sincos_det(phi, sp, cp);
    q.dir = tg * (r * cp) + bt * (r * sp) + nrm * z;
    pdf_d = 0.25f / kPi;
  } else {
    const F3 n1 = load3(s.fnormal, f1);
    const float phi0 = acos_det(dot(n0, n1));
    pdf_d = 0.25f / phi0;
    const F3 zz = normalize(n0 + n1);
    const F3 yy = normalize(cross(n0, zz));
    const F3 xx = cross(yy, zz);
    float phi = (r1 - 0.5f) * phi0;
    phi = fminf(fmaxf(phi, -0.5f * phi0 + kEdgeEps), 0.5f * phi0 - kEdgeEps);
    float sp, cp;
    sincos_det(phi, sp, cp);
    const F3 x1 = xx * cp + zz * sp;
    const bool m0 = r2 > 0.5f;
    const float bq = 4.f * r2 - (m0 ? 3.f : 1.f);
    const float aq = sqrtf(1.f - bq * bq) * (1.f - (m0 ? 1.f : 0.f) * 2.f);
    q.dir = x1 * aq + yy * bq;
  }
  q.pdf = pdf_e * pdf_d;
  return true;
}

// he: emitter-side hit, hs: sensor-side hit.
TRN_D bool indirect_finish(const Params& P, long long gslot, const EdgePoint& q, const Hit& he, const Hit& hs,
                           EdgeState& st) {
  const DeviceScene& s = P.s;
  const SurfF xe = post_intersect(s, he.tri, he.u, he.v);
  const SurfF xs = post_intersect(s, hs.tri, hs.u, hs.v);
  const float dl = length(xe.p - xs.p);
  const float cos2 = fabsf(dot(xe.ng, q.dir));
  const float its_t = length(xs.p - q.p0);
  F3 n;
  const float bval = base_val(its_t / dl, q.edge, -q.dir, xe.ng, q.edge2, n) * cos2;
  if (bval == 0.f) return false;
  st.V = q.V; st.gslot = gslot; st.p = q.p; st.x = xs; st.xe = xe; st.rdir = q.dir; st.p0 = q.p0; st.n = n;
  st.w0 = bval / q.pdf; st.sedge = q.s; st.v0 = q.v0; st.v1 = q.v1; st.far_tri = he.tri;
  return true;
}

TRN_D bool indirect_setup(const Params& P, long long gslot, EdgeState& st, int& vhint, Cnt& cnt) {
  EdgePoint q;
  if (!indirect_point(P, gslot, q, vhint)) return false;
  Hit he, hs;
  cnt.v[kCntClosest] += 2;
  if (!trace_shared<false>(P.s, q.p0, -q.dir, kShadowEps, kRayMax, he, P.err)) return false;
  if (!trace_shared<false>(P.s, q.p0, q.dir, kShadowEps, kRayMax, hs, P.err)) return false;
  return indirect_finish(P, gslot, q, he, hs, st);
}

// Indirect boundary sensor side (BoundaryIndirect.cpp:158-175 pairs sensor
// depth b with the emitter radiance accumulated over D-1-b bounces): the
// importance contributions of every depth, weighted by dL/dI of their pixels.
// Returns the shallowest depth that reached the image with a nonzero weight
// (D when none did).
template <int MAXD>
TRN_D int indirect_sensor(const Params& P, const EdgeState& st, int D, F3* sc, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const ViewDesc& V = *st.V;
  const PathSmp S{&P, V.seed, st.gslot, st.p + V.slot_off};
  int bmin = D;
  F3 T(1.f, 1.f, 1.f);
  F3 rd = st.rdir;
  SurfF xx = st.x;
  for (int b = 0; b < D - 1; b++) sc[b] = F3z();
  for (int b = 0; b < D - 1; b++) {
    const int o = 3 + 5 * (D - 1) + 3 * b;
    F3 c; int pix;
    const bool more = importance_step_shared(s, V.cam, xx, rd, T, S(o), S(o + 1), S(o + 2), c, pix, cnt);
    if (pix >= 0) {
      sc[b] = g_at(P, V, pix) * c;
      if (sc[b].x != 0.f || sc[b].y != 0.f || sc[b].z != 0.f) bmin = min(bmin, b);
    }
    if (!more) break;
  }
  return bmin;
}

// Indirect boundary emitter side: the radiance accumulated over j+1 bounces
// from the emitter-side surface pairs with sensor depth D-2-j; returns the
// weight W of the xDotN scatter.
template <int MAXD>
TRN_D float indirect_emitter(const Params& P, const ViewDesc& V, long long gslot, long long p, const SurfF& xe,
                             const F3& rdir, float w0, int D, int jmax, const F3* sc, Cnt& cnt) {
  const DeviceScene& s = P.s;
  const PathSmp S{&P, V.seed, gslot, p + V.slot_off};
  float W = 0.f;
  F3 T(1.f, 1.f, 1.f);
  F3 rd = -rdir;
  SurfF xx = xe;
  F3 cur = F3z();
  bool alive = true;
  for (int j = 0; j <= jmax; j++) {
    if (alive) {
      const int o = 3 + 5 * j;
      F3 c;
      alive = radiance_step_shared(s, xx, rd, T, S(o), S(o + 1), S(o + 2), S(o + 3), S(o + 4), c, nullptr, cnt);
      cur = cur + c;
      if (T.x == 0.f && T.y == 0.f && T.z == 0.f) alive = false;
    }
    W += dot(sc[D - 2 - j], cur) * w0;
  }
  return W;
}

template <int MAXD>
__global__ void __launch_bounds__(256, TRN_MINB) k_indirect_adj(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<EdgeState>(P,
    [&](long long gslot, EdgeState& st) -> bool { return indirect_setup(P, gslot, st, vhint, cnt); },
    [&](EdgeState& st) {
      const ViewDesc& V = *st.V;
      const int D = min(V.D, MAXD);
      // sensor side first; the emitter side then only runs as deep as the
      // shallowest sensor depth that reached the image needs, and not at all
      // when none did
      F3 sc[MAXD];
      const int bmin = indirect_sensor<MAXD>(P, st, D, sc, cnt);
      if (bmin >= D - 1) return;
      const float W = indirect_emitter<MAXD>(P, V, st.gslot, st.p, st.xe, st.rdir, st.w0, D, D - 2 - bmin, sc, cnt);
      if (W == 0.f || !isfinite(W)) return;
      xdotn_vjp(P, V, W, st.x.p, true, st.x.tri, st.x.u, st.x.v, st.v0, st.v1, st.sedge, st.p0, st.far_tri, st.n,
                cnt);
    });
  flush_cnt(cnt, P.stats);
}

// A sample that passed the indirect set-up; its sensor side, emitter side and
// scatter follow.
struct IndirectItem {
  unsigned p_lo;  // view-local sample index in two halves: 92 bytes without padding
  int p_hi;
  int view, xe_tri, xs_tri, v0, v1, far_tri;
  float xe_u, xe_v, xs_u, xs_v, w0, sedge;
  F3 rdir, p0, n;
  TRN_D long long p() const { return (long long)p_hi << 32 | p_lo; }
};

// Sort keys of one round of a split boundary set-up: view x (E + 1) + the
// edge that the slot's edge sample picks (E when it picks none), value = the
// slot's offset in the round. Run in key order, a warp's rays leave one edge
// (or a few neighbours) instead of 32 random ones; each slot's own result is
// unchanged, only the order of the gradient atomics moves.
// The edge pick restates the set-up functions' first step: primary_setup
// (view silhouette table), direct_setup (scene table, or the AQ leaf when
// guided), indirect_setup (scene table).
// bits_r1 + bits_r2 > 0 (indirect term) appends a direction bin below the
// edge: the set-up rays of one edge leave one point, and sorting them by the
// two samples that pick their direction (Edge.cpp:152-195) puts rays that
// head the same way into one warp. r2 is the major part: it picks the
// quadrant and the angle along the edge (or the azimuth of a boundary edge);
// r1 sweeps the wedge between the face normals, which is narrow on a smooth
// mesh (or the polar angle of a boundary edge).
__global__ void k_edge_keys(TRN_KPARAMS, int term, int bits_r1, int bits_r2, unsigned* keys, unsigned* vals) {
  const long long first = P.order_first, n = P.total - first;
  int vhint = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long g = first + i;
    const ViewDesc& V = view_of(P, g, vhint);
    const PathSmp S{&P, V.seed, g, g - V.begin + V.slot_off};
    int e = P.ne;
    float reuse;
    if (term == TRN_PRIMARY_EDGE) {
      if (__ldg(V.pint) > 0.f) e = sample_discrete(V.pcdf, P.ne, S(0), reuse);
    } else if (__ldg(P.eint) > 0.f && (term != TRN_INDIRECT_EDGE || V.D >= 2)) {
      if (term == TRN_DIRECT_EDGE && P.aq_cdf)
        e = __ldg(P.aq_edge + sample_discrete(P.aq_cdf, __ldg(P.aq_n), S(3 + 3 * V.D), reuse));
      else
        e = sample_discrete(P.ecdf, P.ne, S(0), reuse);
    }
    unsigned key = (unsigned)(&V - P.views) * (unsigned)(P.ne + 1) + (unsigned)e;
    if (bits_r1 + bits_r2 > 0) {
      const unsigned b1 = min((unsigned)(S(1) * (float)(1 << bits_r1)), (1u << bits_r1) - 1u);
      const unsigned b2 = min((unsigned)(S(2) * (float)(1 << bits_r2)), (1u << bits_r2) - 1u);
      key = (key << (bits_r1 + bits_r2)) | (b2 << bits_r1) | b1;
    }
    keys[i] = key;
    vals[i] = (unsigned)i;
  }
}


// ---------------------------------------------------------------------------
// pixel boundary (BoundaryPixel.cpp:36-159, Edge.cpp:377-409, Camera.cpp:433-467)
// ---------------------------------------------------------------------------
// Pixel boundary set-up (SampleBoundarySegmentPixel, Edge.cpp:377-409;
// GeneratePixelBoundarySamples, Camera.cpp:433-467): a point on the pixel's
// boundary from the antithetic copy's sample and the camera ray through it;
// with that ray's hit, the boundary geometry.
struct PixelPoint {
  const ViewDesc* V;
  long long slot;     // of the view's slots, shared by the 4 antithetic copies
  int pixel;
  float pdf;
  F3 p0, dir, edge, edge2;
};

TRN_D void pixel_point(const Params& P, long long gslot, PixelPoint& q, int& vhint) {
  const ViewDesc& V = view_of(P, gslot, vhint);
  q.V = &V;
  const CameraDesc& cam = V.cam;
  const int W_ = cam.w, WH = cam.w * cam.h;
  const long long nanti = V.n / 4;
  // Run order: the 4 antithetic copies of a slot take adjacent lanes. Their
  // camera rays leave one pixel's border and share every later sample, so
  // their paths stay close together (coherent traversal). Sample index p
  // (copy * nanti + slot) and everything derived from it do not depend on it.
  const long long i = gslot - V.begin;
  const long long p = (i & 3) * nanti + (i >> 2);
  q.slot = p % nanti;
  const int anti = (int)(p / nanti);
  // the 4 antithetic copies of a slot share its samples (BoundaryPixel.cpp:135-138)
  const PathSmp S{&P, V.seed, V.begin / 4 + q.slot, q.slot + V.slot_off};
  const float r = S(0);
  float rr;
  if (anti == 0) rr = r;
  else if (anti == 1) rr = r < 0.5f ? r + 0.5f : r - 0.5f;
  else if (anti == 2) rr = r < 0.75f ? 0.75f - r : 1.75f - r;
  else rr = r < 0.25f ? 0.25f - r : 1.25f - r;
  const float r4 = rr * 4.f;
  const int bi = (int)floorf(r4);
  float ox, oy;
  if (bi == 0) { ox = 0.f; oy = r4; }
  else if (bi == 1) { ox = r4 - 1.f; oy = 1.f; }
  else if (bi == 2) { ox = 1.f; oy = 3.f - r4; }
  else { ox = 4.f - r4; oy = 0.f; }
  const int bsel = bi < 0 ? 0 : (bi > 3 ? 3 : bi);
  q.pdf = (bsel & 1) ? 0.25f / (cam.plane_len_x * (float)cam.h) : 0.25f / (cam.plane_len_y * (float)cam.w);
  const F3 dedge = (bsel & 1) ? F3(1.f, 0.f, 0.f) : F3(0.f, 1.f, 0.f);
  const F3 dvis = bsel == 0 ? F3(1.f, 0.f, 0.f) : (bsel == 1 ? F3(0.f, -1.f, 0.f)
                                                : (bsel == 2 ? F3(-1.f, 0.f, 0.f) : F3(0.f, 1.f, 0.f)));
  q.edge = normalize(xform_vector(cam.raster_to_world, dedge));
  q.edge2 = normalize(xform_vector(cam.raster_to_world, dvis));
  q.pixel = (int)(p % WH);
  q.p0 = xform_point(cam.raster_to_world, F3((float)(q.pixel % W_) + ox, (float)(q.pixel / W_) + oy, 0.f));
  q.dir = normalize(q.p0 - cam_pos(cam));
}

TRN_D bool pixel_finish(const Params& P, const PixelPoint& q, const Hit& h, EdgeState& st) {
  const ViewDesc& V = *q.V;
  const CameraDesc& cam = V.cam;
  const F3 cpos = cam_pos(cam);
  const F3 hitP = q.p0 + q.dir * h.t;
  const SensorSample sds = sample_direct(cam, hitP);
  const F3 dirc = sensor_ray_dir(cam, sds.qx, sds.qy);
  const SurfF x = post_intersect(P.s, h.tri, h.u, h.v);
  const float dist = length(x.p - cpos);
  const float dist1 = length(q.p0 - cpos);
  const float cos2 = fabsf(dot(x.ng, -dirc));
  F3 n;
  // BoundaryPixel.cpp:92 reverses the sign convention
  const float bval = -base_val(dist / dist1, q.edge, dirc, x.ng, q.edge2, n) * cos2;
  const F3 g = g_at(P, V, q.pixel);
  if (bval == 0.f || (g.x == 0.f && g.y == 0.f && g.z == 0.f)) return false;
  st.V = &V; st.gslot = V.begin / 4 + q.slot; st.p = q.slot; st.x = x; st.rdir = dirc;
  st.T0 = F3(sds.sensor_val, sds.sensor_val, sds.sensor_val);
  st.p0 = q.p0; st.n = n; st.w0 = bval / q.pdf; st.far_tri = h.tri; st.g = g;
  return true;
}

TRN_D bool pixel_setup(const Params& P, long long gslot, EdgeState& st, int& vhint, Cnt& cnt) {
  PixelPoint q;
  pixel_point(P, gslot, q, vhint);
  Hit h;
  cnt.v[kCntClosest]++;
  if (!trace<false>(P.s, q.p0, q.dir, kShadowEps, kRayMax, h, P.err)) return false;
  return pixel_finish(P, q, h, st);
}

__global__ void __launch_bounds__(256, TRN_MINB) k_pixel_adj(TRN_KPARAMS) {
  Cnt cnt;
  int vhint = 0;
  for_each_valid<EdgeState>(P,
    [&](long long gslot, EdgeState& st) -> bool { return pixel_setup(P, gslot, st, vhint, cnt); },
    [&](EdgeState& st) {
      // the pixel-edge point is not a scene parameter: only the hit triangle moves
      primary_body(P, *st.V, st.gslot, st.p, st.x, st.rdir, st.T0, st.w0, st.g, -1, -1, 0.f, st.p0, st.far_tri,
                   st.n, cnt, 1);
    });
  flush_cnt(cnt, P.stats);
}

// ---------------------------------------------------------------------------
// paths and scatter of the boundary samples that passed their set-up
// ---------------------------------------------------------------------------
// One kernel per side runs a round's samples to their ends, one thread per
// sample, and a lane whose path has ended takes the next sample of the queue at
// once. Each sample scatters when its path ends, together with the lanes of its
// warp that end in the same turn.
//
// Not as a wavefront like the interior term's paths: a few vertices (a ground
// plane's, a light's) get millions of 32-bit adds each, and which small ones are
// lost in the large running sum depends on how many lanes' adds are summed
// before them and on their order. A scatter of 32 queued samples at a time, all
// of one bounce before those of the next, moved nearly cancelling components of
// the 16.8M-sample gradient by 1 to 2 % of its RMS (0.1 % between two runs).
// And few samples pass: 0.5M slots of depth 12 take 0.69, 3.0 and 1.4 ms for
// direct, indirect and pixel here, and 0.92, 3.8 and 1.9 with two launches per
// bounce. The wavefront was ahead for many slots (16.8M of depth 5: primary 11.2
// and here 11.8, direct 2.4 and 2.2, indirect 28.6 and 30.4, pixel 16.0 and
// 18.7).

// Slot of a sample in its launch, which indexes a caller's sample table.
TRN_D long long item_gslot(const Params& P, const ViewDesc& V, long long p) {
  return p + (P.term == TRN_PIXEL_EDGE ? V.begin / 4 : V.begin);
}

// Warp-uniform: hands every lane that wants one the next index of [0, n);
// `done` is set for those that come behind the end.
TRN_D void take_next(unsigned long long* next, unsigned long long n, bool want, unsigned long long& k, bool& done) {
  const unsigned need = __ballot_sync(0xffffffffu, want);
  if (!need) return;
  const int lane = threadIdx.x & 31, leader = __ffs(need) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(next, (unsigned long long)__popc(need));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (want) {
    k = base + __popc(need & ((1u << lane) - 1u));
    done = k >= n;
  }
}

// Primary and pixel terms: detached radiance of the sample, then the scatter.
__global__ void __launch_bounds__(256, TRN_MINB) k_primary_body(TRN_KPARAMS, unsigned long long* next) {
  stage_begin();
  Cnt cnt;
  const DeviceScene& s = P.s;
  const PrimaryItem* q = reinterpret_cast<const PrimaryItem*>(P.queue);
  const unsigned long long n = min(*P.q_count, (unsigned long long)P.q_cap);
  const int dim0 = P.term == TRN_PIXEL_EDGE ? 1 : 2;
  bool active = false, done = false;
  unsigned long long k = 0;
  const ViewDesc* V = nullptr;
  SurfF x;
  F3 T, rdir, L;
  int b = 0, D = 0;
  for (;;) {
    const bool want = !active && !done;
    take_next(next, n, want, k, done);
    if (want && !done) {
      const PrimaryItem& it = q[k];
      V = P.views + it.view;
      D = V->D;
      x = post_intersect(s, it.x_tri, it.x_u, it.x_v);
      T = F3(it.T0, it.T0, it.T0);
      rdir = it.rdir;
      L = scrub(T * emitted(s, x, -rdir));
      b = 0;
      active = true;
    }
    if (!__any_sync(0xffffffffu, active)) break;
    if (active) {
      bool fin = b >= D;
      if (!fin) {
        const long long p = q[k].p;
        const PathSmp S{&P, V->seed, item_gslot(P, *V, p), p + V->slot_off};
        const int o = dim0 + 5 * b;
        F3 c;
        const bool more = radiance_step(s, x, rdir, T, S(o), S(o + 1), S(o + 2), S(o + 3), S(o + 4), c, nullptr, cnt);
        L = L + c;
        b++;
        fin = !more || (T.x == 0.f && T.y == 0.f && T.z == 0.f) || b >= D;
      }
      if (fin) {
        const PrimaryItem& it = q[k];
        const float W = dot(it.g, L * it.w0);
        if (W != 0.f && isfinite(W))
          xdotn_vjp(P, *V, W, cam_pos(V->cam), false, -1, 0.f, 0.f, it.v0, it.v1, it.sedge, it.p0, it.far_tri, it.n,
                    cnt);
        active = false;
      }
    }
  }
  flush_cnt(cnt, P.stats);
}

// Direct term: importance path and scatter. (Few samples pass the set-up, and
// they leave their receiver towards one sensor: no lane waits for long.)
__global__ void __launch_bounds__(256, TRN_MINB) k_direct_body(TRN_KPARAMS) {
  stage_begin();
  Cnt cnt;
  const DirectItem* q = reinterpret_cast<const DirectItem*>(P.queue);
  const unsigned long long n = min(*P.q_count, (unsigned long long)P.q_cap);
  for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < n;
       k += (unsigned long long)gridDim.x * blockDim.x) {
    const DirectItem& it = q[k];
    const ViewDesc& V = P.views[it.view];
    const SurfF x = post_intersect(P.s, it.x_tri, it.x_u, it.x_v);
    direct_body(P, V, item_gslot(P, V, it.p), it.p, x, it.rdir, it.ev0, it.v0, it.v1, it.sedge, it.p0, it.far_tri,
                it.n, cnt);
  }
  flush_cnt(cnt, P.stats);
}

// Indirect term, a sample whose sensor side reached the image: the set-up's
// item, how deep its emitter side has to go, the weight of each sensor depth.
template <int MAXD>
struct IndirectLit {
  unsigned item;
  int jmax;
  F3 sc[MAXD - 1];
};

// Sensor side (the steps of indirect_sensor).
template <int MAXD>
__global__ void __launch_bounds__(256, TRN_MINB) k_indirect_sensor(TRN_KPARAMS, unsigned long long* next,
                                                                   IndirectLit<MAXD>* lit, unsigned long long* n_lit) {
  stage_begin();
  Cnt cnt;
  const DeviceScene& s = P.s;
  const IndirectItem* q = reinterpret_cast<const IndirectItem*>(P.queue);
  const unsigned long long n = min(*P.q_count, (unsigned long long)P.q_cap);
  bool active = false, done = false;
  unsigned long long k = 0;
  const ViewDesc* V = nullptr;
  SurfF x;
  F3 T, rdir;
  F3 sc[MAXD - 1];
  int b = 0, D = 0, bmin = 0;
  for (;;) {
    const bool want = !active && !done;
    take_next(next, n, want, k, done);
    if (want && !done) {
      const IndirectItem& it = q[k];
      V = P.views + it.view;
      D = min(V->D, MAXD);
      x = post_intersect(s, it.xs_tri, it.xs_u, it.xs_v);
      rdir = it.rdir;
      T = F3(1.f, 1.f, 1.f);
      for (int j = 0; j < D - 1; j++) sc[j] = F3z();
      bmin = D;
      b = 0;
      active = true;
    }
    if (!__any_sync(0xffffffffu, active)) break;
    bool fin = false;
    if (active) {
      fin = b >= D - 1;
      if (!fin) {
        const long long p = q[k].p();
        const PathSmp S{&P, V->seed, item_gslot(P, *V, p), p + V->slot_off};
        const int o = 3 + 5 * (D - 1) + 3 * b;
        F3 c;
        int pix;
        const bool more = importance_step(s, V->cam, x, rdir, T, S(o), S(o + 1), S(o + 2), c, pix, cnt);
        if (pix >= 0) {
          sc[b] = g_at(P, *V, pix) * c;
          if (sc[b].x != 0.f || sc[b].y != 0.f || sc[b].z != 0.f) bmin = min(bmin, b);
        }
        b++;
        fin = !more || b >= D - 1;
      }
    }
    const bool push = fin && bmin < D - 1;
    const unsigned m = __ballot_sync(0xffffffffu, push);
    if (m) {
      const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(n_lit, (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (push) {
        IndirectLit<MAXD>& it = lit[base + __popc(m & ((1u << lane) - 1u))];  // at most one per item
        it.item = (unsigned)k;
        it.jmax = D - 2 - bmin;
        for (int j = 0; j < D - 1; j++) it.sc[j] = sc[j];
      }
    }
    if (fin) active = false;
  }
  flush_cnt(cnt, P.stats);
}

// Emitter side of the lit samples (the steps and the additions of
// indirect_emitter: when the path has ended, the remaining depths pair with its
// last radiance), then the scatter.
template <int MAXD>
__global__ void __launch_bounds__(256, TRN_MINB) k_indirect_emitter(TRN_KPARAMS, unsigned long long* next,
                                                                    const IndirectLit<MAXD>* lit,
                                                                    const unsigned long long* n_lit) {
  stage_begin();
  Cnt cnt;
  const DeviceScene& s = P.s;
  const IndirectItem* q = reinterpret_cast<const IndirectItem*>(P.queue);
  const unsigned long long n = *n_lit;
  bool active = false, done = false;
  unsigned long long k = 0;
  const ViewDesc* V = nullptr;
  SurfF x;
  F3 T, rdir, cur;
  float W = 0.f;
  int j = 0;
  for (;;) {
    const bool want = !active && !done;
    take_next(next, n, want, k, done);
    if (want && !done) {
      const IndirectItem& it = q[lit[k].item];
      V = P.views + it.view;
      x = post_intersect(s, it.xe_tri, it.xe_u, it.xe_v);
      rdir = -it.rdir;
      T = F3(1.f, 1.f, 1.f);
      cur = F3z();
      W = 0.f;
      j = 0;
      active = true;
    }
    if (!__any_sync(0xffffffffu, active)) break;
    if (active) {
      const IndirectLit<MAXD>& l = lit[k];
      const IndirectItem& it = q[l.item];
      const int D = min(V->D, MAXD), jmax = l.jmax;
      const long long p = it.p();
      const PathSmp S{&P, V->seed, item_gslot(P, *V, p), p + V->slot_off};
      const int o = 3 + 5 * j;
      F3 c;
      bool alive = radiance_step(s, x, rdir, T, S(o), S(o + 1), S(o + 2), S(o + 3), S(o + 4), c, nullptr, cnt);
      cur = cur + c;
      if (T.x == 0.f && T.y == 0.f && T.z == 0.f) alive = false;
      W += dot(l.sc[D - 2 - j], cur) * it.w0;
      j++;
      if (!alive || j > jmax) {
        for (; j <= jmax; j++) W += dot(l.sc[D - 2 - j], cur) * it.w0;
        if (W != 0.f && isfinite(W)) {
          const SurfF xs = post_intersect(s, it.xs_tri, it.xs_u, it.xs_v);
          xdotn_vjp(P, *V, W, xs.p, true, it.xs_tri, it.xs_u, it.xs_v, it.v0, it.v1, it.sedge, it.p0, it.far_tri,
                    it.n, cnt);
        }
        active = false;
      }
    }
  }
  flush_cnt(cnt, P.stats);
}

#include "wavefront.cuh"

// ---------------------------------------------------------------------------
// primary edge list for one camera (ConstructPrimEdgeList, Edge.cpp:313-348)
// ---------------------------------------------------------------------------
__global__ void k_prim_edges_views(int ne, const int* edges, const float* pos, const float* fn,
                                   const ViewDesc* views, float* func_all) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = blockIdx.y;
  if (e >= ne) return;
  const CameraDesc& c = views[v].cam;
  const F3 cpos(c.pos[0], c.pos[1], c.pos[2]);
  const int v0 = edges[5 * e], v1 = edges[5 * e + 1], f0 = edges[5 * e + 2], f1 = edges[5 * e + 3];
  const F3 p0 = make_f3(pos + 3 * v0);
  const F3 ev = cpos - p0;
  const F3 n0 = make_f3(fn + 3 * f0);
  const F3 n1 = f1 >= 0 ? make_f3(fn + 3 * f1) : F3(0.f, 0.f, 0.f);
  const bool ff0 = dot(ev, n0) > 0.f, ff1 = dot(ev, n1) > 0.f;
  const bool valid = f1 < 0 || (ff0 != ff1);
  func_all[(long long)v * ne + e] = valid ? length(make_f3(pos + 3 * v1) - p0) : 0.f;
}

// 0.5 |I - T|^2 per view and dL/dI = I - T (pyTensorRay/loss.py:34-38)
__global__ void k_view_loss(long long npix, const ViewDesc* views, const long long* pbegin, int nviews,
                            const float* img, const float* tgt, float* dLdI, float* loss) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  float l = 0.f;
  int v = -1;
  if (i < npix) {
    int lo = 0, hi = nviews - 1;
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (pbegin[mid] <= i) lo = mid; else hi = mid - 1; }
    v = lo;
    for (int c = 0; c < 3; c++) {
      const float d = img[3 * i + c] - tgt[3 * i + c];
      if (dLdI) dLdI[3 * i + c] = d;
      l += 0.5f * d * d;
    }
  }
  // warp-aggregate per view
  const unsigned m = __match_any_sync(0xffffffffu, v);
  float sum = 0.f;
  for (int k = 0; k < 32; k++) {
    const float y = __shfl_sync(0xffffffffu, l, k);
    if (m & (1u << k)) sum += y;
  }
  if (v >= 0 && (int)(threadIdx.x & 31) == __ffs(m) - 1 && loss) atomicAdd(loss + v, sum);
}

// Ray queries of a program's own rays. Each warp streams through tiles of
// `chunk` rays, every warp of the grid in turn, so that a run of costly rays (a
// program's rays often come in image order) is spread over all of them. Few
// rays are spread over all warps of the GPU as well, down to one each, since a
// query is then as long as its longest ray (1,000 rays on 7,000 triangles: 56 us
// with four per warp, 46 with one).
template <bool ANY>
__global__ void __launch_bounds__(TRN_TRACE_BLOCK, TRN_TRACE_MINB)
    k_query(const __grid_constant__ DeviceScene s, int n, int chunk, const float* org, const float* dir,
            const float* tmin_, const float* tmax_, int* tri_, float* u_, float* v_, float* t_, int* err) {
  const long long step = (long long)gridDim.x * (blockDim.x >> 5) * chunk;
  long long tile = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * chunk, pos = tile;
  trace_stream(s,
    [&](int k, int& lim, bool& more) {
      const int base = (int)min((long long)n, pos);
      lim = (int)min((long long)n, tile + chunk);
      pos += k;
      if (pos >= lim) pos = tile += step;
      more = pos < n;
      return base;
    },
    [&](int i, F3& o, F3& d, float& tmin, float& tmax, bool& any) {
      o = make_f3(org + 3ll * i); d = make_f3(dir + 3ll * i);
      tmin = tmin_[i]; tmax = tmax_[i]; any = ANY;
    },
    [&](int i, bool, int tri, float u, float v, float t) {
      if (ANY) tri_[i] = tri >= 0 ? 0 : 1;
      else { tri_[i] = tri; u_[i] = u; v_[i] = v; t_[i] = t; }
    }, err);
}

// The same with one ray per thread, for the batches that query_streams() names.
template <bool ANY>
__global__ void __launch_bounds__(128)
    k_query_one(const __grid_constant__ DeviceScene s, int n, const float* org, const float* dir, const float* tmin,
                const float* tmax, int* tri, float* u, float* v, float* t, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Hit h;
  const bool hit = trace<ANY>(s, make_f3(org + 3ll * i), make_f3(dir + 3ll * i), tmin[i], tmax[i], h, err);
  if (ANY) tri[i] = hit ? 0 : 1;
  else { tri[i] = h.tri; u[i] = h.u; v[i] = h.v; t[i] = h.t; }
}

}  // namespace trn

using namespace trn;

// Pinned staging slots of a view set's table uploads. An upload waits only
// for the upload this many before it to have left its slot, so a loop that
// changes its views every call (a serving loop) runs that many uploads ahead
// of the device instead of waiting for the previous call's kernels.
constexpr int kStageRing = 4;

// A set of camera views rendered by one launch per integrator: the device view
// table plus per-view silhouette-edge workspace.
struct trn_viewset {
  trn_scene* scene = nullptr;
  int nviews = 0;
  int cap = 0;                    // allocated view capacity
  // pinned staging of the view table: kStageRing slots of `cap` views and
  // 2 * `cap` offsets (view begins, then pixel begins) each
  ViewDesc* h_stage = nullptr;
  long long* h_stage_begin = nullptr;
  cudaEvent_t stage_done[kStageRing] = {};
  int stage_next = 0;
  bool pbegin_dirty = true;
  long long npix = 0;
  std::vector<trn_view> h_views;
  std::vector<long long> h_pbegin;
  std::vector<long long> h_slots;  // of each view, in the uploaded table
  ViewDesc* views = nullptr;      // device [nviews]
  long long* vbegin = nullptr;    // device [nviews], rewritten per integrator (spp differs)
  long long* pbegin = nullptr;    // device [nviews] first pixel of each view
  float* pfunc = nullptr;         // device [nviews][E]
  float* pcdf = nullptr;          // device [nviews][E]
  float* pint = nullptr;          // device [nviews]
  double* pint_part = nullptr;    // device [nviews][kCdfChunks]
  unsigned long long* work = nullptr;
  // buffers of one wavefront round (items, rays, path state) and its counters
  void* iq = nullptr;
  size_t iq_bytes = 0;
  unsigned long long* iq_count = nullptr;
  // A captured launch holds the addresses of iq and sq: from then on a growth
  // keeps the old buffer until the set is destroyed (one per capture and growth
  // at most; none is above a full round, 3.4 GB and 0.3 GB at depth <= 8).
  bool iq_captured = false, sq_captured = false;
  std::vector<void*> kept;
  // run order of the split set-up rounds: keys and values double-buffered for
  // one round, then the radix sort's temporary storage
  void* sq = nullptr;
  long long sq_cap = 0;  // slots per round the order buffers hold
  size_t sq_tmp = 0;     // bytes of the sort's temporary storage
  // path cache: interior path records of the last forward render, reused by
  // the gradient call of the same paths (same scene version, views, seed and
  // depth; hash samples only)
  void* pc = nullptr;
  size_t pc_bytes = 0;
  unsigned long long* pc_count = nullptr;  // [2] records, paths ended
  long long pc_limit = 0;  // bytes the records may take (0 = off)
  bool pc_valid = false;
  std::vector<char> pc_key;
  int ne = 0;
  // slot layout currently uploaded: spp multiplier and per-view spp
  int uploaded_key = -2;
  long long total = 0;
  // image / dL/dI base buffers of the uploaded table (views without their own)
  int cur_depth = -1;
  int max_depth = kMaxDepth;
};

namespace {

int sms() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

int check_common(trn_scene* s, const trn_render_options* o, int integrator) {
  if (!s || !o) { set_error("null argument"); return -1; }
  if (!s->configured) { set_error("scene is not configured (call trn_scene_configure)"); return -1; }
  if (integrator < 0 || integrator > 4) { set_error("unknown integrator id"); return -1; }
  if (o->max_bounces < 0 || o->max_bounces > kMaxDepth) { set_error("max_bounces must be in [0, 16]"); return -1; }
  return 0;
}

int spp_of(const trn_render_options* o, int integrator) {
  switch (integrator) {
    case TRN_PATH_TRACER: return o->spp;
    case TRN_PRIMARY_EDGE: return o->sppe;
    case TRN_DIRECT_EDGE: return o->sppse0;
    case TRN_INDIRECT_EDGE: return o->sppse1;
    default: return o->sppe0;
  }
}

// Upload the view table for one integrator: per-view spp comes from the view
// (spp_override < 0) or from the options (single-view calls).
// The next staging slot, once the upload that last used it has left it.
int next_stage(trn_viewset* vs) {
  const int k = vs->stage_next;
  vs->stage_next = (k + 1) % kStageRing;
  if (vs->stage_done[k]) cudaEventSynchronize(vs->stage_done[k]);
  return k;
}

// Every staging slot free (before the staging is freed or reallocated).
void wait_stages(trn_viewset* vs) {
  for (cudaEvent_t e : vs->stage_done)
    if (e) cudaEventSynchronize(e);
}

int upload_views(trn_viewset* vs, const trn_render_options* o, int integrator, int spp_override, long long& total,
                 cudaStream_t st) {
  (void)o;
  float* s_gpos = vs->scene->g_pos;
  float* s_gvn = vs->scene->g_vnormal;
  float* s_gtex = vs->scene->g_texels;
  const int key = spp_override;  // the layout depends on the per-view spp, buffers and depth
  if (vs->uploaded_key == key && key != -2 && vs->cur_depth == o->max_bounces) {
    total = vs->total;
    if (integrator == TRN_PIXEL_EDGE)
      for (int v = 0; v < vs->nviews; v++) {
        const int spp = spp_override >= 0 ? spp_override : vs->h_views[v].spp;
        if (((long long)vs->h_views[v].camera.width * vs->h_views[v].camera.height * spp) % 4 != 0) {
          set_error("pixel boundary needs W*H*spp divisible by 4");
          return -1;
        }
      }
    return 0;
  }
  vs->cur_depth = o->max_bounces;
  vs->max_depth = 0;
  for (int v = 0; v < vs->nviews; v++)
    vs->max_depth = std::max(vs->max_depth, vs->h_views[v].max_bounces > 0 ? vs->h_views[v].max_bounces
                                                                            : o->max_bounces);
  const int slot = next_stage(vs);
  ViewDesc* d = vs->h_stage + (size_t)slot * vs->cap;
  long long* begin = vs->h_stage_begin + (size_t)slot * 2 * vs->cap;
  total = 0;
  vs->h_slots.assign(vs->nviews, 0);
  for (int v = 0; v < vs->nviews; v++) {
    const trn_view& hv = vs->h_views[v];
    const int spp = spp_override >= 0 ? spp_override : hv.spp;
    if (spp < 0) { set_error("negative spp"); return -1; }
    std::memcpy(&d[v].cam, &hv.camera, sizeof(CameraDesc));
    d[v].begin = total;
    d[v].n = (long long)hv.camera.width * hv.camera.height * spp;
    if (integrator == TRN_PIXEL_EDGE && (d[v].n % 4) != 0) {
      set_error("pixel boundary needs W*H*spp divisible by 4");
      return -1;
    }
    d[v].pix_off = vs->h_pbegin[v];
    d[v].inv_spp = hv.weight > 0.f ? hv.weight : (spp > 0 ? 1.0f / (float)spp : 0.f);
    d[v].slot_off = hv.slot_offset;
    d[v].D = hv.max_bounces > 0 ? std::min(hv.max_bounces, (int)kMaxDepth) : o->max_bounces;
    d[v].image = hv.image;
    d[v].dLdI = hv.dLdI;
    d[v].gpos = hv.grad_positions ? hv.grad_positions : s_gpos;
    d[v].gvn = hv.grad_vertex_normals ? hv.grad_vertex_normals : s_gvn;
    d[v].gtex = hv.grad_texels ? hv.grad_texels : s_gtex;
    d[v].seed = (uint32_t)hv.seed;  // independent of the view's position in the set
    d[v].spp = spp;
    d[v].pad_ = 0;
    d[v].pfunc = vs->pfunc ? vs->pfunc + (long long)v * vs->ne : nullptr;
    d[v].pcdf = vs->pcdf ? vs->pcdf + (long long)v * vs->ne : nullptr;
    d[v].pint = vs->pint ? vs->pint + v : nullptr;
    begin[v] = total;
    vs->h_slots[v] = d[v].n;
    total += d[v].n;
  }
  TRN_CUDA_TRY(cudaMemcpyAsync(vs->views, d, sizeof(ViewDesc) * vs->nviews, cudaMemcpyHostToDevice, st));
  TRN_CUDA_TRY(cudaMemcpyAsync(vs->vbegin, begin, sizeof(long long) * vs->nviews, cudaMemcpyHostToDevice, st));
  TRN_CUDA_TRY(cudaEventRecord(vs->stage_done[slot], st));
  vs->uploaded_key = key;
  vs->total = total;
  return 0;
}

Params base_params(trn_scene* s, trn_viewset* vs, const trn_render_options* o, int integrator,
                   const trn_samples* smp, const trn_launch* ln, long long total) {
  Params P;
  P.s = s->view();
  P.views = vs->views;
  P.vbegin = vs->vbegin;
  P.nviews = vs->nviews;
  P.total = total;
  P.work = vs->work;
  P.chunk = (ln && ln->chunk > 0) ? ln->chunk : 1;
  P.table = smp ? smp->samples : nullptr;
  P.stride = smp && smp->samples ? smp->stride : 0;
  P.term = (uint32_t)integrator;
  P.seed = (uint32_t)o->seed;
  P.D = o->max_bounces;
  P.g_pos = s->g_pos; P.g_vn = s->g_vnormal; P.g_tex = s->g_texels; P.diff_tex = s->ntexel > 0;
  P.edges = s->edges; P.ecdf = s->sec_cdf; P.efunc = s->sec_func; P.eint = s->sec_integral_dev; P.ne = s->ne;
  P.err = s->err;
  P.stats = s->stats_on ? s->stats : nullptr;
  P.aq_poly = P.aq_cdf = P.aq_int = nullptr;
  P.aq_box = nullptr;
  P.aq_edge = P.aq_n = nullptr;
  P.aq_cap = 0;
  P.queue = nullptr;
  P.q_count = nullptr;
  P.q_cap = 0;
  P.order = nullptr;
  P.order_first = 0;
  return P;
}

// Grow the guiding tree's arrays to `cap` leaves (the first refining call, or
// a larger g_direct_max_size); the depth-0 arrays are allocated with the scene.
int aq_reserve(trn_scene* s, long long cap) {
  if (cap <= s->aq_cap && s->aq_eval) return 0;
  cap = std::max(cap, s->aq_cap);
  float* f[4] = {nullptr, nullptr, nullptr, nullptr};
  int* i3[3] = {nullptr, nullptr, nullptr};
  float* eval = nullptr;
  const size_t n = (size_t)cap;
  bool ok = cudaMalloc(&f[0], n * sizeof(float)) == cudaSuccess && cudaMalloc(&f[1], n * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&f[2], n * sizeof(float)) == cudaSuccess && cudaMalloc(&f[3], 6 * n * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&i3[0], n * sizeof(int)) == cudaSuccess && cudaMalloc(&i3[1], n * sizeof(int)) == cudaSuccess &&
            cudaMalloc(&i3[2], n * sizeof(int)) == cudaSuccess &&
            cudaMalloc(&eval, (size_t)kAqPoints * n * sizeof(float)) == cudaSuccess;
  if (!ok) {
    for (float* p : f) if (p) cudaFree(p);
    for (int* p : i3) if (p) cudaFree(p);
    if (eval) cudaFree(eval);
    cudaGetLastError();
    set_error("guiding: cannot allocate the refined tree (g_direct_max_size leaves)");
    return -1;
  }
  void* old[] = {s->aq_poly, s->aq_func, s->aq_cdf, s->aq_box, s->aq_edge, s->aq_flag, s->aq_prefix, s->aq_eval};
  for (void* p : old) {
    if (p && s->aq_captured) s->aq_kept.push_back(p);
    else if (p) cudaFree(p);
  }
  s->aq_captured = false;
  s->aq_poly = f[0]; s->aq_func = f[1]; s->aq_cdf = f[2]; s->aq_box = f[3];
  s->aq_edge = i3[0]; s->aq_flag = i3[1]; s->aq_prefix = i3[2]; s->aq_eval = eval;
  s->aq_cap = cap;
  return 0;
}

void launch_dims(const trn_launch* ln, long long total, int& grid, int& block) {
  block = (ln && ln->block > 0) ? ln->block : 128;
  const int per_sm = (ln && ln->blocks_per_sm > 0) ? ln->blocks_per_sm : 1024 / block;
  const long long chunk = (ln && ln->chunk > 0) ? ln->chunk : 1;
  long long want = (long long)sms() * per_sm;
  const long long need = (total + 32 * chunk - 1) / (32 * chunk) * 32 / block + 1;
  grid = (int)std::max<long long>(1, std::min(want, need));
}

// Whether a query of n rays runs as a stream. A stream wins where most lanes
// would idle (few rays: one per warp) and where rays are many (its warps refill).
// In between, some warps hold several rays from the start and none is refilled
// for long: a lone long ray decides, and its box step takes a fifth longer in the
// stream. That holds longer in a large tree, whose longest rays are ten times the
// mean (324 nodes against 32 on 102,400 triangles; 70 against 20 on 1,284).
// One ray per thread against the stream, closest hit / occlusion in us:
//   triangles        16,000 rays         32,000             128,000            300,000            600,000
//     1,284     48/42 and 39/37     49/44 and 48/45    65/56 and 60/55  123/107 and 102/91  220/183 and 179/156
//     7,000     84/76 and 80/70     88/81 and 93/87  114/99 and 121/103 205/181 and 177/160 349/285 and 258/231
//   102,400   121/101 and 122/102 208/195 and 251/242 262/191 and 314/222 318/258 and 322/242 528/432 and 472/456
//   200,000   136/120 and 131/129 138/125 and 154/133 267/233 and 297/253 343/284 and 428/327 545/440 and 456/357
bool query_streams(int n, int triangles) {
  const int lanes = sms() * TRN_TRACE_MINB * TRN_TRACE_BLOCK;
  return n < lanes / 8 || n >= (triangles > 32768 ? lanes * 5 / 2 : lanes * 3 / 2);
}

// Rays per tile of a stream: as few as give every warp that fits the GPU one
// tile, up to 32.
void query_dims(int n, int& grid, int& chunk) {
  const long long blocks = (long long)sms() * TRN_TRACE_MINB, warps = blocks * (TRN_TRACE_BLOCK / 32);
  chunk = (int)std::min<long long>(32, std::max<long long>(1, (n + warps - 1) / warps));
  const long long per_block = (long long)chunk * (TRN_TRACE_BLOCK / 32);
  grid = (int)std::min(blocks, (n + per_block - 1) / per_block);
}

int validate_launch(const trn_launch* ln) {
  if (!ln) return 0;
  if (ln->block != 0 && (ln->block < 32 || ln->block > 256 || ln->block % 32 != 0)) {
    set_error("launch block must be a multiple of 32 in [32, 256]");
    return -1;
  }
  if (ln->blocks_per_sm < 0 || ln->blocks_per_sm > 64 || ln->chunk < 0 || ln->chunk > 64) {
    set_error("launch blocks_per_sm must be in [0, 64] and chunk in [0, 64]");
    return -1;
  }
  if (ln->round_log2 != 0 && (ln->round_log2 < 16 || ln->round_log2 > 40)) {
    set_error("launch round_log2 must be 0 (default) or in [16, 40]");
    return -1;
  }
  return 0;
}

template <class K>
void launch(K kernel, const trn_launch* ln, long long total, const Params& P, cudaStream_t st) {
  int grid, block;
  launch_dims(ln, total, grid, block);
  kernel<<<grid, block, 0, st>>>(P);
  count_launch(1);
}

// Slots per round of the boundary terms and the image, and paths per round of
// the replaying adjoint. Larger rounds give each edge more samples per sort and
// the terms fewer kernel tails, at up to 205 bytes per slot (direct term; an image
// 181): 16.8M samples of depth 5 on 102,400 triangles, image 16.8 ms in rounds of
// 2^22, 15.3 of 2^23, 14.6 of 2^24. The replay keeps 2^22, where it takes as long as
// with 2^24 (0.74 kB of records and state per path at depth 8).
#ifndef TRN_ROUND_LOG2
#define TRN_ROUND_LOG2 24
#endif
#ifndef TRN_PATH_ROUND_LOG2
#define TRN_PATH_ROUND_LOG2 22
#endif
constexpr long long kRound = 1LL << TRN_ROUND_LOG2;
constexpr long long kReplayRound = 1LL << TRN_PATH_ROUND_LOG2;
constexpr int kWaveCounters = 256;
#ifndef TRN_TAIL_LOG2
#define TRN_TAIL_LOG2 17
#endif

// Slots (or paths) per round: the launch's round_log2 when set, never above
// the default that the buffers are sized for.
long long round_cap(const trn_launch* ln, long long dflt) {
  if (ln && ln->round_log2 > 0) return std::min(dflt, 1LL << ln->round_log2);
  return dflt;
}

size_t item_bytes(int integrator) {
  switch (integrator) {
    case TRN_PATH_TRACER: return 0;
    case TRN_DIRECT_EDGE: return sizeof(DirectItem);
    case TRN_INDIRECT_EDGE: return sizeof(IndirectItem);
    default: return sizeof(PrimaryItem);
  }
}

// Places a round's buffers for `cap` samples from `base` on (the term's items
// first) and returns the bytes they take.
size_t wave_layout(Wave& W, void** items, void* base, long long cap, int integrator, int depth) {
  char* c = static_cast<char*>(base);
  size_t off = 0;
  const size_t n = (size_t)cap;
  auto take = [&](size_t bytes) { char* r = c + off; off += (bytes + 255) / 256 * 256; return static_cast<void*>(r); };
  const bool edge = integrator != TRN_PATH_TRACER;
  *items = take(item_bytes(integrator) * n);
  W.cap = cap;
  const size_t setup = off;
  W.ro = static_cast<float4*>(take(2 * n * sizeof(float4)));
  W.rd = static_cast<float4*>(take(2 * n * sizeof(float4)));
  for (float4*& h : W.hit) h = static_cast<float4*>(take(edge || &h == W.hit ? n * sizeof(float4) : 0));
  W.occ = static_cast<unsigned char*>(take(n));
  W.list[0] = static_cast<unsigned*>(take(n * sizeof(unsigned)));
  W.list[1] = static_cast<unsigned*>(take(n * sizeof(unsigned)));
  W.W = static_cast<float*>(take(integrator == TRN_DIRECT_EDGE ? n * sizeof(float) : 0));
  if (!edge) {
    for (float4*& s : W.st) s = static_cast<float4*>(take(n * sizeof(float4)));
    W.p = static_cast<long long*>(take(n * sizeof(long long)));
    W.view = static_cast<int*>(take(n * sizeof(int)));
    W.rec = static_cast<unsigned*>(take(n * sizeof(unsigned)));
    W.L = static_cast<F3*>(take(n * sizeof(F3)));
  }
  if (integrator == TRN_INDIRECT_EDGE) {  // in the place of the set-up's buffers, which are done with by then
    const size_t end = off;
    off = setup;
    W.lit = take((depth <= 8 ? sizeof(IndirectLit<8>) : sizeof(IndirectLit<kMaxDepth>)) * n);
    off = std::max(off, end);
  }
  return off;
}

// Bytes of the interior term's round: wavefront buffers and, for the replaying
// adjoint, its records.
size_t path_round_bytes(long long cap, int depth, bool records) {
  Wave W;
  PathSoA R;
  void* items;
  return wave_layout(W, &items, nullptr, cap, TRN_PATH_TRACER, depth) + (records ? path_soa(R, nullptr, cap, depth) : 0);
}

// Largest round any term needs (depth <= 8 when shallow, else up to kMaxDepth).
size_t full_queue_bytes(bool shallow) {
  const int depth = shallow ? 8 : kMaxDepth;
  size_t most = std::max(path_round_bytes(kReplayRound, depth, true), path_round_bytes(kRound, depth, false));
  for (int t = 1; t < 5; t++) {
    Wave W;
    void* items;
    most = std::max(most, wave_layout(W, &items, nullptr, kRound, t, depth));
  }
  return most;
}

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
}

// The view set's round buffers, grown on first use to at least `need` bytes
// (not inside stream capture: run the integrator once before capturing it, or
// reserve with trn_viewset_reserve). A growth at least doubles them, up to `most`
// (one full round), so that a set whose batches grow (a serving loop) reallocates a
// few times at most. Returns 1, with the error text set, when the call cannot
// have them: inside a capture, or out of memory.
int ensure_queue(trn_viewset* vs, size_t need, size_t most, cudaStream_t st) {
  const bool cap = capturing(st);
  if (vs->iq_bytes >= need && vs->iq_count) {
    vs->iq_captured |= cap;
    return 0;
  }
  if (cap) {
    set_error("round buffers must be allocated before stream capture (run the call once first, or reserve them)");
    return 1;
  }
  TRN_CUDA_TRY(cudaStreamSynchronize(st));
  if (vs->iq_bytes < need) {
    const size_t bytes = std::max(need, std::min(2 * vs->iq_bytes, most));
    if (vs->iq && vs->iq_captured) vs->kept.push_back(vs->iq);
    else if (vs->iq) cudaFree(vs->iq);
    vs->iq_captured = false;
    vs->iq = nullptr;
    vs->iq_bytes = 0;
    if (cudaMalloc(&vs->iq, bytes) != cudaSuccess) {
      cudaGetLastError();
      vs->iq = nullptr;
      set_error("out of memory for the round buffers");
      return 1;
    }
    vs->iq_bytes = bytes;
  }
  if (!vs->iq_count && cudaMalloc(&vs->iq_count, kWaveCounters * sizeof(unsigned long long)) != cudaSuccess) {
    set_error("out of memory for the round counters");
    return -1;
  }
  return 0;
}

// One round's launches. Counters are handed out in launch order and zeroed
// together at the start of the round.
struct WaveRun {
  trn_viewset* vs;
  Params P;
  Wave W;
  PathSoA R;
  const trn_launch* ln;
  cudaStream_t st;
  int used;

  // Launches K over the round: as many blocks as fit the GPU at once (the
  // kernels stride over a count they read on the device), or the shape the
  // caller asked for; fewer when the round is small.
  // ALL: the GPU's worth of blocks for any round (for_each_spread).
  template <auto K, bool ALL = false, class... A>
  void go(A... args) const {
    const int block = ln && ln->block > 0 ? ln->block : 128;
    int per_sm = ln && ln->blocks_per_sm > 0 ? ln->blocks_per_sm : 0;
    if (!per_sm) {
      static const int fit = [] {
        int n = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, K, 128, 0) == cudaSuccess && n > 0 ? n : 4;
      }();
      per_sm = std::max(1, fit * 128 / block);
    }
    const long long most = (long long)sms() * per_sm;
    launch<K>(ALL ? most : std::min<long long>(most, (W.cap + block - 1) / block), block, args...);
  }
  template <auto K, class... A>
  void launch(long long grid, int block, A... args) const {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)std::max(1LL, grid));
    c.blockDim = dim3(block);
    c.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = attr;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, K, args...);
    count_launch(1);
  }

  unsigned long long* ctr() { return vs->iq_count + used++; }
  int begin() {
    used = 0;
    TRN_CUDA_TRY(cudaMemsetAsync(vs->iq_count, 0, kWaveCounters * sizeof(unsigned long long), st));
    return 0;
  }
  // rays [r0, r0 + *n): hits to W.hit[which], occlusion to W.occ
  void trace(long long r0, const unsigned long long* n, int which) {
    const long long need = (2 * W.cap + TRN_TRACE_BLOCK / 32 - 1) / (TRN_TRACE_BLOCK / 32);  // one ray per warp
    launch<k_trace>(std::min((long long)sms() * TRN_TRACE_MINB, need), TRN_TRACE_BLOCK, P.s, W, r0, n, ctr(),
                    W.hit[which], P.err);
  }
  // First bounce that the tail kernel runs for a round of n samples. A bounce by
  // launches is as long as its longest ray twice over; it is worth that while
  // there are more paths than the GPU holds threads (2^17). About half of the paths
  // are left after each bounce. Images of depth 12 on 102,400 triangles, us, with a
  // launch pair per bounce / the tail from 2^16, 2^17 or 2^18 paths on / one thread
  // per path: 768 samples 440 / 266 / 374, 12,288 781 / 454 / 587, 131,072 1308 /
  // 877, 865, 879 / 1018, 393,216 1569 / 1232, 1107, 1415 / 1593, 1,048,576 2393 /
  // 1977, 1881, 2165 / 3253, 4,194,304 5148 / 4879, 4741, 4989 / 9914.
  static int tail_bounce(long long n) {
    int b = 1;
    while ((n >> b) > (1 << TRN_TAIL_LOG2)) b++;
    return b;
  }
  // bounces of the entries that the start kernel left in list[0]
  template <int MODE>
  void bounces(const unsigned long long* n, unsigned long long* n_ray, int depth, int tail) {
    for (int b = 0; b < depth; b++) {
      trace(0, n_ray, 0);
      Stage S{n, W.list[b & 1], ctr(), W.list[(b + 1) & 1], ctr(), nullptr, b};
      if (b + 1 >= tail && b + 1 < depth) {
        go<k_wf_shade<MODE, true>, true>(P, W, S, R);
        return;
      }
      go<k_wf_shade<MODE, false>>(P, W, S, R);
      n = S.n_out; n_ray = S.n_ray;
    }
  }
  // set-up rays and geometry of a boundary term: items to P.queue
  template <int TERM>
  void setup(long long first) {
    unsigned long long* n = ctr();
    go<k_setup_rays<TERM>>(P, W, first, n);
    trace(0, n, 0);
    if constexpr (TERM != TRN_PIXEL_EDGE) {
      unsigned long long* n2 = ctr();
      go<k_setup_rays2<TERM>>(P, W, first, n, n2);
      trace(W.cap, n2, 1);
      n = n2;
    }
    go<k_setup_finish<TERM>>(P, W, first, n);
  }
};

WaveRun wave_run(trn_viewset* vs, const Params& P, const trn_launch* ln, cudaStream_t st) {
  WaveRun r;
  std::memset(&r.W, 0, sizeof(r.W));
  std::memset(&r.R, 0, sizeof(r.R));
  r.vs = vs;
  r.P = P;
  r.st = st;
  r.used = 0;
  r.ln = ln;
  return r;
}

// Image of a round of n slots from its radiance.
void pixel_sums(const WaveRun& r, long long n) {
  int deep = 0, rest = 0;
  for (int v = 0; v < r.vs->nviews; v++) {
    const trn_camera& c = r.vs->h_views[v].camera;
    (deep_pixels((long long)c.width * c.height, r.vs->h_slots[v]) ? deep : rest)++;
  }
  if (rest) r.go<k_wf_pixels>(r.P, r.W, n);
  if (!deep) return;
  // 16 blocks of 4 warps per SM over the deep views
  const int per_view = std::max(1, sms() * 16 / deep);
  r.launch<k_wf_deep_pixels>((long long)per_view * r.vs->nviews, 128, r.P, r.W, n, per_view);
}

// Interior term over all slots, in rounds: forward image (kWfFwd), with records
// into P.queue (kWfRec, records given by `cache`), or replayed records and the
// reverse sweep of each round (kWfReplay). Returns 1 when there are no buffers
// for it (ensure_queue).
template <int MODE>
int path_wave(trn_viewset* vs, const Params& P0, const trn_launch* ln, long long total, const PathSoA* cache,
              cudaStream_t st) {
  const int depth = vs->max_depth;
  const long long cap = std::min(total, round_cap(ln, MODE == kWfReplay ? kReplayRound : kRound));
  // an image-only set stays at an image's round
  const size_t most = MODE == kWfReplay ? full_queue_bytes(depth <= 8) : path_round_bytes(kRound, depth, false);
  const int rc = ensure_queue(vs, path_round_bytes(cap, depth, MODE == kWfReplay), most, st);
  if (rc) return rc;
  WaveRun r = wave_run(vs, P0, ln, st);
  void* items;
  const size_t wb = wave_layout(r.W, &items, vs->iq, cap, TRN_PATH_TRACER, depth);
  if (MODE == kWfRec) {
    r.R = *cache;
    if (total <= kEndOrder) r.R.n_end = vs->pc_count + 1;
  }
  if (MODE == kWfReplay) {
    path_soa(r.R, static_cast<char*>(vs->iq) + wb, cap, depth);
    r.P.q_cap = cap;
  }
  for (long long first = 0; first < total; first += cap) {
    const long long n = std::min(cap, total - first);
    if (r.begin()) return -1;
    r.W.first = first;
    if (MODE == kWfReplay) {
      r.P.q_count = r.ctr();
      if (total <= kEndOrder) r.R.n_end = r.ctr();
    }
    unsigned long long* rays = r.ctr();
    r.go<k_wf_camera>(r.P, r.W, n, MODE == kWfReplay, rays);
    r.trace(0, rays, 0);
    Stage S{rays, r.W.list[1], r.ctr(), r.W.list[0], r.ctr(), r.ctr(), 0};
    r.go<k_wf_start<MODE>>(r.P, r.W, S, r.R);
    r.bounces<MODE>(S.n_out, S.n_ray, depth, WaveRun::tail_bounce(n));
    if (MODE == kWfReplay) r.go<k_path_reverse<false>>(r.P, r.R);
    else pixel_sums(r, n);
  }
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

// |baseVal| of the guiding tree's samples, in rounds of whole leaves: to value
// (EVAL: tree.per per leaf) or as leaf means to poly. Returns 1 when there are
// no buffers for it (ensure_queue).
template <bool EVAL>
int guide_wave(trn_viewset* vs, const Params& P, const trn_launch* ln, const GuideTree& tree, long long limit,
               float* value, float* poly, cudaStream_t st) {
  const long long leaves = std::min(limit, std::max(1LL, round_cap(ln, kRound) / tree.per));
  const long long cap = leaves * tree.per;
  WaveRun r = wave_run(vs, P, ln, st);
  void* items;
  const int rc = ensure_queue(vs, wave_layout(r.W, &items, nullptr, cap, TRN_DIRECT_EDGE, vs->max_depth),
                              full_queue_bytes(vs->max_depth <= 8), st);
  if (rc) return rc;
  wave_layout(r.W, &items, vs->iq, cap, TRN_DIRECT_EDGE, vs->max_depth);
  for (long long leaf = 0; leaf < limit; leaf += leaves) {
    const long long nl = std::min(leaves, limit - leaf), n = nl * tree.per, first = leaf * tree.per;
    float* v = EVAL ? value + first : r.W.W;
    if (r.begin()) return -1;
    unsigned long long *a = r.ctr(), *b = r.ctr();
    r.go<k_guide_rays<EVAL>>(r.P, r.W, tree, first, n, v, a);
    r.trace(0, a, 0);
    r.go<k_guide_rays2<EVAL>>(r.P, r.W, tree, first, a, b);
    r.trace(r.W.cap, b, 1);
    r.go<k_guide_values<EVAL>>(r.P, r.W, tree, first, b, v);
    if (!EVAL) {
      k_guide_mean<<<(unsigned)((nl + 255) / 256), 256, 0, st>>>(tree.count, tree.per, leaf, nl, v, poly);
      count_launch(1);
    }
  }
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

// AdaptiveQuadratureDistribution::setup (AQ_distrb.h:83-173) for one
// direct-boundary call: the depth-0 tree, g_direct_depth refinement passes
// (the loop the reference keeps commented out, AQ_distrb.h:121-136, with
// gen_eval_point and cut_tree of NEE.cu:91-396), leaf weights from
// g_direct_spp samples per leaf, eps mixing, leaf distribution. The tree
// holds at most max(E, g_direct_max_size) leaves. The set-up samples come
// from the counter hash (their own terms), also when the call's samples come
// from a table. The allocation-free entry point refuses a refinement that would
// need larger arrays than the scene holds.
// With a view set (vs), the samples' ray queries run as a wavefront in its
// round buffers; without one (allocation-free), or without room for them, each
// thread traces its own.
int guide_setup(trn_scene* s, trn_viewset* vs, const trn_render_options* o, const trn_launch* ln, Params& P,
                cudaStream_t st) {
  if (!o->g_direct || s->ne == 0) return 0;
  if (o->g_direct_spp <= 0) { set_error("g_direct_spp must be positive when g_direct is set"); return -1; }
  if (!(o->g_eps >= 0.f && o->g_eps <= 1.f)) { set_error("g_eps must be in [0, 1]"); return -1; }
  if (o->g_direct_depth < 0) { set_error("g_direct_depth must be >= 0"); return -1; }
  const int depth = o->g_direct_depth;
  const long long limit = depth > 0 ? std::max<long long>(s->ne, o->g_direct_max_size) : s->ne;
  if (limit > 0x7FFFFFFFLL / kAqPoints) { set_error("guiding: g_direct_max_size is too large"); return -1; }
  if (limit * o->g_direct_spp > 0xFFFFFFFFLL) {
    set_error("guiding: leaves x g_direct_spp exceeds 2^32 set-up samples");
    return -1;
  }
  if (depth > 0) {
    if (!(o->g_direct_thold >= 0.f)) { set_error("g_direct_thold must be >= 0"); return -1; }
    if ((limit > s->aq_cap || !s->aq_eval) && !vs) {
      set_error("refining the guiding tree (g_direct_depth > 0) allocates its arrays on first use; call "
                "trn_render_grad once with the same options first");
      return -1;
    }
    if (aq_reserve(s, limit)) return -1;
  }
  s->aq_captured |= capturing(st);
  Params G = P;
  G.table = nullptr;
  G.stats = nullptr;
  const long long cap = s->aq_cap;
  const uint32_t stream = (uint32_t)o->seed * 1000003u;
  k_aq_init<<<(s->ne + 255) / 256, 256, 0, st>>>(s->ne, s->sec_cdf, s->aq_box, s->aq_edge, s->aq_count, cap);
  int launches = 1;
  for (int pass = 0; pass < depth; pass++) {
    const uint32_t ps = stream + (uint32_t)pass;
    const GuideTree tree{s->aq_box, s->aq_edge, s->aq_count, cap, ps, kAqPoints};
    const int rc = vs ? guide_wave<true>(vs, G, ln, tree, limit, s->aq_eval, nullptr, st) : 1;
    if (rc < 0) return -1;
    if (rc)
      k_aq_eval<<<(unsigned)((limit * kAqPoints + 255) / 256), 256, 0, st>>>(G, ps, s->aq_box, s->aq_edge, s->aq_count,
                                                                             cap, s->aq_eval);
    k_aq_flag<<<(unsigned)((limit + 255) / 256), 256, 0, st>>>(s->aq_box, s->aq_count, cap, s->aq_eval,
                                                               o->g_direct_thold, ps, s->aq_flag);
    k_aq_scan<<<1, 1024, 0, st>>>(s->aq_count, s->aq_flag, s->aq_prefix, s->aq_count, (int)limit);
    k_aq_split<<<(unsigned)((limit + 255) / 256), 256, 0, st>>>(s->aq_count, s->aq_flag, s->aq_prefix, s->aq_box,
                                                                s->aq_edge, cap);
    k_aq_commit<<<1, 1, 0, st>>>(s->aq_count);
    launches += 5;
  }
  const GuideTree tree{s->aq_box, s->aq_edge, s->aq_count, cap, stream, o->g_direct_spp};
  const int rc = vs ? guide_wave<false>(vs, G, ln, tree, limit, nullptr, s->aq_poly, st) : 1;
  if (rc < 0) return -1;
  if (rc)
    k_aq_poly<<<(unsigned)((limit + 255) / 256), 256, 0, st>>>(G, stream, o->g_direct_spp, s->aq_box, s->aq_edge,
                                                                s->aq_count, cap, s->aq_poly);
  k_aq_mix<<<1, 1024, 0, st>>>(s->aq_count, s->aq_poly, s->aq_box, cap, o->g_eps, s->aq_func, s->aq_int);
  count_launch(launches + 2 +
               cdf_launch(1, (int)limit, s->aq_count, s->aq_func, s->aq_cdf, s->aq_int, s->cdf_part, st));
  TRN_CUDA_TRY(cudaGetLastError());
  P.aq_poly = s->aq_poly;
  P.aq_cdf = s->aq_cdf;
  P.aq_int = s->aq_int;
  P.aq_box = s->aq_box;
  P.aq_edge = s->aq_edge;
  P.aq_n = s->aq_count;
  P.aq_cap = cap;
  return 0;
}

#ifndef TRN_EDGE_ORDER
#define TRN_EDGE_ORDER 1
#endif

// Direction bins per edge in the indirect term's run order: bits of the sort
// key below the edge index taken from the samples r1 and r2 (0 and 0 sort by
// edge alone).
#ifndef TRN_INDIRECT_DIR_R1_BITS
#define TRN_INDIRECT_DIR_R1_BITS 2
#endif
#ifndef TRN_INDIRECT_DIR_R2_BITS
#define TRN_INDIRECT_DIR_R2_BITS 6
#endif

// Buffers of the edge-sorted run order for rounds of up to `cap` slots: keys
// and values double-buffered (16 bytes per slot) plus the radix sort's
// temporary storage for vs->sq_cap slots. Grown like the queue (at least
// doubling, up to one full round; not inside stream capture).
int alloc_order(trn_viewset* vs, long long cap, cudaStream_t st) {
  const bool captured = capturing(st);
  if (vs->sq && vs->sq_cap >= cap) {
    vs->sq_captured |= captured;
    return 0;
  }
  if (captured) {
    set_error("boundary term: its sort buffers must be allocated before stream capture (run it once first)");
    return -1;
  }
  const long long n = std::max(cap, std::min(2 * vs->sq_cap, kRound));
  cub::DoubleBuffer<unsigned> k(nullptr, nullptr), v(nullptr, nullptr);
  size_t tmp = 0;
  TRN_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp, k, v, (int)n, 0, 32, st));
  TRN_CUDA_TRY(cudaStreamSynchronize(st));
  if (vs->sq && vs->sq_captured) vs->kept.push_back(vs->sq);
  else if (vs->sq) cudaFree(vs->sq);
  vs->sq_captured = false;
  vs->sq = nullptr;
  vs->sq_cap = 0;
  if (cudaMalloc(&vs->sq, (16 * (size_t)n + 255) / 256 * 256 + tmp) != cudaSuccess) {
    set_error("boundary term: out of memory for its sort buffers");
    return -1;
  }
  vs->sq_cap = n;
  vs->sq_tmp = tmp;
  return 0;
}

// Order buffers for this launch's rounds; returns 1 (run in slot order) when
// the keys of this view set do not fit 32 bits.
int ensure_order(trn_viewset* vs, const Params& P, long long cap, cudaStream_t st) {
  if ((unsigned long long)P.nviews * (unsigned long long)(P.ne + 1) > 0xffffffffull) return 1;
  return alloc_order(vs, cap, st);
}

// Edge-sorted run order of the round [P.order_first, P.total): keys, then a
// stable radix sort over the bits the keys use; sets P.order.
int order_round(trn_viewset* vs, Params& P, int term, cudaStream_t st) {
  const long long n = P.total - P.order_first, cap = vs->sq_cap;
  unsigned* base = static_cast<unsigned*>(vs->sq);
  cub::DoubleBuffer<unsigned> k(base, base + cap), v(base + 2 * cap, base + 3 * cap);
  P.order = nullptr;
  const int grid = (int)std::min<long long>((n + 255) / 256, 16LL * sms());
  unsigned long long keys = (unsigned long long)P.nviews * (unsigned long long)(P.ne + 1);
  // direction bits of the indirect term, r2's given up last, as many as fit
  // the 32-bit key
  int bits_r1 = term == TRN_INDIRECT_EDGE ? TRN_INDIRECT_DIR_R1_BITS : 0;
  int bits_r2 = term == TRN_INDIRECT_EDGE ? TRN_INDIRECT_DIR_R2_BITS : 0;
  while (bits_r1 > 0 && (keys << (bits_r1 + bits_r2)) > 0x100000000ull) bits_r1--;
  while (bits_r2 > 0 && (keys << bits_r2) > 0x100000000ull) bits_r2--;
  keys <<= bits_r1 + bits_r2;
  k_edge_keys<<<grid, 256, 0, st>>>(P, term, bits_r1, bits_r2, k.Current(), v.Current());
  count_launch(1);
  int bits = 1;
  while (bits < 32 && (1ull << bits) < keys) bits++;
  void* tmp = reinterpret_cast<char*>(vs->sq) + (16 * (size_t)cap + 255) / 256 * 256;
  size_t tb = vs->sq_tmp;
  TRN_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, k, v, (int)n, 0, bits, st));
  P.order = v.Current();
  return 0;
}

// Sensor side, then the emitter side of the samples that it leaves.
template <int MAXD>
void indirect_sides(WaveRun& r) {
  IndirectLit<MAXD>* lit = static_cast<IndirectLit<MAXD>*>(r.W.lit);
  unsigned long long* n_lit = r.ctr();
  r.go<k_indirect_sensor<MAXD>>(r.P, r.ctr(), lit, n_lit);
  r.go<k_indirect_emitter<MAXD>>(r.P, r.ctr(), lit, n_lit);
}

// A boundary term over all slots, in rounds: run order, set-up, the paths of
// the samples that passed, scatter.
template <int TERM>
int edge_wave(trn_viewset* vs, const Params& P0, const trn_launch* ln, long long total, cudaStream_t st) {
  const int depth = vs->max_depth;
  if (TERM == TRN_INDIRECT_EDGE && depth < 2) return 0;  // a sensor and an emitter side take a bounce each
  const long long cap = std::min(total, round_cap(ln, kRound));
  WaveRun r = wave_run(vs, P0, ln, st);
  void* items;
  if (ensure_queue(vs, wave_layout(r.W, &items, nullptr, cap, TERM, depth), full_queue_bytes(depth <= 8), st))
    return -1;
  wave_layout(r.W, &items, vs->iq, cap, TERM, depth);
  r.P.queue = items;
  r.P.q_cap = cap;
  const int ordered = TRN_EDGE_ORDER && TERM != TRN_PIXEL_EDGE ? ensure_order(vs, r.P, cap, st) : 1;
  if (ordered < 0) return -1;
  for (long long first = 0; first < total; first += cap) {
    r.P.total = std::min(total, first + cap);
    r.P.order_first = first;
    if (!ordered && order_round(vs, r.P, TERM, st)) return -1;
    if (r.begin()) return -1;
    r.P.q_count = r.ctr();
    if (TERM == TRN_DIRECT_EDGE && r.P.total - first <= 1 << 19) r.go<k_setup_direct>(r.P, first);
    else r.setup<TERM>(first);
    if constexpr (TERM == TRN_DIRECT_EDGE) {
      r.go<k_direct_body>(r.P);
    } else if constexpr (TERM == TRN_INDIRECT_EDGE) {
      if (depth <= 8) indirect_sides<8>(r);
      else indirect_sides<kMaxDepth>(r);
    } else {
      r.go<k_primary_body>(r.P, r.ctr());
    }
  }
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

#ifndef TRN_PATH_CACHE
#define TRN_PATH_CACHE 1
#endif

// What the interior paths of a launch depend on: the scene version, seed,
// depth, slot count and, per view, camera, spp, seed, slot offset and depth.
// (Weights, pixel offsets and buffers only enter the image write and dL/dI.)
std::vector<char> path_key(const trn_viewset* vs, const trn_render_options* o, int spp_override, long long total) {
  std::vector<char> k;
  auto put = [&](const void* p, size_t n) {
    const char* c = static_cast<const char*>(p);
    k.insert(k.end(), c, c + n);
  };
  put(&vs->scene->version, sizeof(vs->scene->version));
  put(&o->seed, sizeof(o->seed));
  put(&o->max_bounces, sizeof(o->max_bounces));
  put(&spp_override, sizeof(spp_override));
  put(&total, sizeof(total));
  for (const trn_view& v : vs->h_views) {
    put(&v.camera, sizeof(v.camera));
    put(&v.spp, sizeof(v.spp));
    put(&v.seed, sizeof(v.seed));
    put(&v.slot_offset, sizeof(v.slot_offset));
    put(&v.max_bounces, sizeof(v.max_bounces));
  }
  return k;
}

// Recording forward render of the interior term into the view set's path
// cache. Returns 1 when the cache is not used (off, a sample table, stream
// capture, above the limit, or no memory for it): the caller then renders
// without records.
int path_cache_fwd(trn_viewset* vs, Params P, const trn_launch* ln, const trn_render_options* o, int spp_override,
                   long long total, cudaStream_t st) {
  vs->pc_valid = false;
  if (!TRN_PATH_CACHE || vs->pc_limit <= 0 || P.table || capturing(st)) return 1;
  PathSoA R;
  const size_t bytes = path_soa(R, nullptr, total, vs->max_depth);
  if (bytes > (size_t)vs->pc_limit) return 1;
  if (vs->pc_bytes < bytes || !vs->pc_count) {
    TRN_CUDA_TRY(cudaStreamSynchronize(st));
    if (vs->pc) cudaFree(vs->pc);
    vs->pc = nullptr;
    vs->pc_bytes = 0;
    if (cudaMalloc(&vs->pc, bytes) != cudaSuccess ||
        (!vs->pc_count && cudaMalloc(&vs->pc_count, 2 * sizeof(unsigned long long)) != cudaSuccess)) {
      cudaGetLastError();  // out of memory: render without records
      if (vs->pc) cudaFree(vs->pc);
      vs->pc = nullptr;
      return 1;
    }
    vs->pc_bytes = bytes;
  }
  TRN_CUDA_TRY(cudaMemsetAsync(vs->pc_count, 0, 2 * sizeof(unsigned long long), st));
  P.q_count = vs->pc_count;
  P.q_cap = total;
  path_soa(R, vs->pc, total, vs->max_depth);
  const int rc = path_wave<kWfRec>(vs, P, ln, total, &R, st);
  if (rc) return rc;
  vs->pc_key = path_key(vs, o, spp_override, total);
  vs->pc_valid = true;
  return 0;
}

// Reverse sweep over the cached records when they are the paths of this
// gradient call. Returns 1 when they are not (the caller replays).
int path_cache_grad(trn_viewset* vs, Params P, const trn_launch* ln, const trn_render_options* o, int spp_override,
                    long long total, cudaStream_t st) {
  if (!vs->pc_valid || P.table || capturing(st)) return 1;
  if (vs->pc_key != path_key(vs, o, spp_override, total)) return 1;
  P.q_count = vs->pc_count;
  P.q_cap = total;
  PathSoA R;
  path_soa(R, vs->pc, total, vs->max_depth);
  if (total <= kEndOrder) R.n_end = vs->pc_count + 1;
  int grid, block;
  launch_dims(ln, total, grid, block);
  k_path_reverse<true><<<grid, block, 0, st>>>(P, R);
  count_launch(1);
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

int render_views(trn_scene* s, trn_viewset* vs, const trn_render_options* o, int integrator,
                 const trn_samples* smp, const trn_launch* ln, int spp_override, bool forward, float* image,
                 const float* dLdI, cudaStream_t st) {
  if (check_common(s, o, integrator)) return -1;
  if (!vs || vs->nviews <= 0) { set_error("empty view set"); return -1; }
  if (validate_launch(ln)) return -1;
  long long total = 0;
  if (upload_views(vs, o, integrator, spp_override, total, st)) return -1;
  Params P = base_params(s, vs, o, integrator, smp, ln, total);
  P.image = forward ? image : nullptr;
  P.dLdI = forward ? nullptr : dLdI;
  const long long slots = integrator == TRN_PIXEL_EDGE ? total / 4 : total;
  if (P.table && P.stride < slots) { set_error("sample table too small"); return -1; }
  if (forward) {
    // a call buffer is cleared; views with their own image accumulate into it
    if (image) TRN_CUDA_TRY(cudaMemsetAsync(image, 0, sizeof(float) * 3 * vs->npix, st));
    if (integrator != TRN_PATH_TRACER || total == 0) return 0;  // edge terms have no primal image
    TRN_CUDA_TRY(cudaMemsetAsync(vs->work, 0, sizeof(unsigned long long), st));
    const int cached = path_cache_fwd(vs, P, ln, o, spp_override, total, st);
    if (cached <= 0) return cached;
    const int rc = path_wave<kWfFwd>(vs, P, ln, total, nullptr, st);
    if (rc <= 0) return rc;
    // without round buffers: one thread per path
    launch(k_path_fwd, ln, total, P, st);
    TRN_CUDA_TRY(cudaGetLastError());
    return 0;
  }
  if (total == 0) return 0;
  s->grads_finalized = false;
  if (integrator == TRN_PRIMARY_EDGE) {
    if (s->ne == 0) return 0;
    dim3 g((s->ne + 255) / 256, vs->nviews);
    k_prim_edges_views<<<g, 256, 0, st>>>(s->ne, s->edges, s->pos, s->fnormal, vs->views, vs->pfunc);
    count_launch(1 + cdf_launch(vs->nviews, s->ne, nullptr, vs->pfunc, vs->pcdf, vs->pint, vs->pint_part, st));
  } else if ((integrator == TRN_DIRECT_EDGE || integrator == TRN_INDIRECT_EDGE) && s->ne == 0) {
    return 0;
  }
  if (integrator == TRN_DIRECT_EDGE && guide_setup(s, vs, o, ln, P, st)) return -1;
  TRN_CUDA_TRY(cudaMemsetAsync(vs->work, 0, sizeof(unsigned long long), st));
  switch (integrator) {
    case TRN_PATH_TRACER: {
      const int cached = path_cache_grad(vs, P, ln, o, spp_override, total, st);
      if (cached <= 0) return cached;
      return path_wave<kWfReplay>(vs, P, ln, total, nullptr, st) ? -1 : 0;
    }
    case TRN_PRIMARY_EDGE: return edge_wave<TRN_PRIMARY_EDGE>(vs, P, ln, total, st);
    case TRN_DIRECT_EDGE: return edge_wave<TRN_DIRECT_EDGE>(vs, P, ln, total, st);
    case TRN_INDIRECT_EDGE: return edge_wave<TRN_INDIRECT_EDGE>(vs, P, ln, total, st);
    default: return edge_wave<TRN_PIXEL_EDGE>(vs, P, ln, total, st);
  }
}

// (Re)define the views of a set. Device arrays grow to the largest view count
// seen; the per-view silhouette workspace is E floats x 2 per view.
int set_views(trn_viewset* vs, int nviews, const trn_view* views) {
  std::vector<long long> pb;
  long long pix = 0;
  for (int v = 0; v < nviews; v++) {
    const trn_view& hv = views[v];
    if (hv.camera.width <= 0 || hv.camera.height <= 0 || hv.spp < 0 || hv.max_bounces < 0 ||
        hv.max_bounces > kMaxDepth) {
      set_error("viewset: invalid view (resolution, spp or max_bounces)");
      return -1;
    }
    const long long off = hv.pixel_offset >= 0 ? hv.pixel_offset : pix;
    if (!pb.empty() && off < pb.back()) { set_error("viewset: pixel offsets must be non-decreasing"); return -1; }
    pb.push_back(off);
    pix = std::max(pix, off + (long long)hv.camera.width * hv.camera.height);
  }
  if (nviews > vs->cap) {
    wait_stages(vs);
    void* old[] = {vs->views, vs->vbegin, vs->pbegin, vs->pfunc, vs->pcdf, vs->pint, vs->pint_part};
    for (void* q : old) if (q) cudaFree(q);
    if (vs->h_stage) cudaFreeHost(vs->h_stage);
    if (vs->h_stage_begin) cudaFreeHost(vs->h_stage_begin);
    vs->views = nullptr; vs->vbegin = vs->pbegin = nullptr; vs->pfunc = vs->pcdf = vs->pint = nullptr;
    vs->pint_part = nullptr;
    vs->h_stage = nullptr; vs->h_stage_begin = nullptr;
    const int cap = std::max(nviews, 2 * vs->cap);
    bool ok = cudaMalloc(&vs->views, sizeof(ViewDesc) * cap) == cudaSuccess &&
              cudaMalloc(&vs->vbegin, sizeof(long long) * cap) == cudaSuccess &&
              cudaMalloc(&vs->pbegin, sizeof(long long) * cap) == cudaSuccess &&
              cudaMalloc(&vs->pint, sizeof(float) * cap) == cudaSuccess &&
              cudaMalloc(&vs->pint_part, sizeof(double) * kCdfChunks * cap) == cudaSuccess &&
              cudaMallocHost(&vs->h_stage, sizeof(ViewDesc) * cap * kStageRing) == cudaSuccess &&
              cudaMallocHost(&vs->h_stage_begin, sizeof(long long) * 2 * cap * kStageRing) == cudaSuccess;
    if (ok && vs->ne > 0)
      ok = cudaMalloc(&vs->pfunc, sizeof(float) * (size_t)cap * vs->ne) == cudaSuccess &&
           cudaMalloc(&vs->pcdf, sizeof(float) * (size_t)cap * vs->ne) == cudaSuccess;
    if (!ok) { set_error("viewset: out of memory"); vs->cap = 0; return -1; }
    cudaMemset(vs->pint, 0, sizeof(float) * cap);
    vs->cap = cap;
  }
  vs->nviews = nviews;
  vs->h_views.assign(views, views + nviews);
  vs->h_pbegin = pb;
  vs->npix = pix;
  vs->uploaded_key = -2;
  vs->pbegin_dirty = true;
  return 0;
}

// upload the per-view pixel offsets (used by the loss kernel) when they changed
int upload_pbegin(trn_viewset* vs, cudaStream_t st) {
  if (!vs->pbegin_dirty) return 0;
  const int slot = next_stage(vs);
  long long* stage = vs->h_stage_begin + (size_t)slot * 2 * vs->cap + vs->cap;
  std::memcpy(stage, vs->h_pbegin.data(), sizeof(long long) * vs->nviews);
  TRN_CUDA_TRY(cudaMemcpyAsync(vs->pbegin, stage, sizeof(long long) * vs->nviews, cudaMemcpyHostToDevice, st));
  TRN_CUDA_TRY(cudaEventRecord(vs->stage_done[slot], st));
  vs->pbegin_dirty = false;
  return 0;
}

// The scene's cached one-view set, re-pointed at `cam`: the first call
// allocates it, later calls only restage the view table (a pinned slot of
// the set's staging ring). A call for more samples than any before it grows the
// set's round buffers (ensure_queue), which waits for the stream; others neither
// allocate nor wait.
int single_view(trn_scene* s, const trn_camera* cam, trn_viewset** out) {
  if (!cam) { set_error("null camera"); return -1; }
  trn_view v;
  std::memset(&v, 0, sizeof(v));
  std::memcpy(&v.camera, cam, sizeof(trn_camera));
  if (s->single) {
    // an unchanged camera keeps the uploaded table: no restaging, so the host
    // does not wait for the previous call's upload and can run ahead
    const bool same = s->single->nviews == 1 && s->single->h_views.size() == 1 &&
                      std::memcmp(&s->single->h_views[0], &v, sizeof(v)) == 0;
    if (!same && set_views(s->single, 1, &v)) return -1;
  } else if (trn_viewset_create(s, 1, &v, &s->single)) {
    return -1;
  }
  s->single->pc_limit = s->single_path_cache;
  *out = s->single;
  return 0;
}

}  // namespace

extern "C" {

int trn_viewset_create(trn_scene* s, int nviews, const trn_view* views, trn_viewset** out) {
  if (!s || !views || !out || nviews <= 0) { set_error("trn_viewset_create: invalid arguments"); return -1; }
  *out = nullptr;
  trn_viewset* vs = new trn_viewset();
  vs->scene = s;
  vs->ne = s->ne;
  bool ok = cudaMalloc(&vs->work, sizeof(unsigned long long)) == cudaSuccess;
  for (cudaEvent_t& e : vs->stage_done) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    set_error("trn_viewset_create: out of memory");
    trn_viewset_destroy(vs);
    return -1;
  }
  if (set_views(vs, nviews, views)) { trn_viewset_destroy(vs); return -1; }
  *out = vs;
  return 0;
}

int trn_viewset_update(trn_viewset* vs, int nviews, const trn_view* views) {
  if (!vs || !views || nviews <= 0) { set_error("trn_viewset_update: invalid arguments"); return -1; }
  return set_views(vs, nviews, views);
}

int trn_viewset_destroy(trn_viewset* vs) {
  if (!vs) return 0;
  wait_stages(vs);
  void* ptrs[] = {vs->views, vs->vbegin, vs->pbegin, vs->pfunc, vs->pcdf, vs->pint, vs->pint_part, vs->work, vs->iq, vs->iq_count, vs->sq, vs->pc, vs->pc_count};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  for (void* p : vs->kept) cudaFree(p);
  if (vs->h_stage) cudaFreeHost(vs->h_stage);
  if (vs->h_stage_begin) cudaFreeHost(vs->h_stage_begin);
  for (cudaEvent_t e : vs->stage_done)
    if (e) cudaEventDestroy(e);
  delete vs;
  return 0;
}

int trn_viewset_num_pixels(const trn_viewset* vs, long long* npix) {
  if (!vs || !npix) { set_error("trn_viewset_num_pixels: null argument"); return -1; }
  *npix = vs->npix;
  return 0;
}

int trn_viewset_reserve(trn_viewset* vs, int max_bounces, cudaStream_t st) {
  if (!vs) { set_error("trn_viewset_reserve: null view set"); return -1; }
  if (max_bounces < 0 || max_bounces > kMaxDepth) { set_error("trn_viewset_reserve: max_bounces must be in [0, 16]"); return -1; }
  const size_t most = full_queue_bytes(max_bounces <= 8);
  if (ensure_queue(vs, most, most, st)) return -1;
  if (TRN_EDGE_ORDER && alloc_order(vs, kRound, st)) return -1;
  return 0;
}

int trn_viewset_path_cache(trn_viewset* vs, long long max_bytes) {
  if (!vs || max_bytes < 0) { set_error("trn_viewset_path_cache: invalid arguments"); return -1; }
  vs->pc_limit = max_bytes;
  vs->pc_valid = false;
  if (max_bytes == 0 && vs->pc) {
    wait_stages(vs);
    TRN_CUDA_TRY(cudaDeviceSynchronize());
    cudaFree(vs->pc);
    vs->pc = nullptr;
    vs->pc_bytes = 0;
  }
  return 0;
}

int trn_scene_path_cache(trn_scene* s, long long max_bytes) {
  if (!s || max_bytes < 0) { set_error("trn_scene_path_cache: invalid arguments"); return -1; }
  s->single_path_cache = max_bytes;
  if (s->single) return trn_viewset_path_cache(s->single, max_bytes);
  return 0;
}

int trn_render_views_fwd(trn_scene* s, trn_viewset* vs, const trn_render_options* o, int integrator,
                         const trn_samples* smp, const trn_launch* ln, float* images, cudaStream_t st) {
  if (!images)
    for (const trn_view& v : vs->h_views)
      if (!v.image) { set_error("trn_render_views_fwd: no image buffer for a view"); return -1; }
  return render_views(s, vs, o, integrator, smp, ln, -1, true, images, nullptr, st);
}

int trn_render_views_grad(trn_scene* s, trn_viewset* vs, const trn_render_options* o, int integrator,
                          const trn_samples* smp, const trn_launch* ln, const float* dLdI, cudaStream_t st) {
  if (!dLdI)
    for (const trn_view& v : vs->h_views)
      if (!v.dLdI) { set_error("trn_render_views_grad: no dL/dI buffer for a view"); return -1; }
  return render_views(s, vs, o, integrator, smp, ln, -1, false, nullptr, dLdI, st);
}

int trn_views_loss(trn_viewset* vs, const float* images, const float* targets, float* dLdI, float* loss,
                   cudaStream_t st) {
  if (!vs || !images || !targets) { set_error("trn_views_loss: null argument"); return -1; }
  if (upload_pbegin(vs, st)) return -1;
  if (loss) TRN_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(float) * vs->nviews, st));
  const long long n = vs->npix;
  k_view_loss<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, vs->views, vs->pbegin, vs->nviews, images, targets,
                                                          dLdI, loss);
  count_launch(1);
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

int trn_render_fwd(trn_scene* s, const trn_camera* cam, const trn_render_options* o, int integrator,
                   const trn_samples* smp, float* image, cudaStream_t st) {
  if (check_common(s, o, integrator)) return -1;
  if (!image) { set_error("trn_render_fwd: null image"); return -1; }
  trn_viewset* vs = nullptr;
  if (single_view(s, cam, &vs)) return -1;
  return render_views(s, vs, o, integrator, smp, nullptr, spp_of(o, integrator), true, image, nullptr, st);
}

int trn_render_grad(trn_scene* s, const trn_camera* cam, const trn_render_options* o, int integrator,
                    const trn_samples* smp, const float* dLdI, cudaStream_t st) {
  if (check_common(s, o, integrator)) return -1;
  if (!dLdI) { set_error("trn_render_grad: null dLdI"); return -1; }
  trn_viewset* vs = nullptr;
  if (single_view(s, cam, &vs)) return -1;
  return render_views(s, vs, o, integrator, smp, nullptr, spp_of(o, integrator), false, nullptr, dLdI, st);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free single-view gradient.
//
// trn_render_grad allocates device memory: the scene's one-view table, work
// counter and silhouette-edge distribution on a scene's first single-view call,
// and round buffers whenever a call has more samples than those before. Callers that may not allocate (a host that forbids cudaMalloc
// between set-up and teardown, a caching allocator that must not be bypassed,
// a real-time loop that cannot afford the implicit synchronisation of
// cudaFree) use trn_render_grad_noalloc instead: all of its scratch lives in
// the fixed-size array below, which is part of the loaded module.
//
// Scratch layout (each part 256-byte aligned): the view table (one ViewDesc),
// the first-sample index of that view, the work counter, the silhouette
// integral, then the silhouette function and its CDF (kNoAllocMaxEdges floats
// each), then the CDF's chunk sums. Every call rewrites all of it that it reads, so it keeps the last
// call's contents but never needs clearing from the outside. Two calls that
// overlap in time on one device share this one array and race; such callers
// must serialise them.
constexpr int kNoAllocMaxEdges = 1 << 20;
constexpr size_t kNoAllocHeader = 4096;  // ViewDesc, vbegin, work counter, integral
constexpr size_t kNoAllocScratchBytes =
    kNoAllocHeader + 2 * sizeof(float) * (size_t)kNoAllocMaxEdges + kCdfChunks * sizeof(double);
static_assert(sizeof(ViewDesc) + 3 * 256 <= kNoAllocHeader, "view table does not fit the scratch header");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {

constexpr int kNoAllocMaxDevices = 64;
std::atomic<unsigned char*> g_noalloc_base[kNoAllocMaxDevices];

// Device address of the scratch array for the current device. In host code
// the array's name only stands in for it, so the address comes from
// cudaGetSymbolAddress, once per device (this may load the module on that
// device, which is why the first call must not run inside stream capture).
// The scene's buffers must live on the current device: the address looked up
// is that device's copy of the array, and kernels launched there would
// otherwise read another GPU's scene.
unsigned char* noalloc_scratch(const trn_scene* s) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
    set_error("trn_render_grad_noalloc: no usable current device");
    return nullptr;
  }
  cudaPointerAttributes pa;
  if (cudaPointerGetAttributes(&pa, s->pos) != cudaSuccess || pa.type != cudaMemoryTypeDevice) {
    cudaGetLastError();
    set_error("trn_render_grad_noalloc: cannot tell which device holds the scene");
    return nullptr;
  }
  if (pa.device != dev) {
    set_error("trn_render_grad_noalloc: the scene lives on device " + std::to_string(pa.device) +
              " but device " + std::to_string(dev) + " is current; make the scene's device current");
    return nullptr;
  }
  unsigned char* p = g_noalloc_base[dev].load(std::memory_order_acquire);
  if (p) return p;
  void* addr = nullptr;
  const cudaError_t rc = cudaGetSymbolAddress(&addr, g_noalloc_scratch);
  if (rc != cudaSuccess || !addr) {
    set_error(std::string("trn_render_grad_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(rc));
    return nullptr;
  }
  g_noalloc_base[dev].store((unsigned char*)addr, std::memory_order_release);
  return (unsigned char*)addr;
}

// Write the one-view table, its first-sample index (0) and a zero work
// counter into the scratch header; the view is passed by value, so no host
// staging buffer is involved.
__global__ void k_noalloc_setup(ViewDesc v, ViewDesc* table, long long* vbegin, unsigned long long* work) {
  if (threadIdx.x == 0) {
    *table = v;
    *vbegin = 0;
    *work = 0ull;
  }
}

}  // namespace

extern "C" {

int trn_render_grad_noalloc(trn_scene* s, const trn_camera* cam, const trn_render_options* o, int integrator,
                            const trn_samples* smp, const float* dLdI, cudaStream_t st) {
  if (check_common(s, o, integrator)) return -1;
  if (!cam || !dLdI) { set_error("trn_render_grad_noalloc: null camera or dLdI"); return -1; }
  if (cam->width <= 0 || cam->height <= 0) { set_error("trn_render_grad_noalloc: invalid resolution"); return -1; }
  if (integrator == TRN_PRIMARY_EDGE && s->ne > kNoAllocMaxEdges) {
    set_error("trn_render_grad_noalloc: the scene has " + std::to_string(s->ne) +
              " edges; the static scratch holds the silhouette distribution of at most " +
              std::to_string(kNoAllocMaxEdges));
    return -1;
  }
  const int spp = spp_of(o, integrator);
  if (spp < 0) { set_error("trn_render_grad_noalloc: negative spp"); return -1; }
  const long long total = (long long)cam->width * cam->height * spp;
  if (integrator == TRN_PIXEL_EDGE && total % 4 != 0) {
    set_error("pixel boundary needs W*H*spp divisible by 4");
    return -1;
  }
  unsigned char* base = noalloc_scratch(s);
  if (!base) return -1;
  ViewDesc* table = (ViewDesc*)base;
  long long* vbegin = (long long*)(base + kNoAllocHeader - 3 * 256);
  unsigned long long* work = (unsigned long long*)(base + kNoAllocHeader - 2 * 256);
  float* pint = (float*)(base + kNoAllocHeader - 256);
  float* pfunc = (float*)(base + kNoAllocHeader);
  float* pcdf = pfunc + kNoAllocMaxEdges;
  double* part = (double*)(pcdf + kNoAllocMaxEdges);

  ViewDesc v;
  std::memset(&v, 0, sizeof(v));
  std::memcpy(&v.cam, cam, sizeof(CameraDesc));
  v.begin = 0;
  v.n = total;
  v.pix_off = 0;
  v.slot_off = 0;
  v.inv_spp = spp > 0 ? 1.0f / (float)spp : 0.f;
  v.seed = 0;
  v.spp = spp;
  v.D = o->max_bounces;
  v.gpos = s->g_pos;
  v.gvn = s->g_vnormal;
  v.gtex = s->g_texels;
  v.pfunc = pfunc;
  v.pcdf = pcdf;
  v.pint = pint;

  // host-side view of the scratch (no device memory of its own)
  trn_viewset vs;
  vs.scene = s;
  vs.nviews = 1;
  vs.ne = s->ne;
  vs.views = table;
  vs.vbegin = vbegin;
  vs.work = work;
  Params P = base_params(s, &vs, o, integrator, smp, nullptr, total);
  P.image = nullptr;
  P.dLdI = dLdI;
  const long long slots = integrator == TRN_PIXEL_EDGE ? total / 4 : total;
  if (P.table && P.stride < slots) { set_error("sample table too small"); return -1; }
  if (total == 0) return 0;
  if ((integrator == TRN_PRIMARY_EDGE || integrator == TRN_DIRECT_EDGE || integrator == TRN_INDIRECT_EDGE) &&
      s->ne == 0)
    return 0;

  k_noalloc_setup<<<1, 32, 0, st>>>(v, table, vbegin, work);
  count_launch(1);
  s->grads_finalized = false;
  if (integrator == TRN_PRIMARY_EDGE) {
    dim3 g((s->ne + 255) / 256, 1);
    k_prim_edges_views<<<g, 256, 0, st>>>(s->ne, s->edges, s->pos, s->fnormal, table, pfunc);
    count_launch(1 + cdf_launch(1, s->ne, nullptr, pfunc, pcdf, pint, part, st));
  }
  // the guiding distribution lives in buffers the scene allocated at creation
  // (a refined tree in those of an earlier allocating call)
  if (integrator == TRN_DIRECT_EDGE && guide_setup(s, nullptr, o, nullptr, P, st)) return -1;
  const bool shallow = o->max_bounces <= 8;
  switch (integrator) {
    case TRN_PATH_TRACER:
      if (shallow) launch(k_path_adj<8>, nullptr, total, P, st); else launch(k_path_adj<kMaxDepth>, nullptr, total, P, st);
      break;
    case TRN_PRIMARY_EDGE: launch(k_primary_adj, nullptr, total, P, st); break;
    case TRN_DIRECT_EDGE: launch(k_direct_adj, nullptr, total, P, st); break;
    case TRN_INDIRECT_EDGE:
      if (shallow) launch(k_indirect_adj<8>, nullptr, total, P, st);
      else launch(k_indirect_adj<kMaxDepth>, nullptr, total, P, st);
      break;
    default: launch(k_pixel_adj, nullptr, total, P, st); break;
  }
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

int trn_intersect(trn_scene* s, int n, const float* org, const float* dir, const float* tmin, const float* tmax,
                  int* tri, float* u, float* v, float* t, cudaStream_t st) {
  if (!s || !s->configured) { set_error("trn_intersect: scene not configured"); return -1; }
  if (n <= 0) return 0;
  if (!org || !dir || !tmin || !tmax || !tri || !u || !v || !t) { set_error("trn_intersect: null argument"); return -1; }
  if (query_streams(n, s->nt)) {
    int grid, chunk;
    query_dims(n, grid, chunk);
    k_query<false><<<grid, TRN_TRACE_BLOCK, 0, st>>>(s->view(), n, chunk, org, dir, tmin, tmax, tri, u, v, t, s->err);
  } else {
    k_query_one<false><<<(n + 127) / 128, 128, 0, st>>>(s->view(), n, org, dir, tmin, tmax, tri, u, v, t, s->err);
  }
  count_launch(1);
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

int trn_occluded(trn_scene* s, int n, const float* org, const float* dir, const float* tmin, const float* tmax,
                 int* vis, cudaStream_t st) {
  if (!s || !s->configured) { set_error("trn_occluded: scene not configured"); return -1; }
  if (n <= 0) return 0;
  if (!org || !dir || !tmin || !tmax || !vis) { set_error("trn_occluded: null argument"); return -1; }
  if (query_streams(n, s->nt)) {
    int grid, chunk;
    query_dims(n, grid, chunk);
    k_query<true><<<grid, TRN_TRACE_BLOCK, 0, st>>>(s->view(), n, chunk, org, dir, tmin, tmax, vis, nullptr, nullptr,
                                                    nullptr, s->err);
  } else {
    k_query_one<true><<<(n + 127) / 128, 128, 0, st>>>(s->view(), n, org, dir, tmin, tmax, vis, nullptr, nullptr,
                                                       nullptr, s->err);
  }
  count_launch(1);
  TRN_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // extern "C"
