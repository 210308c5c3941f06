// Wavefront form of the interior term and of the boundary terms' set-ups: paths
// of one round advance together, one bounce per pair of launches. A shading
// kernel ends the previous bounce with its ray results and decides the next
// bounce's rays; k_trace runs all of them. Between them only the rays, their
// results and 64 bytes of path state pass through memory (an L2's worth at a
// time).
//
// Why: with one thread per path, traversal and shading of 32 unrelated paths
// shared a warp, with 6 to 8 of 32 lanes active per instruction. Here a
// traversal warp refills its free lanes with rays of any path (trace_stream),
// and a shading warp holds 32 paths at the same bounce. 16.8M samples of depth
// 5 on 102,400 triangles, one thread per path and here: image 27.6 and 15.8 ms.
//
// The price is a launch pair per bounce, each as long as its longest ray: the
// late bounces of few paths run in one kernel instead (WaveRun::tail_bounce).
// (The paths of a boundary term's samples run in one kernel each, behind these
// set-ups: render.cu says why.)
//
// Included by render.cu (uses its parameter block and path functions).
#pragma once

// Buffers of one round of up to `cap` samples.
struct Wave {
  long long cap;
  float4 *ro, *rd;          // [2 cap] rays: origin + id bits, direction + end
  float4* hit[2];           // [cap] closest-hit results by ray id: tri, u, v, t
  unsigned char* occ;       // [cap] occlusion results by ray id
  unsigned* list[2];        // [cap] active samples of a stage, ping-pong; a set-up's samples by ray id
  float4* st[4];            // [cap] path state
  long long* p;             // [cap] view-local sample index
  int* view;                // [cap]
  unsigned* rec;            // [cap] record index (recording modes)
  F3* L;                    // [cap] radiance by slot of the round (forward modes)
  long long first;          // first slot of the round (interior term)
  float* W;                 // [cap] values of the guiding samples
  void* lit;                // [cap] indirect samples that go on to the emitter side
};

// ray ids: bit 31 marks an occlusion query
constexpr unsigned kAnyRay = 0x80000000u;
// list entries: the sample, and which rays its current bounce has cast
constexpr unsigned kCastShadow = 0x80000000u, kCastCont = 0x40000000u, kEntryMask = 0x3fffffffu;

// One stage: its input list with the count, its output list with the count,
// and the ray counter. All counts are device counters zeroed with the round.
struct Stage {
  const unsigned long long* n;
  const unsigned* in;
  unsigned long long* n_out;
  unsigned* out;
  unsigned long long* n_ray;
  unsigned long long* n_state;  // path states handed out (first stage of the camera modes)
  int b;                    // bounce
};

// Position of each wanting lane behind `counter` (one atomic per warp; all
// lanes of the warp call it).
TRN_D unsigned long long warp_append(unsigned long long* counter, bool want) {
  const unsigned m = __ballot_sync(0xffffffffu, want);
  if (!m) return 0;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

TRN_D void put_ray(const Wave& W, unsigned long long k, const F3& o, const F3& d, float tmax, unsigned id) {
  __stcs(W.ro + k, make_float4(o.x, o.y, o.z, __uint_as_float(id)));
  __stcs(W.rd + k, make_float4(d.x, d.y, d.z, tmax));
}
TRN_D void push_ray(const Wave& W, unsigned long long* n_ray, bool want, const F3& o, const F3& d, float tmax,
                    unsigned id) {
  const unsigned long long k = warp_append(n_ray, want);
  if (want) put_ray(W, k, o, d, tmax, id);
}
TRN_D Hit get_hit(const float4* h, unsigned long long i) {
  const float4 a = __ldcs(h + i);
  Hit r;
  r.tri = __float_as_int(a.x); r.u = a.y; r.v = a.z; r.t = a.w;
  return r;
}

// Warp-uniform loop over [0, n): body(index, exists).
template <class F>
TRN_D void for_each_entry(unsigned long long n, F&& body) {
  const int lane = threadIdx.x & 31;
  for (unsigned long long k0 = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) & ~31ull; k0 < n;
       k0 += (unsigned long long)gridDim.x * blockDim.x)
    body(k0 + lane, k0 + lane < n);
}

// The same with the entries spread over all warps, down to one each, for work
// that takes every lane another way: few lanes of a warp then wait for each other.
template <class F>
TRN_D void for_each_spread(unsigned long long n, F&& body) {
  const int lane = threadIdx.x & 31;
  const unsigned long long warps = gridDim.x * (blockDim.x >> 5), w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const unsigned long long own = min(32ull, max(1ull, (n + warps - 1) / warps));
  for (unsigned long long k0 = w * own; k0 < n; k0 += warps * own) body(k0 + lane, lane < own && k0 + lane < n);
}

// ---------------------------------------------------------------------------
// ray queries of a stage: rays [r0, r0 + *n_ray) of the queue
// ---------------------------------------------------------------------------
#ifndef TRN_TRACE_MINB
#define TRN_TRACE_MINB 8
#endif

// Each warp starts on rays of its own and then fetches from `next`; few rays
// are spread over all warps (a query is as long as its longest ray, and a warp
// of few rays takes fewer turns). (One ray per thread for batches of 19K to 230K,
// as for a program's own rays: images of 131,072 samples 130 -> 163 us.)
__global__ void __launch_bounds__(TRN_TRACE_BLOCK, TRN_TRACE_MINB)
    k_trace(const __grid_constant__ DeviceScene s, const __grid_constant__ Wave W, long long r0, const unsigned long long* n_ray,
            unsigned long long* next, float4* hits, int* err) {
  stage_begin();
  const int n = (int)*n_ray;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const float4* ro = W.ro + r0;
  const float4* rd = W.rd + r0;
  const int own = min(32, max(1, (n + warps - 1) / warps));
  bool first = true;
  trace_stream(s,
    [&](int k, int& lim, bool& more) -> int {
      if (first) {
        first = false;
        lim = min(n, own * (w + 1));
        more = own * warps < n;
        return min(n, own * w);
      }
      unsigned long long base = 0;
      if ((threadIdx.x & 31) == 0) base = atomicAdd(next, (unsigned long long)k);
      lim = n;
      const int r = (int)min((unsigned long long)n, (unsigned long long)(own * warps) + __shfl_sync(0xffffffffu, base, 0));
      more = r + k < n;
      return r;
    },
    [&](int i, F3& o, F3& d, float& tmin, float& tmax, bool& any) {
      const float4 a = __ldcs(ro + i), b = __ldcs(rd + i);
      o = F3(a.x, a.y, a.z); d = F3(b.x, b.y, b.z);
      tmin = kShadowEps; tmax = b.w;
      any = (__float_as_uint(a.w) & kAnyRay) != 0u;
    },
    [&](int i, bool any, int tri, float u, float v, float t) {
      const unsigned id = __float_as_uint(ro[i].w) & ~kAnyRay;
      if (any) W.occ[id] = tri >= 0;
      else __stcs(hits + id, make_float4(__int_as_float(tri), u, v, t));
    }, err);
}

// ---------------------------------------------------------------------------
// radiance paths of the interior term (image, records, replay)
// ---------------------------------------------------------------------------
// kWfFwd: forward image; kWfRec: forward image and path records; kWfReplay:
// path records for the adjoint.
enum WfMode { kWfFwd = 0, kWfRec, kWfReplay };

struct WfPath {
  SurfF x;
  F3 rdir, T, L;
};

TRN_D bool is_dark(const F3& T) { return T.x == 0.f && T.y == 0.f && T.z == 0.f; }

// Bounce k's light sample, and what the bounce came to (the vertex q when it
// goes on), into record kr.
TRN_D void wf_record_light(const PathSoA& R, unsigned kr, int k, const BounceRec& br) {
  LRec& l = R.br(kr, k);
  l.ltri = br.ltri; l.lu = br.lu; l.lv = br.lv; l.lpdf = br.lpdf; l.lmis = br.lmis;
}
TRN_D void wf_record(const PathSoA& R, unsigned kr, int k, const BounceRec& br, bool more, const WfPath& q) {
  // a scrubbed (non-finite) bounce contributes nothing and carries no gradient
  if (br.nee_ok && !br.scrubbed) R.nee(kr) |= 1u << k;
  if (!more) return;
  R.br(kr, k).ppdf = br.prev_pdf;
  R.vr(kr, k + 1) = {q.x.tri, q.x.u, q.x.v};
  R.Tk(kr, k + 1) = q.T;
  R.Mk(kr, k + 1) = (br.scrubbed || br.emis == 0.f) ? F3z() : br.eLe * br.emis;
  R.K(kr) = k + 1;
}

// Decides the rays of bounce b for the lanes that go on, appends them and the
// lanes' list entries, and stores the path state. All lanes of the warp call it.
template <int MODE>
TRN_D void wf_advance(const Params& P, const Wave& W, const Stage& S, int b, bool go, unsigned i, const ViewDesc* V,
                      long long p, const WfPath& q, const PathSoA& R, Cnt& cnt) {
  RadianceGen g;
  g.shadow = g.cont = false;
  if (go) {
    const PathSmp smp{&P, V->seed, p + V->begin, p + V->slot_off};
    const int o = 2 + 5 * b;
    BounceRec br;
    constexpr bool rec = MODE != kWfFwd;
    radiance_gen(P.s, q.x, shading_at(P.s, q.x), q.rdir, q.T, smp(o), smp(o + 1), smp(o + 2), smp(o + 3), smp(o + 4), g, rec ? &br : nullptr,
                 cnt, [](const F3&, float) { return true; });
    W.st[0][i] = make_float4(__int_as_float(q.x.tri), q.x.u, q.x.v, g.pdf);
    W.st[1][i] = make_float4(q.rdir.x, q.rdir.y, q.rdir.z, q.T.x);
    W.st[2][i] = make_float4(q.T.y, q.T.z, q.L.x, q.L.y);
    W.st[3][i] = make_float4(q.L.z, g.nee.x, g.nee.y, g.nee.z);
    if (rec && g.shadow) wf_record_light(R, W.rec[i], b + 1, br);
  }
  const unsigned long long j = warp_append(S.n_out, go);
  push_ray(W, S.n_ray, g.shadow, q.x.p, g.sdir, g.stmax, (unsigned)j | kAnyRay);
  push_ray(W, S.n_ray, g.cont, q.x.p, g.wi, kRayMax, (unsigned)j);
  if (go) S.out[j] = i | (g.shadow ? kCastShadow : 0u) | (g.cont ? kCastCont : 0u);
}

// Ends the path of sample p of view V.
template <int MODE>
TRN_D void wf_finish(const Wave& W, const ViewDesc& V, long long p, const F3& L, Cnt& cnt) {
  if (MODE == kWfReplay) return;
  cnt.v[kCntPixel]++;
  W.L[p + V.begin - W.first] = L;
}

// Lists the records of the paths that end here (all lanes of the warp call it).
template <int MODE>
TRN_D void wf_record_end(const Wave& W, const PathSoA& R, bool ends, unsigned i) {
  if constexpr (MODE != kWfFwd) {
    if (!R.n_end) return;
    const unsigned long long j = warp_append(R.n_end, ends);
    if (ends) R.order[j] = W.rec[i];
  }
}

// Camera rays of the round's n slots. For the adjoint (grad), slots whose pixel
// has a zero dL/dI are left out (they carry no gradient); for an image, the
// radiance of slots that end without a path is zero.
__global__ void __launch_bounds__(256, 4) k_wf_camera(TRN_KPARAMS, const __grid_constant__ Wave W, long long n, bool grad,
                            unsigned long long* n_out) {
  stage_begin();
  Cnt cnt;
  int vhint = 0;
  for_each_entry((unsigned long long)n, [&](unsigned long long k, bool in) {
    F3 org, dir;
    if (in) {
      const long long slot = W.first + (long long)k;
      const ViewDesc& V = view_of(P, slot, vhint);
      const long long p = slot - V.begin;
      const int pix = (int)(p % ((long long)V.cam.w * V.cam.h));
      if (grad) {
        cnt.v[kCntPixel]++;
        const F3 g = g_at(P, V, pix);
        in = !(g.x == 0.f && g.y == 0.f && g.z == 0.f);
      } else {
        W.L[k] = F3z();
      }
      if (in) {
        cnt.v[kCntClosest]++;
        const PathSmp S{&P, V.seed, slot, p + V.slot_off};
        org = cam_pos(V.cam);
        dir = camera_ray_dir(V.cam, pix % V.cam.w, pix / V.cam.w, S(0), S(1));
      }
    }
    const unsigned long long j = warp_append(n_out, in);
    if (in) {
      put_ray(W, j, org, dir, kRayMax, (unsigned)j);
      W.list[1][j] = (unsigned)k;
    }
  });
  flush_cnt(cnt, P.stats);
}

// Whether a view's pixels are summed by a warp each: so few pixels that a thread
// each leaves most of the GPU idle, and samples enough for a warp.
TRN_HD bool deep_pixels(long long pixels, long long samples) { return pixels <= 16384 && samples >= 32 * pixels; }

// Adds the round's radiance to the image: one thread per pixel sums its samples
// of this round in slot order (a view's samples of one pixel lie W * H slots
// apart). The image does not depend on the order in which paths end.
__global__ void __launch_bounds__(256) k_wf_pixels(TRN_KPARAMS, const __grid_constant__ Wave W, long long n) {
  stage_begin();
  int vhint = 0;
  const long long end = W.first + n;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const long long slot = W.first + k;
    const ViewDesc& V = view_of(P, slot, vhint);
    const long long WH = (long long)V.cam.w * V.cam.h;
    // the view's first W * H slots of the round stand for its pixels
    if (slot - max(W.first, V.begin) >= WH || deep_pixels(WH, V.n)) continue;
    const long long last = min(end, V.begin + V.n);
    F3 acc = F3z();
    for (long long q = slot; q < last; q += WH) acc = acc + W.L[q - W.first] * V.inv_spp;
    atomic_add3((V.image ? V.image : P.image + 3 * V.pix_off) + 3 * ((slot - V.begin) % WH), acc);
  }
}

// The same for the views with deep pixels, `per_view` blocks each: a warp per
// pixel, every 32nd sample by a lane, then the lanes in a fixed order. Bound by the
// chain of a lane's adds (16 x 16 pixels of 65,536 samples of depth 1: the image took 39 ms with a thread
// per pixel, 9.2 here, 1.2 of them in this kernel).
__global__ void __launch_bounds__(256) k_wf_deep_pixels(TRN_KPARAMS, const __grid_constant__ Wave W, long long n, int per_view) {
  stage_begin();
  const ViewDesc& V = P.views[blockIdx.x / per_view];
  if (!deep_pixels((long long)V.cam.w * V.cam.h, V.n)) return;
  const int lane = threadIdx.x & 31;
  const int WH = V.cam.w * V.cam.h;
  const long long first = max(W.first, V.begin), last = min(W.first + n, V.begin + V.n);
  for (int i = blockIdx.x % per_view * (blockDim.x >> 5) + (threadIdx.x >> 5); i < WH; i += per_view * (blockDim.x >> 5)) {
    F3 acc = F3z();
#pragma unroll 4
    for (long long q = first + i + (long long)lane * WH; q < last; q += 32ll * WH)
      acc = acc + W.L[q - W.first] * V.inv_spp;
    for (int o = 16; o > 0; o >>= 1)
      acc = acc + F3(__shfl_xor_sync(0xffffffffu, acc.x, o), __shfl_xor_sync(0xffffffffu, acc.y, o),
                     __shfl_xor_sync(0xffffffffu, acc.z, o));
    if (lane == 0 && first + i < last)
      atomic_add3((V.image ? V.image : P.image + 3 * V.pix_off) + 3 * ((first + i - V.begin) % WH), acc);
  }
}

// First vertex of every path.
template <int MODE>
__global__ void __launch_bounds__(256, 3) k_wf_start(TRN_KPARAMS, const __grid_constant__ Wave W, const __grid_constant__ Stage S,
                           const __grid_constant__ PathSoA R) {
  stage_begin();
  Cnt cnt;
  const DeviceScene& s = P.s;
  int vhint = 0;
  for_each_entry(*S.n, [&](unsigned long long k, bool in) {
    WfPath q;
    unsigned i = 0;
    const ViewDesc* V = nullptr;
    long long p = 0;
    Hit h;
    h.tri = -1;
    int D = 0;
    if (in) h = get_hit(W.hit[0], k);
    in = h.tri >= 0;
    // a state and, in the recording modes, a record for the path
    const unsigned long long j = warp_append(S.n_state, in);
    unsigned long long kr = 0;
    if (MODE != kWfFwd) {
      kr = warp_append(P.q_count, in);
      if (in && kr >= (unsigned long long)P.q_cap) { atomicExch(P.err, 2); in = false; }
    }
    if (in) {
      i = (unsigned)j;
      const long long slot = W.first + (long long)S.in[k];
      V = &view_of(P, slot, vhint);
      p = slot - V->begin;
      W.p[i] = p;
      W.view[i] = (int)(V - P.views);
      D = V->D;
      const CameraDesc& cam = V->cam;
      const F3 org = cam_pos(cam);
      q.x = post_intersect(s, h.tri, h.u, h.v);
      const float t1 = camera_factor<float>(cam, q.x.p, q.x.ng, 1.f);
      q.T = F3(t1, t1, t1);
      q.rdir = normalize(q.x.p - org);
      const F3 m1 = emitted(s, q.x, -q.rdir);
      if (MODE == kWfFwd) {
        q.L = scrub(q.T * m1);
      } else {
        W.rec[i] = (unsigned)kr;
        const F3 m = finite3(q.T * m1) ? m1 : F3z();
        q.L = q.T * m;
        R.p(kr) = p; R.view(kr) = (int)(V - P.views);
        R.g(kr) = MODE == kWfReplay ? g_at(P, *V, (int)(p % ((long long)cam.w * cam.h))) : F3z();
        R.vr(kr, 1) = {h.tri, h.u, h.v};
        R.Tk(kr, 1) = q.T;
        R.Mk(kr, 1) = m;
        R.K(kr) = 1; R.D(kr) = D; R.nee(kr) = 0u;
      }
    }
    const bool go = in && D > 0;
    if (in && !go) wf_finish<MODE>(W, *V, p, q.L, cnt);
    wf_record_end<MODE>(W, R, in && !go, i);
    wf_advance<MODE>(P, W, S, 0, go, i, V, p, q, R, cnt);
  });
  flush_cnt(cnt, P.stats);
}

// One bounce: ends bounce S.b with its ray results, and decides the rays of the
// next for the paths that go on. Bound by the gathers of the two vertices
// (latency) and the state traffic; 32 paths of a warp take the same branches
// but for material and light.
// TAIL: runs those paths to their ends instead, one thread each, with the fused
// bounce, for the late bounces of few paths (WaveRun::tail_bounce). Bound by the
// chain of the longest path: its paths are spread over all warps (12,288 samples
// of depth 5 on 1,284 triangles: 236 us packed, 163 spread).
template <int MODE, bool TAIL>
__global__ void __launch_bounds__(256, 3) k_wf_shade(TRN_KPARAMS, const __grid_constant__ Wave W, const __grid_constant__ Stage S,
                           const __grid_constant__ PathSoA R) {
  stage_begin();
  Cnt cnt;
  const DeviceScene& s = P.s;
  constexpr bool rec = MODE != kWfFwd;
  const int b = S.b;
  auto each = [&](unsigned long long idx, bool in) {
    WfPath q;
    unsigned i = 0;
    const ViewDesc* V = nullptr;
    long long p = 0;
    bool go = false;
    if (in) {
      const unsigned e = __ldcs(S.in + idx);
      i = e & kEntryMask;
      const bool nee_ok = (e & kCastShadow) && !W.occ[idx];
      Hit h;
      h.tri = -1;
      if (e & kCastCont) h = get_hit(W.hit[0], idx);
      const float4 a = W.st[0][i], c1 = W.st[1][i], c2 = W.st[2][i], c3 = W.st[3][i];
      p = W.p[i];
      V = P.views + W.view[i];
      q.rdir = F3(c1.x, c1.y, c1.z);
      q.T = F3(c1.w, c2.x, c2.y);
      q.L = F3(c2.z, c2.w, c3.x);
      q.x = post_intersect(s, __float_as_int(a.x), a.y, a.z);
      F3 c;
      BounceRec br;
      const bool more = radiance_resolve(s, q.x, [&] { return shading_at(s, q.x); }, q.rdir, q.T, nee_ok, F3(c3.y, c3.z, c3.w), a.w, h, c, rec ? &br : nullptr);
      q.L = q.L + c;
      if constexpr (rec) wf_record(R, W.rec[i], b + 1, br, more, q);
      go = more && !is_dark(q.T) && b + 1 < V->D;
      if constexpr (TAIL) {
        const PathSmp smp{&P, V->seed, p + V->begin, p + V->slot_off};
        for (int t = b + 1; go; t++) {
          const int o = 2 + 5 * t;
          const bool on = radiance_step(s, q.x, q.rdir, q.T, smp(o), smp(o + 1), smp(o + 2), smp(o + 3), smp(o + 4), c,
                                        rec ? &br : nullptr, cnt);
          q.L = q.L + c;
          if constexpr (rec) {
            if (br.nee_ok) wf_record_light(R, W.rec[i], t + 1, br);
            wf_record(R, W.rec[i], t + 1, br, on, q);
          }
          go = on && !is_dark(q.T) && t + 1 < V->D;
        }
      }
      if (!go) wf_finish<MODE>(W, *V, p, q.L, cnt);
    }
    wf_record_end<MODE>(W, R, in && !go, i);
    if constexpr (!TAIL) wf_advance<MODE>(P, W, S, b + 1, go, i, V, p, q, R, cnt);
  };
  if constexpr (TAIL) for_each_spread(*S.n, each);
  else for_each_entry(*S.n, each);
  flush_cnt(cnt, P.stats);
}

// ---------------------------------------------------------------------------
// boundary set-ups: a ray per sample, a second ray for the samples whose first
// one hit, and the boundary geometry for those that are left
// ---------------------------------------------------------------------------
// Whether every sample keeps its place in the ray queues, with a ray that hits
// nothing where it has none. Most samples of the indirect term have both rays. In
// compacted queues, each filled in the order in which warps come, neighbours in the
// run order (one edge, nearby directions) moved apart twice more before the items,
// fewer lanes of a body's warp then ended together, and more of the term's small
// adds were lost beside the direct term's large ones: nearly cancelling components
// moved by 0.5 % of the 16.8M-sample gradient's RMS (two runs 0.1 %). The term takes
// the same time either way (30.4 ms).
template <int TERM>
constexpr bool kSetupInPlace = TERM == TRN_INDIRECT_EDGE;

// First rays of the round's samples in run order (slot_at); list[0][ray id] is
// the sample's offset in the round.
template <int TERM>
__global__ void __launch_bounds__(256, 4) k_setup_rays(TRN_KPARAMS, const __grid_constant__ Wave W, long long first, unsigned long long* n_ray) {
  stage_begin();
  Cnt cnt;
  int vhint = 0;
  const unsigned long long n = (unsigned long long)(P.total - first);
  for_each_entry(n, [&](unsigned long long k, bool in) {
    long long slot = 0;
    F3 o, d;
    if (in) {
      slot = slot_at(P, first + (long long)k);
      if constexpr (TERM == TRN_PRIMARY_EDGE) {
        EdgePoint q;
        in = primary_point(P, slot, q, vhint);
        if (in) { cnt.v[kCntClosest]++; o = q.p0; d = q.dir; }
      } else if constexpr (TERM == TRN_DIRECT_EDGE) {
        DirectPoint q;
        in = direct_point(P, slot, q, vhint, cnt);
        if (in) { o = q.e.p0; d = q.e.dir; }
      } else if constexpr (TERM == TRN_INDIRECT_EDGE) {
        EdgePoint q;
        in = indirect_point(P, slot, q, vhint);
        if (in) { cnt.v[kCntClosest] += 2; o = q.p0; d = -q.dir; }
      } else {
        PixelPoint q;
        pixel_point(P, slot, q, vhint);
        cnt.v[kCntClosest]++;
        o = q.p0; d = q.dir;
      }
    }
    if constexpr (kSetupInPlace<TERM>) {
      if (k >= n) return;
      put_ray(W, k, in ? o : F3z(), in ? d : F3z(), kRayMax, (unsigned)k);  // (no direction: hits nothing)
      W.list[0][k] = (unsigned)(slot - first);
      if (k == 0) *n_ray = n;
    } else {
      const unsigned long long j = warp_append(n_ray, in);
      if (in) {
        put_ray(W, j, o, d, kRayMax, (unsigned)j);
        W.list[0][j] = (unsigned)(slot - first);
      }
    }
  });
  flush_cnt(cnt, P.stats);
}

// Second rays, behind the first ones in the ray queue; list[1][second ray id]
// is the first ray's id.
template <int TERM>
__global__ void __launch_bounds__(256, 4) k_setup_rays2(TRN_KPARAMS, const __grid_constant__ Wave W, long long first, const unsigned long long* n_ray,
                              unsigned long long* n_ray2) {
  stage_begin();
  Cnt cnt;
  int vhint = 0;
  const unsigned long long n = *n_ray;
  for_each_entry(n, [&](unsigned long long k, bool in) {
    F3 o, d;
    float tmax = kRayMax;
    if (in) {
      const Hit h = get_hit(W.hit[0], k);
      in = h.tri >= 0;
      if (in) {
        if constexpr (TERM == TRN_DIRECT_EDGE) {
          DirectPoint q;
          Cnt again;  // counted by the first pass
          direct_point(P, first + W.list[0][k], q, vhint, again);
          in = direct_lit(q, h.t);
          o = q.e.p0; d = -q.e.dir;
        } else {
          const float4 a = __ldcs(W.ro + k), b = __ldcs(W.rd + k);
          o = F3(a.x, a.y, a.z); d = F3(b.x, b.y, b.z);
          if constexpr (TERM == TRN_PRIMARY_EDGE) {
            const CameraDesc& cam = view_of(P, first + W.list[0][k], vhint).cam;
            SensorSample sds;
            F3 dirc;
            in = primary_sensor(cam, o, d, h.t, sds, dirc, tmax);
            o = cam_pos(cam); d = dirc;
            if (in) cnt.v[kCntShadow]++;
          } else {
            d = -d;
          }
        }
      }
    }
    if constexpr (kSetupInPlace<TERM>) {
      if (k >= n) return;
      put_ray(W, (unsigned long long)W.cap + k, in ? o : F3z(), in ? d : F3z(), kRayMax, (unsigned)k);
      W.list[1][k] = (unsigned)k;
      if (k == 0) *n_ray2 = n;
    } else {
      const unsigned long long j = warp_append(n_ray2, in);
      if (in) {
        put_ray(W, (unsigned long long)W.cap + j, o, d, tmax, (unsigned)j | (TERM == TRN_PRIMARY_EDGE ? kAnyRay : 0u));
        W.list[1][j] = (unsigned)k;
      }
    }
  });
  flush_cnt(cnt, P.stats);
}

// Queues the boundary samples of the lanes that have one as the term's items
// (all lanes of the warp call it).
template <int TERM>
TRN_D void queue_item(const Params& P, const EdgeState& st, bool in) {
  const unsigned long long j = warp_append(P.q_count, in);
  if (in && j >= (unsigned long long)P.q_cap) { atomicExch(P.err, 2); in = false; }
  if (!in) return;
  if constexpr (TERM == TRN_DIRECT_EDGE) {
    DirectItem& it = reinterpret_cast<DirectItem*>(P.queue)[j];
    it.p = st.p; it.view = (int)(st.V - P.views);
    it.x_tri = st.x.tri; it.x_u = st.x.u; it.x_v = st.x.v; it.v0 = st.v0; it.v1 = st.v1; it.far_tri = st.far_tri;
    it.sedge = st.sedge; it.rdir = st.rdir; it.ev0 = st.T0 * st.w0; it.p0 = st.p0; it.n = st.n;
  } else if constexpr (TERM == TRN_INDIRECT_EDGE) {
    IndirectItem& it = reinterpret_cast<IndirectItem*>(P.queue)[j];
    it.p_lo = (unsigned)st.p; it.p_hi = (int)(st.p >> 32); it.view = (int)(st.V - P.views);
    it.xe_tri = st.xe.tri; it.xe_u = st.xe.u; it.xe_v = st.xe.v;
    it.xs_tri = st.x.tri; it.xs_u = st.x.u; it.xs_v = st.x.v;
    it.v0 = st.v0; it.v1 = st.v1; it.far_tri = st.far_tri; it.w0 = st.w0; it.sedge = st.sedge;
    it.rdir = st.rdir; it.p0 = st.p0; it.n = st.n;
  } else {
    constexpr bool pixel = TERM == TRN_PIXEL_EDGE;
    PrimaryItem& it = reinterpret_cast<PrimaryItem*>(P.queue)[j];
    it.p = st.p; it.view = (int)(st.V - P.views);
    it.x_tri = st.x.tri; it.x_u = st.x.u; it.x_v = st.x.v; it.T0 = st.T0.x; it.w0 = st.w0;
    it.sedge = pixel ? 0.f : st.sedge;
    it.v0 = pixel ? -1 : st.v0; it.v1 = pixel ? -1 : st.v1;  // a pixel-edge point is no scene parameter
    it.far_tri = st.far_tri;
    it.rdir = st.rdir; it.p0 = st.p0; it.n = st.n; it.g = st.g;
  }
}

// Boundary geometry of the samples whose rays allow one, queued as the term's
// items. n: the rays of the last query (the pixel term has only one).
template <int TERM>
__global__ void __launch_bounds__(256, 3) k_setup_finish(TRN_KPARAMS, const __grid_constant__ Wave W, long long first, const unsigned long long* n) {
  stage_begin();
  int vhint = 0;
  for_each_entry(*n, [&](unsigned long long k2, bool in) {
    EdgeState st;
    if (in) {
      const unsigned long long k = TERM == TRN_PIXEL_EDGE ? k2 : W.list[1][k2];
      if constexpr (TERM == TRN_PRIMARY_EDGE) in = !W.occ[k2];
      Hit h2;
      if constexpr (TERM == TRN_DIRECT_EDGE || TERM == TRN_INDIRECT_EDGE) {
        h2 = get_hit(W.hit[1], k2);
        in = h2.tri >= 0;
      }
      if (in) {
        const Hit h = get_hit(W.hit[0], k);
        in = h.tri >= 0;
        const long long slot = first + W.list[0][k];
        if (in) {
          if constexpr (TERM == TRN_PRIMARY_EDGE) {
            EdgePoint q;
            primary_point(P, slot, q, vhint);
            SensorSample sds;
            F3 dirc;
            float tmax;
            primary_sensor(q.V->cam, q.p0, q.dir, h.t, sds, dirc, tmax);
            in = primary_finish(P, slot, q, h, sds, dirc, st);
          } else if constexpr (TERM == TRN_DIRECT_EDGE) {
            DirectPoint q;
            Cnt again;
            direct_point(P, slot, q, vhint, again);
            in = direct_finish(P, slot, q, h, h2, st);
          } else if constexpr (TERM == TRN_INDIRECT_EDGE) {
            EdgePoint q;
            indirect_point(P, slot, q, vhint);
            in = indirect_finish(P, slot, q, h, h2, st);
          } else {
            PixelPoint q;
            pixel_point(P, slot, q, vhint);
            in = pixel_finish(P, q, h, st);
          }
        }
      }
    }
    queue_item<TERM>(P, st, in);
  });
}

// The whole direct set-up by one thread per slot, for small rounds: most slots
// end before their first ray (the edge lies wrong for the light), and the
// launches between the rays then cost more than the lanes that wait. The term
// at depth 3 in the wavefront's launches / here, us, on 1,284 and on 102,400
// triangles: 12,288 slots 204 / 186 and 334 / 323, 393,216 287 / 265 and 499 /
// 436, 1,048,576 342 / 365 and 577 / 557; 16.8M slots of depth 5 on 102,400
// triangles 2,200 / 3,430.
__global__ void __launch_bounds__(256, 4) k_setup_direct(TRN_KPARAMS, long long first) {
  stage_begin();
  Cnt cnt;
  int vhint = 0;
  for_each_entry((unsigned long long)(P.total - first), [&](unsigned long long k, bool in) {
    EdgeState st;
    in = in && direct_setup(P, slot_at(P, first + (long long)k), st, vhint, cnt);
    queue_item<TRN_DIRECT_EDGE>(P, st, in);
  });
  flush_cnt(cnt, P.stats);
}

// ---------------------------------------------------------------------------
// guiding samples of the direct boundary term: |baseVal| of `per` samples in
// each leaf of the guiding tree (guide_base_val, one ray query per launch).
// One thread per leaf traced all of its samples' rays one after the other, with
// a few thousand threads in all: an inverse-rendering step of four views with
// guiding took 43 ms and takes 17 with a slot per sample.
// ---------------------------------------------------------------------------
struct GuideTree {
  const float* box;       // [6][cap]
  const int* edge;
  const int* count;       // leaves
  long long cap;
  uint32_t stream;
  int per;                // samples per leaf
};

// Sample point of (leaf, k): uniform in the leaf's box, or (EVAL) the
// refinement's evaluation point.
template <bool EVAL>
TRN_D bool guide_sample(const Params& P, const GuideTree& g, long long t, DirectPoint& q) {
  const int leaf = (int)(t / g.per), k = (int)(t % g.per);
  if (leaf >= __ldg(g.count) || !(P.efunc[g.edge[leaf]] > 0.f) || !(__ldg(P.eint) > 0.f)) return false;
  float x[3];
  if (EVAL) {
    aq_point(g.box, g.cap, leaf, k, g.stream, x);
  } else {
    for (int a = 0; a < 3; a++)
      x[a] = aq_lerp(g.box, g.cap, leaf, a, hash_uniform(g.stream, kGuideTerm, (uint32_t)a, (uint32_t)t));
  }
  return guide_point(P, x[0], x[1], x[2], q);
}

// Rays from the edge points to the light points of samples [first, first + n);
// value[] of the round starts at 0.
template <bool EVAL>
__global__ void __launch_bounds__(256, 4) k_guide_rays(TRN_KPARAMS, const __grid_constant__ Wave W, const __grid_constant__ GuideTree g,
                             long long first, long long n, float* value, unsigned long long* n_ray) {
  stage_begin();
  for_each_entry((unsigned long long)n, [&](unsigned long long k, bool in) {
    DirectPoint q;
    if (in) {
      value[k] = 0.f;
      in = guide_sample<EVAL>(P, g, first + (long long)k, q);
    }
    const unsigned long long j = warp_append(n_ray, in);
    if (in) {
      put_ray(W, j, q.e.p0, q.e.dir, kRayMax, (unsigned)j);
      W.list[0][j] = (unsigned)k;
    }
  });
}

// Rays away from the light, for the samples whose first ray met the light point.
template <bool EVAL>
__global__ void __launch_bounds__(256, 4) k_guide_rays2(TRN_KPARAMS, const __grid_constant__ Wave W, const __grid_constant__ GuideTree g,
                              long long first, const unsigned long long* n_ray, unsigned long long* n_ray2) {
  stage_begin();
  for_each_entry(*n_ray, [&](unsigned long long k, bool in) {
    DirectPoint q;
    if (in) {
      const Hit h = get_hit(W.hit[0], k);
      in = h.tri >= 0;
      if (in) {
        guide_sample<EVAL>(P, g, first + W.list[0][k], q);
        in = direct_lit(q, h.t);
      }
    }
    const unsigned long long j = warp_append(n_ray2, in);
    if (in) {
      put_ray(W, (unsigned long long)W.cap + j, q.e.p0, -q.e.dir, kRayMax, (unsigned)j);
      W.list[1][j] = W.list[0][k];
    }
  });
}

template <bool EVAL>
__global__ void __launch_bounds__(256, 4) k_guide_values(TRN_KPARAMS, const __grid_constant__ Wave W, const __grid_constant__ GuideTree g,
                               long long first, const unsigned long long* n_ray2, float* value) {
  stage_begin();
  const unsigned long long n = *n_ray2;
  for (unsigned long long j = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; j < n;
       j += (unsigned long long)gridDim.x * blockDim.x) {
    const Hit h = get_hit(W.hit[1], j);
    if (h.tri < 0) continue;
    DirectPoint q;
    guide_sample<EVAL>(P, g, first + W.list[1][j], q);
    value[W.list[1][j]] = guide_value(P, q, h);
  }
}

// Leaf weights of the round's leaves: the mean of their values, added in order.
__global__ void k_guide_mean(const int* count, int per, long long leaf0, long long n_leaf, const float* value, float* poly) {
  stage_begin();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n_leaf || leaf0 + i >= __ldg(count)) return;
  const float fs = (float)per;
  float acc = 0.f;
  for (int k = 0; k < per; k++) acc = __fadd_rn(acc, __fdiv_rn(value[i * per + k], fs));
  poly[leaf0 + i] = acc;
}
