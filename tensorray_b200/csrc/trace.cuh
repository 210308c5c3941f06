// Ray queries against the project's BVH: closest hit and occlusion.
//
// Replaces the OptiX ray-query seam RayIntersectOptix (LibTensorRay/Renderer/
// Optix.cpp:252-305) and its programs (ptx.cu:61-113). Hit semantics:
//   * a hit is a triangle whose watertight intersection (Woop, Benthin and
//     Wald, "Watertight Ray/Triangle Intersection", JCGT 2013) has
//     tmin < t < tmax, both faces count (no culling, like OptiX's default);
//   * the closest hit is the lexicographic minimum of (t, triangle id), so the
//     result does not depend on traversal order;
//   * a miss returns triangle -1 (ptx.cu:61-113 writes -1 on a miss);
//   * Scene::Occluded (Scene.cpp:548-562) is "no hit inside (tmin, tmax)".
// The triangle test is written with explicitly rounded float operations so it
// is bit-identical to the CPU restatement of the same formula.
#pragma once
#include "scene_types.cuh"

namespace trn {

struct Hit {
  int tri;
  float u, v, t;  // u weights P1, v weights P2 (Scene.cpp:677-684)
};

// Two floats for the packed multiply-add (one instruction for both).
struct Pair { float a, b; };
TRN_D Pair fma2(const Pair& x, const Pair& y, const Pair& z) {
  Pair r;
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  asm("{\n\t.reg .b64 x, y, z, r;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 r, x, y, z;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.a), "=f"(r.b) : "f"(x.a), "f"(x.b), "f"(y.a), "f"(y.b), "f"(z.a), "f"(z.b));
#else
  r.a = fmaf(x.a, y.a, z.a);
  r.b = fmaf(x.b, y.b, z.b);
#endif
  return r;
}

// The shear of the watertight triangle test.
struct RayShear {
  F3 o;
  int kx, ky, kz;
  float sx, sy, sz;
};

TRN_D void ray_shear(RayShear& r, const F3& o, const F3& d) {
  r.o = o;
  float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  int kz = 0; float m = ax;
  if (ay > m) { kz = 1; m = ay; }
  if (az > m) { kz = 2; }
  int kx = kz + 1; if (kx == 3) kx = 0;
  int ky = kx + 1; if (ky == 3) ky = 0;
  if (d[kz] < 0.f) { int t = kx; kx = ky; ky = t; }
  r.kx = kx; r.ky = ky; r.kz = kz;
  r.sx = __fdiv_rn(d[kx], d[kz]);
  r.sy = __fdiv_rn(d[ky], d[kz]);
  r.sz = __fdiv_rn(1.f, d[kz]);
}

// reciprocal direction for the box slabs (culling only)
TRN_D float ray_inv(float d) { return 1.f / (fabsf(d) < 1e-20f ? copysignf(1e-20f, d) : d); }

// A ray with its reciprocal direction (one ray per thread).
struct RayInv : RayShear { F3 inv; };

TRN_D RayInv ray_inverse(const F3& o, const F3& d) {
  RayInv r;
  ray_shear(r, o, d);
  r.inv = F3(ray_inv(d.x), ray_inv(d.y), ray_inv(d.z));
  return r;
}

// A ray with the origin folded into the slabs (the stream traversal): the
// distances of an axis' two planes are one packed multiply-add, (lo, hi) * inv +
// c. c holds -o * inv, moved by |o * inv| 2^-22 away from the box (down for the
// plane that is entered, up for the one that is left): more than the rounding of
// o * inv and of its product, so that a box is never missed (see `slab`).
struct RayPre : RayShear {
  Pair ix, iy, iz, cx, cy, cz;
};

TRN_D RayPre ray_setup(const F3& o, const F3& d) {
  RayPre r;
  ray_shear(r, o, d);
  auto axis = [&](float o, float d, Pair& inv, Pair& c) {
    inv.a = inv.b = ray_inv(d);
    const float k = -(o * inv.a), e = fabsf(k) * 2.384185791015625e-7f;  // 2^-22
    c.a = inv.a < 0.f ? k + e : k - e;
    c.b = inv.a < 0.f ? k - e : k + e;
  };
  axis(o.x, d.x, r.ix, r.cx);
  axis(o.y, d.y, r.iy, r.cy);
  axis(o.z, d.z, r.iz, r.cz);
  return r;
}

// Woop et al. 2013, section 3 (algorithm of figure 1), with the double
// precision fallback when an edge function is exactly zero.
TRN_D bool intersect_tri(const RayShear& r, const F3& p0, const F3& p1, const F3& p2,
                         float tmin, float tmax, float& t_out, float& u_out, float& v_out) {
  F3 A(__fsub_rn(p0.x, r.o.x), __fsub_rn(p0.y, r.o.y), __fsub_rn(p0.z, r.o.z));
  F3 B(__fsub_rn(p1.x, r.o.x), __fsub_rn(p1.y, r.o.y), __fsub_rn(p1.z, r.o.z));
  F3 C(__fsub_rn(p2.x, r.o.x), __fsub_rn(p2.y, r.o.y), __fsub_rn(p2.z, r.o.z));
  const float Akz = A[r.kz], Bkz = B[r.kz], Ckz = C[r.kz];
  const float Ax = __fsub_rn(A[r.kx], __fmul_rn(r.sx, Akz));
  const float Ay = __fsub_rn(A[r.ky], __fmul_rn(r.sy, Akz));
  const float Bx = __fsub_rn(B[r.kx], __fmul_rn(r.sx, Bkz));
  const float By = __fsub_rn(B[r.ky], __fmul_rn(r.sy, Bkz));
  const float Cx = __fsub_rn(C[r.kx], __fmul_rn(r.sx, Ckz));
  const float Cy = __fsub_rn(C[r.ky], __fmul_rn(r.sy, Ckz));
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.f || V == 0.f || W == 0.f) {
    U = (float)__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx));
    V = (float)__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx));
    W = (float)__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax));
  }
  if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
  const float det = __fadd_rn(__fadd_rn(U, V), W);
  if (det == 0.f) return false;
  const float Az = __fmul_rn(r.sz, Akz);
  const float Bz = __fmul_rn(r.sz, Bkz);
  const float Cz = __fmul_rn(r.sz, Ckz);
  const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
  const float rcp = __fdiv_rn(1.f, det);
  const float t = __fmul_rn(T, rcp);
  if (!(t > tmin && t < tmax)) return false;
  t_out = t;
  u_out = __fmul_rn(V, rcp);
  v_out = __fmul_rn(W, rcp);
  return true;
}

// ---- box steps ---------------------------------------------------------------
// What bounds traversal here is instruction issue and the L1's data path (one
// lane's line per cycle and SM). The stream traversal fetches a node in two
// 32-byte loads and a triangle in two; its plane distances are one multiply-add
// each and the slab's extremes three-input min/max.
TRN_D float max3(float a, float b, float c) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fmaxf(fmaxf(a, b), c);
#endif
}
TRN_D float min3(float a, float b, float c) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
#else
  return fminf(fminf(a, b), c);
#endif
}

// 32 bytes at a 32-byte aligned address in one load. (Not in the fused kernels:
// ptxas 12.9 crashes on it where registers are spilled.)
TRN_D void load8(const void* p, float4& a, float4& b) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
#else
  a = static_cast<const float4*>(p)[0];
  b = static_cast<const float4*>(p)[1];
#endif
}

// traversal states beside the node to visit next (>= 0 inner, < 0 leaf)
constexpr int kTraceDone = 0x7fffffff;  // nothing left
constexpr int kTracePop = 0x7ffffffe;   // the stack's next entry

// One box (lo, hi per axis) against the ray's interval [tmin, tmax]. Culling is
// conservative: the ray's c covers the origin's share of the rounding, boxes
// are padded at build time, and for the relative error of at most 2^-23 per
// distance (reciprocal and final rounding) the far distance gets a slack of
// 4e-7.
TRN_D bool slab(const RayPre& r, const Pair& bx, const Pair& by, const Pair& bz, float tmin, float tmax, float& tnear) {
  const Pair x = fma2(bx, r.ix, r.cx), y = fma2(by, r.iy, r.cy), z = fma2(bz, r.iz, r.cz);
  tnear = fmaxf(max3(fminf(x.a, x.b), fminf(y.a, y.b), fminf(z.a, z.b)), tmin);
  const float tf = fminf(min3(fmaxf(x.a, x.b), fmaxf(y.a, y.b), fmaxf(z.a, z.b)), tmax);
  return tnear <= tf * 1.0000004f;
}

// The same with an axis at a time and no slack in the ray.
TRN_D bool slab(const RayInv& r, float lx, float hx, float ly, float hy, float lz, float hz, float tmin, float tmax,
                float& tnear) {
  const float x0 = (lx - r.o.x) * r.inv.x, x1 = (hx - r.o.x) * r.inv.x;
  const float y0 = (ly - r.o.y) * r.inv.y, y1 = (hy - r.o.y) * r.inv.y;
  const float z0 = (lz - r.o.z) * r.inv.z, z1 = (hz - r.o.z) * r.inv.z;
  tnear = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fmaxf(fminf(z0, z1), tmin));
  const float tf = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fminf(fmaxf(z0, z1), tmax));
  return tnear <= tf * 1.0000004f;
}

// Traversal stack of the stream: entries are (child, bits of its box's entry
// distance).
// The stream traversal's first entries lie in shared memory: the lanes of a
// warp stand at different depths, and an access to local memory then takes a
// pass through the L1 for every depth among them, where here each lane has its
// own banks (672 -> 580 us for 2^20 rays). Deeper entries are rare.
#ifndef TRN_SHARED_STACK
#define TRN_SHARED_STACK 12
#endif
#ifndef TRN_TRACE_BLOCK
#define TRN_TRACE_BLOCK 128
#endif
struct SharedStack {
  int2* top;                                 // this thread's column
  int2 e[kStackSize - TRN_SHARED_STACK];
  TRN_D void set(int i, int2 v) {
    if (i < TRN_SHARED_STACK) top[i * TRN_TRACE_BLOCK] = v;
    else e[i - TRN_SHARED_STACK] = v;
  }
  TRN_D int2 get(int i) const { return i < TRN_SHARED_STACK ? top[i * TRN_TRACE_BLOCK] : e[i - TRN_SHARED_STACK]; }
};
TRN_D int2* shared_stack() {
  __shared__ int2 s[TRN_SHARED_STACK * TRN_TRACE_BLOCK];
  return s + threadIdx.x;
}

// Farthest entry distance that can still matter. (A popped entry whose box
// starts behind the closest hit is dropped without a fetch.)
TRN_D float pop_limit(float best_t) { return best_t + fabsf(best_t) * 4e-7f; }

// One box step. Returns the nearer child that is hit (inner node >= 0, leaf <
// 0) or kTracePop; the farther one goes to the stack as (child, bits of its
// entry distance). Straight-line code: lanes of a warp differ in which children
// they hit, and every branch would run once more per warp.
template <class Stack>
TRN_D int visit_node(const DeviceScene& s, const RayPre& r, int node, float tmin, float best_t, Stack& stack, int& sp,
                     int* err) {
  const char* n = reinterpret_cast<const char*>(s.nodes) + ((size_t)(unsigned)node << 6);
  float4 a, b, c, d;
  load8(n, a, b);
  load8(n + 32, c, d);
  float t0, t1;
  const bool h0 = slab(r, {a.x, a.y}, {a.z, a.w}, {b.x, b.y}, tmin, best_t, t0);
  const bool h1 = slab(r, {b.z, b.w}, {c.x, c.y}, {c.z, c.w}, tmin, best_t, t1);
  const int c0 = __float_as_int(d.x), c1 = __float_as_int(d.y);
  const bool both = h0 && h1;
  const bool second = h1 && (!h0 || t1 < t0);   // the nearer one is child 1
  if (both) {
    stack.set(sp, make_int2(second ? c0 : c1, __float_as_int(second ? t0 : t1)));
    sp++;
    if (sp >= kStackSize) {  // (the build's bound on the height excludes it)
      sp = kStackSize - 1;
      if (err) atomicExch(err, 1);
    }
  }
  return h0 || h1 ? (second ? c1 : c0) : kTracePop;
}

// One attempt to take the next entry.
template <class Stack>
TRN_D void pop_entry(const Stack& stack, int& sp, float limit, int& cur) {
  if (cur == kTracePop) {
    sp--;
    const int2 e = stack.get(max(sp, 0));
    cur = sp < 0 ? kTraceDone : (__int_as_float(e.y) <= limit ? e.x : kTracePop);
  }
}

// The triangle of a leaf, read in two loads (WIDE) or three.
template <bool WIDE>
TRN_D void leaf_tri(const DeviceScene& s, int leaf, F3& p0, F3& p1, F3& p2, int& tri) {
  const char* q = reinterpret_cast<const char*>(s.tri_verts) + ((size_t)(unsigned)leaf << 6);
  float4 a, b;
  if (WIDE) {
    load8(q, a, b);
  } else {
    a = __ldg(reinterpret_cast<const float4*>(q));
    b = __ldg(reinterpret_cast<const float4*>(q) + 1);
  }
  const float2 c = __ldg(reinterpret_cast<const float2*>(q + 32));
  p0 = F3(a.x, a.y, a.z); tri = __float_as_int(a.w);
  p1 = F3(b.x, b.y, b.z); p2 = F3(b.w, c.x, c.y);
}

// A ray that can meet no triangle: any NaN makes every edge function NaN, and
// a zero direction has no largest axis. (The box tests above would let such a
// ray into every node.)
TRN_D bool ray_is_void(const F3& o, const F3& d) {
  return isnan(o.x) || isnan(o.y) || isnan(o.z) || isnan(d.x) || isnan(d.y) || isnan(d.z) ||
         (d.x == 0.f && d.y == 0.f && d.z == 0.f);
}

// Closest hit (ANY == false) or occlusion (ANY == true) of one ray by one
// thread. Returns true on hit. The stack holds nodes alone and the slab is the
// plain one: next to the stream traversal's steps this is a shorter chain for a
// lone ray and half the local memory for a fused kernel (allocation-free terms
// of 1M samples of depth 12 on 102,400 triangles with the stream's steps and
// here, in ms: interior 11.0 and 9.8, primary 7.0 and 5.5, indirect 15.0 and
// 12.5, pixel 4.2 and 3.1).
template <bool ANY>
TRN_D bool trace(const DeviceScene& s, const F3& o, const F3& d, float tmin, float tmax, Hit& hit,
                 int* err = nullptr) {
  hit.tri = -1; hit.u = 0.f; hit.v = 0.f; hit.t = -1.f;
  if (s.nt <= 0 || ray_is_void(o, d)) return false;
  const RayInv r = ray_inverse(o, d);
  float best_t = tmax;
  int best_tri = -1;
  int stack[kStackSize];
  int sp = 0, cur = s.nt == 1 ? ~0 : 0;
  // leaves are visited through the loop like inner nodes, so the triangle
  // test is instantiated once per traversal (smaller code)
  for (;;) {
    if (cur < 0) {
      F3 p0, p1, p2; int tri;
      leaf_tri<false>(s, ~cur, p0, p1, p2, tri);
      float t, u, v;
      // best_tri = -1 before the first hit: a hit at exactly the ray's end is none
      if (intersect_tri(r, p0, p1, p2, tmin, INFINITY, t, u, v) && (t < best_t || (t == best_t && tri < best_tri))) {
        best_t = t; best_tri = tri; hit.u = u; hit.v = v;
        if (ANY) break;
      }
      if (sp == 0) break;
      cur = stack[--sp];
      continue;
    }
    const BvhNode* n = &s.nodes[cur];
    const float4 a = __ldg(&n->a), b = __ldg(&n->b), c = __ldg(&n->c);
    const int4 e = __ldg(&n->d);
    float t0, t1;
    const bool h0 = slab(r, a.x, a.y, a.z, a.w, b.x, b.y, tmin, best_t, t0);
    const bool h1 = slab(r, b.z, b.w, c.x, c.y, c.z, c.w, tmin, best_t, t1);
    if (h0 && h1) {
      const bool second = t1 < t0;   // the nearer one is child 1
      if (sp < kStackSize) stack[sp++] = second ? e.x : e.y;  // (the build's bound on the height excludes the rest)
      else if (err) atomicExch(err, 1);
      cur = second ? e.y : e.x;
    } else if (h0 || h1) {
      cur = h0 ? e.x : e.y;
    } else {
      if (sp == 0) break;
      cur = stack[--sp];
    }
  }
  if (best_tri < 0) return false;
  hit.tri = best_tri; hit.t = best_t;
  return true;
}

TRN_D bool occluded(const DeviceScene& s, const F3& o, const F3& d, float tmin, float tmax) {
  Hit h;
  return trace<true>(s, o, d, tmin, tmax, h);
}

// ---- many rays by one warp ---------------------------------------------------
// Traversal of a stream of rays by a whole warp. A lane whose ray has ended
// takes the next ray as soon as TRN_REFILL lanes are free, instead of waiting
// for the warp's longest ray. A ray visits about ten nodes for each triangle
// it tests, so a lane that meets a leaf puts it aside and goes on with its
// nodes until it meets a second one; the warp turns to the triangles when
// TRN_LEAF_SHARE / 4 of its busy lanes have one. Between those decisions lie
// TRN_NODE_STEPS box steps of straight-line code.
//
// Bound by instruction issue and the L1 (62 % each of their peaks, 14 of 32
// lanes active; one ray per thread left 5 to 8). 2^20 rays against 102,400
// triangles: closest hit 814 us with one ray per thread, 564 here; occlusion
// 587 and 502. Of the steps on the way: one step per turn and a vote between
// nodes and triangles 672, stacks in shared memory 580, four steps a turn 564
// (six 589); stacks of 8 and 16 shared entries are no better than 12.
//   fetch(k, lim, more)  warp-uniform: the first of k new rays; rays at or above
//                        lim are not among them; more: a later fetch has rays
//   load(i, o, d, tmin, tmax, any)   ray i
//   store(i, any, tri, u, v, t)      its result (tri < 0: no hit)
#ifndef TRN_REFILL
#define TRN_REFILL 8
#endif
#ifndef TRN_LEAF_SHARE
#define TRN_LEAF_SHARE 1
#endif
#ifndef TRN_NODE_STEPS
#define TRN_NODE_STEPS 4
#endif

template <class Fetch, class Load, class Store>
TRN_D void trace_stream(const DeviceScene& s, Fetch&& fetch, Load&& load, Store&& store, int* err) {
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
  RayPre r;
  float tmin = 0.f, best_t = 0.f, bu = 0.f, bv = 0.f;
  // leaf: the leaf put aside (< 0), else 0
  int best_tri = -1, cur = kTraceDone, leaf = 0, sp = 0;
  int id = -1;  // -1: no result to store
  bool any = false, more = s.nt > 0;
  SharedStack stack;
  stack.top = shared_stack();
  for (;;) {
    const bool free_ = cur == kTraceDone && leaf == 0;
    const unsigned idle = __ballot_sync(0xffffffffu, free_);
    if (idle == 0xffffffffu || (more && __popc(idle) >= TRN_REFILL)) {
      // results are stored when their lanes get new rays: together
      if (free_ && id >= 0) {
        store(id, any, best_tri, bu, bv, best_tri < 0 ? -1.f : best_t);
        id = -1;
      }
      if (!more) break;
      int lim;
      const int base = fetch(__popc(idle), lim, more);
      const int rank = __popc(idle & lt);
      if (free_ && rank < lim - base) {  // (base + rank may not fit an int)
        id = base + rank;
        F3 o, d;
        load(id, o, d, tmin, best_t, any);
        best_tri = -1; bu = bv = 0.f;
        if (!ray_is_void(o, d)) {
          r = ray_setup(o, d);
          sp = 0;
          cur = s.nt == 1 ? ~0 : 0;
        }
      }
      continue;
    }
    const float limit = pop_limit(best_t);
#pragma unroll
    for (int k = 0; k < TRN_NODE_STEPS; k++) {
      pop_entry(stack, sp, limit, cur);
      if (cur < 0 && leaf == 0) {
        leaf = cur;
        cur = kTracePop;
      }
      if (cur >= 0 && cur < kTracePop) cur = visit_node(s, r, cur, tmin, best_t, stack, sp, err);
    }
    const unsigned leaves = __ballot_sync(0xffffffffu, leaf < 0);
    if (4 * __popc(leaves) < TRN_LEAF_SHARE * (32 - __popc(idle)) &&
        __any_sync(0xffffffffu, (cur >= 0 && cur != kTraceDone) || (cur < 0 && leaf == 0)))
      continue;
    if (leaf < 0) {
      F3 p0, p1, p2;
      int tri;
      leaf_tri<true>(s, ~leaf, p0, p1, p2, tri);
      leaf = 0;
      float t, u, v;
      // best_tri = -1 before the first hit: a hit at exactly the ray's end is none
      if (intersect_tri(r, p0, p1, p2, tmin, INFINITY, t, u, v) && (t < best_t || (t == best_t && tri < best_tri))) {
        best_t = t; best_tri = tri; bu = u; bv = v;
        if (any) cur = kTraceDone;
      }
    }
  }
}

// One shared, non-inlined copy of the traversal, for fused kernels that trace
// at several places.
template <bool ANY>
__device__ __noinline__ bool trace_shared(const DeviceScene& s, const F3& o, const F3& d, float tmin, float tmax,
                                          Hit& hit, int* err) {
  return trace<ANY>(s, o, d, tmin, tmax, hit, err);
}

}  // namespace trn
