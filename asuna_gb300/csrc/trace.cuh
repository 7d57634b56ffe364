// trace.cuh — two-level BVH traversal (closest hit and occlusion), shared by the
// traversal kernels (trace.cu) and the path kernel (path.cu).
//
// Software replacement for the RT-core traversal behind traceRayEXT
// (src/shaders/raytrace.projective.rgen:108-109 closest hit with tmin 1e-5 and
// tmax 1e10; rgen:117-122 occlusion with tmin 0, tmax dist - 2*EPS,
// terminate-on-first-hit).  Facing culling is off, as the reference's
// instances set VK_GEOMETRY_INSTANCE_TRIANGLE_FACING_CULL_DISABLE_BIT_KHR
// (src/pipeline/pipeline_raytrace.cpp:132).
//
// Persistent warps refill their idle lanes from the queue (one atomic per
// refill and warp); each thread walks the top level, then an instance's
// bottom level, over 8-wide nodes of 80 bytes (bvh_wide.cu).  A node step
// tests eight child boxes at once: the 8-bit planes become floats by byte
// permutation (1 + q 2^-15) and the distances are one packed fused
// multiply-add per plane pair.  What bounds the kernel is the chain of
// dependent node fetches of a ray and the lanes that idle along: the wide
// node makes that chain 2.8 times shorter than a binary one's.  On the
// 21M-triangle benchmark scene (1920x1080, 8 frames, depth 12; ms per render):
// closest hits 14.97 -> 10.06, occlusion 7.47 -> 3.89, nodes per ray
// 24.4 -> 8.9; the issue slots are 73% busy with 14 of 32 lanes active.
// The ray is moved into object space and tested against triangles with the
// watertight algorithm of Woop, Benthin and Wald (JCGT 2013) using explicitly
// rounded operations, so the hits equal the CPU oracle's bit for bit: they
// depend on the triangle tests alone, not on the tree.
//
// The box tests are conservative.  With cell = 2^e, plane = p + q cell and
// c = fl(fl(p - o) inv), a plane distance is fma(1 + q 2^-15, s, c - s) with
// s = 2^15 cell inv.  Its error has a part relative to the distance itself
// (the subtraction, the reciprocal, the products: under 2^-21 of it) and a
// part of the frame: 2^-9 cell from rounding c - s, 2^-14 cell from the
// cancellation between c and the offset.  The far distance is widened by
// 2^-20, and every child box was quantised with 2^-5 cell to spare.
#pragma once
#include <cuda_runtime.h>

#include "kernels.h"

namespace asuna {
namespace {

struct WT {
  int kx, ky, kz;
  float Sx, Sy, Sz;
};

__device__ __forceinline__ float sel(float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

__device__ __forceinline__ WT wtPre(float3 d) {
  WT w;
  float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
  int kx = kz + 1 == 3 ? 0 : kz + 1;
  int ky = kx + 1 == 3 ? 0 : kx + 1;
  float dz = sel(d, kz);
  if (dz < 0.0f) {
    int t = kx;
    kx = ky;
    ky = t;
  }
  w.kx = kx;
  w.ky = ky;
  w.kz = kz;
  w.Sx = __fdiv_rn(sel(d, kx), dz);
  w.Sy = __fdiv_rn(sel(d, ky), dz);
  w.Sz = __fdiv_rn(1.0f, dz);
  return w;
}

// Watertight test; same operations and order as the CPU oracle.
__device__ __forceinline__ bool wtTri(const WT& w, float3 o, float4 p0, float4 p1, float4 p2, float tmin, float tmax,
                                      float& t, float& b1, float& b2) {
  const float3 A = make_float3(__fsub_rn(p0.x, o.x), __fsub_rn(p0.y, o.y), __fsub_rn(p0.z, o.z));
  const float3 B = make_float3(__fsub_rn(p1.x, o.x), __fsub_rn(p1.y, o.y), __fsub_rn(p1.z, o.z));
  const float3 C = make_float3(__fsub_rn(p2.x, o.x), __fsub_rn(p2.y, o.y), __fsub_rn(p2.z, o.z));
  const float Akz = sel(A, w.kz), Bkz = sel(B, w.kz), Ckz = sel(C, w.kz);
  const float Ax = __fsub_rn(sel(A, w.kx), __fmul_rn(w.Sx, Akz)), Ay = __fsub_rn(sel(A, w.ky), __fmul_rn(w.Sy, Akz));
  const float Bx = __fsub_rn(sel(B, w.kx), __fmul_rn(w.Sx, Bkz)), By = __fsub_rn(sel(B, w.ky), __fmul_rn(w.Sy, Bkz));
  const float Cx = __fsub_rn(sel(C, w.kx), __fmul_rn(w.Sx, Ckz)), Cy = __fsub_rn(sel(C, w.ky), __fmul_rn(w.Sy, Ckz));
  float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
  float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
  float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = __double2float_rn(__dsub_rn(__dmul_rn(double(Cx), double(By)), __dmul_rn(double(Cy), double(Bx))));
    V = __double2float_rn(__dsub_rn(__dmul_rn(double(Ax), double(Cy)), __dmul_rn(double(Ay), double(Cx))));
    W = __double2float_rn(__dsub_rn(__dmul_rn(double(Bx), double(Ay)), __dmul_rn(double(By), double(Ax))));
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
  const float det = __fadd_rn(__fadd_rn(U, V), W);
  if (det == 0.0f) return false;
  const float Az = __fmul_rn(w.Sz, Akz), Bz = __fmul_rn(w.Sz, Bkz), Cz = __fmul_rn(w.Sz, Ckz);
  const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
  const float rcp = __fdiv_rn(1.0f, det);
  const float tt = __fmul_rn(T, rcp);
  if (!(tt >= tmin && tt <= tmax)) return false;
  t = tt;
  b1 = __fmul_rn(V, rcp);
  b2 = __fmul_rn(W, rcp);
  return true;
}

// Three-input min / max (one instruction each on sm_100 and later; exact,
// like fminf / fmaxf, for the finite values the slab test produces).
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Inverse direction for the slab tests, from the hardware reciprocal
// (rcp.approx, within one ulp of 1/x for the normal values it is given):
// the box tests stay conservative, as the far distance is widened by 2^-20
// (16 ulp), far more than the reciprocal's error; hits come from the
// watertight triangle test alone, so they do not depend on it.
__device__ __forceinline__ float rcpApprox(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// (magnitudes clamped to [1e-30, 1e30], so the reciprocal stays a normal
// number that the flush-to-zero form returns unchanged)
__device__ __forceinline__ float3 safeInv(float3 d) {
  auto inv = [](float x) { return rcpApprox(copysignf(fminf(fmaxf(fabsf(x), 1e-30f), 1e30f), x)); };
  return make_float3(inv(d.x), inv(d.y), inv(d.z));
}

// Packed pairs of IEEE single-precision values in one 64-bit register pair:
// the f32x2 fma of sm_100 and later issues as one instruction and rounds each
// lane to nearest.
typedef unsigned long long F2;
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// byte j of w as the float 1 + q 2^-15
template <int J>
__device__ __forceinline__ float planeOf(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604 | (J << 4)));
}

__device__ __forceinline__ void xformRay(const float4* w, float3 o, float3 d, float3& oo, float3& dd) {
  float4 r0 = __ldg(&w[0]), r1 = __ldg(&w[1]), r2 = __ldg(&w[2]);
  auto po = [&](float4 r) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.x, o.x), __fmul_rn(r.y, o.y)), __fmul_rn(r.z, o.z)), r.w);
  };
  auto pd = [&](float4 r) { return __fadd_rn(__fadd_rn(__fmul_rn(r.x, d.x), __fmul_rn(r.y, d.y)), __fmul_rn(r.z, d.z)); };
  oo = make_float3(po(r0), po(r1), po(r2));
  dd = make_float3(pd(r0), pd(r1), pd(r2));
}

constexpr float kFarScale = 1.00000095367431640625f;  // 1 + 2^-20
constexpr uint32_t kTriGroup = 0x80000000u;            // stack entry: a leaf group (else a node group)
constexpr uint32_t kHits = 0xffu;
constexpr uint32_t kTraceSpinCap = 1u << 20;           // node steps of one warp pass
constexpr uint32_t kTraceRayCap = 1u << 16;            // leaves + transitions of one ray
// Lanes (of 32) that must want a node step for the warp to go on with node
// steps while others wait at a leaf or a transition (closest hits of the
// benchmark scene: 13.3 ms per render with 1, 10.4 with 8, 10.1 with 12, 11.7
// with 16 on an earlier state of the kernel).
constexpr int kNodeLanes = 12;

// Traversal state of one ray.  A node group is a set of children of one node
// that the ray's box tests kept: (index of the first inner child, inner-child
// mask << 8 | children left); a leaf group likewise (node, leaf slots left).
// nodeStep() takes the next child of the node group in octant order, leaves
// the rest on the stack and tests that child's eight boxes; leafStep() tests
// the triangles of one leaf; move() enters an instance or leaves it.
//
// The state is kept small (64 registers with the node's 20 words in flight):
// the world-space ray is read again from its source at the few instance
// transitions instead of being held, the watertight test's axis permutation
// is packed into one word, a closer hit goes to memory at once and only its
// distance is held, and tmin and the stack cap come from the source and the
// launch.
template <int TB, int SHS>  // threads per block, 8-byte stack entries in shared memory
struct Trav {
  float ox, oy, oz, ix, iy, iz;  // ray origin and inverse direction in the current space
  float Sx, Sy, Sz;  // watertight shear of the current space's direction
  uint32_t kxyz;     // its axis permutation, kx | ky << 2 | kz << 4
  uint32_t pref;     // slots on the near side, one byte per axis
  float best;  // tmax, then the closest hit's distance
  uint32_t curInst;
  int sp;      // stack entries in use
  int bottom;  // entries below the current instance's (0: in the top level)
  uint32_t gBase, gMask;
  uint32_t tNode, tMask;
  bool found;

  __device__ __forceinline__ void setShear(const WT& w) {
    Sx = w.Sx;
    Sy = w.Sy;
    Sz = w.Sz;
    kxyz = uint32_t(w.kx) | uint32_t(w.ky) << 2 | uint32_t(w.kz) << 4;
  }
  __device__ __forceinline__ WT shear() const {
    WT w;
    w.kx = int(kxyz & 3u);
    w.ky = int((kxyz >> 2) & 3u);
    w.kz = int(kxyz >> 4);
    w.Sx = Sx;
    w.Sy = Sy;
    w.Sz = Sz;
    return w;
  }

  __device__ __forceinline__ void init(const SceneDev& S, float3 ro, float3 rd, float tmax) {
    setSpace(ro, safeInv(rd));
    best = tmax;
    curInst = 0;
    sp = 0;
    bottom = 0;
    enterTree(uint32_t(S.tlasRoot));
    found = false;
  }
  // the root as the only child of a node group
  __device__ __forceinline__ void enterTree(uint32_t root) {
    gBase = root;
    gMask = 0x101u;
    tMask = 0u;
  }

  __device__ __forceinline__ void setSpace(float3 o, float3 inv) {
    ox = o.x;
    oy = o.y;
    oz = o.z;
    ix = inv.x;
    iy = inv.y;
    iz = inv.z;
    pref = (ix < 0.0f ? 0xAAu : 0x55u) | (iy < 0.0f ? 0xCC00u : 0x3300u) | (iz < 0.0f ? 0xF00000u : 0x0F0000u);
  }

  __device__ __forceinline__ bool hasNodes() const { return (gMask & kHits) != 0u; }
  __device__ __forceinline__ bool idle() const { return !hasNodes() && tMask == 0u; }

  // the slot to visit next: the near side first, axis by axis
  __device__ __forceinline__ uint32_t pick(uint32_t hits) const {
    uint32_t a = hits & (pref >> 16);
    hits = a ? a : hits;
    a = hits & (pref >> 8);
    hits = a ? a : hits;
    a = hits & pref;
    hits = a ? a : hits;
    return hits & (0u - hits);
  }

  // Stack: the first SHS entries in shared memory (stride TB: bank-conflict
  // free), deeper ones in thread-local memory.
  __device__ __forceinline__ void push(uint2* sh, uint2* loc, uint2 v, int lim, bool& ovf) {
    if (sp >= lim) {
      ovf = true;
      return;
    }
    if (sp < SHS)
      sh[sp * TB] = v;
    else
      loc[sp - SHS] = v;
    ++sp;
  }
  __device__ __forceinline__ uint2 top(const uint2* sh, const uint2* loc) {
    --sp;
    return sp < SHS ? sh[sp * TB] : loc[sp - SHS];
  }
  // the next group of the current level, if there is one
  __device__ __forceinline__ void next(const uint2* sh, const uint2* loc) {
    if (sp > bottom) {
      const uint2 e = top(sh, loc);
      if (e.y & kTriGroup) {
        tNode = e.x;
        tMask = e.y & kHits;
      } else {
        gBase = e.x;
        gMask = e.y;
      }
    }
  }

  // Child J of four: shifts a 1 into `miss` where the ray misses its box.
  // (the sign of tf (1 + 2^-20) - tn, one rounding; where an infinity makes
  // it NaN the child counts as hit, which is conservative)
  template <int J>
  __device__ __forceinline__ void testChild(uint32_t& miss, float tmin, uint32_t nx, uint32_t fx, uint32_t ny,
                                            uint32_t fy, uint32_t nz, uint32_t fz, F2 sx, F2 sy, F2 sz, F2 cx, F2 cy,
                                            F2 cz) const {
    float tnx, tfx, tny, tfy, tnz, tfz;
    unpack2(fma2(pack2(planeOf<J>(nx), planeOf<J>(fx)), sx, cx), tnx, tfx);
    unpack2(fma2(pack2(planeOf<J>(ny), planeOf<J>(fy)), sy, cy), tny, tfy);
    unpack2(fma2(pack2(planeOf<J>(nz), planeOf<J>(fz)), sz, cz), tnz, tfz);
    const float tn = fmaxf(fmax3(tnx, tny, tnz), tmin);
    const float tf = fminf(fmin3(tfx, tfy, tfz), best);
    miss = __funnelshift_l(__float_as_uint(__fmaf_rn(tf, kFarScale, -tn)), miss, 1);
  }

  template <bool COUNT>
  __device__ __forceinline__ void nodeStep(const SceneDev& S, float tmin, uint2* sh, uint2* loc, int lim, uint32_t& nNodes,
                                           bool& ovf) {
    const uint32_t bit = pick(gMask & kHits);
    const uint32_t child = gBase + __popc((gMask >> 8) & (bit - 1u));
    gMask ^= bit;
    const uint4* n = S.nodes[child].w;
    const uint4 n0 = __ldg(n), n1 = __ldg(n + 1), n2 = __ldg(n + 2), n3 = __ldg(n + 3), n4 = __ldg(n + 4);
    if (hasNodes()) push(sh, loc, make_uint2(gBase, gMask), lim, ovf);
    if (COUNT) ++nNodes;
    const bool gx = ix < 0.0f, gy = iy < 0.0f, gz = iz < 0.0f;
    const float sx = __uint_as_float((n0.w & 0xffu) << 23) * ix, sy = __uint_as_float((n0.w & 0xff00u) << 15) * iy,
                sz = __uint_as_float((n0.w & 0xff0000u) << 7) * iz;
    const float cx = __fmaf_rn(__uint_as_float(n0.x) - ox, ix, -sx), cy = __fmaf_rn(__uint_as_float(n0.y) - oy, iy, -sy),
                cz = __fmaf_rn(__uint_as_float(n0.z) - oz, iz, -sz);
    const F2 sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
    const F2 cx2 = pack2(cx, cx), cy2 = pack2(cy, cy), cz2 = pack2(cz, cz);
    uint32_t miss = 0u;
    {
      const uint32_t nx = gx ? n3.w : n2.y, fx = gx ? n2.y : n3.w, ny = gy ? n4.y : n2.w, fy = gy ? n2.w : n4.y,
                     nz = gz ? n4.w : n3.y, fz = gz ? n3.y : n4.w;
      testChild<3>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<2>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<1>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<0>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
    }
    {
      const uint32_t nx = gx ? n3.z : n2.x, fx = gx ? n2.x : n3.z, ny = gy ? n4.x : n2.z, fy = gy ? n2.z : n4.x,
                     nz = gz ? n4.z : n3.x, fz = gz ? n3.x : n4.z;
      testChild<3>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<2>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<1>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
      testChild<0>(miss, tmin, nx, fx, ny, fy, nz, fz, sx2, sy2, sz2, cx2, cy2, cz2);
    }
    const uint32_t hits = ~miss & kHits, inner = n0.w >> 24, leaves = hits & ~inner;
    gBase = n1.x;
    gMask = inner << 8 | (hits & inner);
    if (leaves) {
      // (a lane that walked on with a leaf group in hand keeps the older one below)
      if (tMask) push(sh, loc, make_uint2(tNode, kTriGroup | tMask), lim, ovf);
      tNode = child;
      tMask = leaves;
    }
    if (idle()) next(sh, loc);
  }

  // The next leaf of the leaf group: its first record and their number.
  __device__ __forceinline__ uint32_t takeLeaf(const SceneDev& S, uint32_t& count) {
    const uint32_t bit = pick(tMask);
    tMask ^= bit;
    const WideNode* n = S.nodes + tNode;
    const uint32_t m = __ldg(reinterpret_cast<const uint8_t*>(&n->w[1].z) + (31 - __clz(int(bit))));
    count = m >> 5;
    return __ldg(&n->w[1].y) + (m & 31u);
  }

  // Tests one leaf; true when an occlusion ray is done.
  template <bool ANY, bool COUNT, class Src>
  __device__ __forceinline__ bool leafStep(const SceneDev& S, Src& src, uint32_t idx, uint2* sh, uint2* loc,
                                           uint32_t& nTris) {
    uint32_t cnt;
    const uint32_t first = takeLeaf(S, cnt);
    const WT wt = shear();
    const float3 o = make_float3(ox, oy, oz);
    const float tmin = src.tmin(idx);
    for (uint32_t k = 0; k < cnt; ++k) {
      const TriDev* tr = S.tris + first + k;
      const float4 p0 = __ldg(&tr->v0), p1 = __ldg(&tr->v1), p2 = __ldg(&tr->v2);
      if (COUNT) ++nTris;
      float t, b1, b2;
      if (wtTri(wt, o, p0, p1, p2, tmin, best, t, b1, b2)) {
        if (ANY || src.stopAtHit()) {
          found = true;
          return true;
        }
        const uint32_t prim = __float_as_uint(p0.w);
        // exact ties resolve to the lowest (instance, primitive), so the
        // result does not depend on traversal order
        if (!found || t < best || src.later(idx, curInst, prim)) {
          found = true;
          best = t;
          src.store(idx, t, b1, b2, prim, curInst);
        }
      }
    }
    if (idle()) next(sh, loc);
    return false;
  }

  // Leaves the current instance, if the ray is in one, and enters the next one
  // of the top-level leaf group whose box the ray meets (both in one round: in
  // scenes of overlapping instances each round of a warp costs as much as a
  // leaf; a room of eight, 256x256, 16 frames: 1.40 -> 1.29 ms).  True when the
  // traversal is over.  `src.world(i, o, d)` gives ray i's world-space origin
  // and direction again.
  template <class Src>
  __device__ __forceinline__ bool move(const SceneDev& S, const Src& src, uint32_t idx, uint2* sh, uint2* loc, int lim,
                                       bool& ovf) {
    if (bottom != 0) {
      float3 wo, wd;
      src.world(idx, wo, wd);
      setSpace(wo, safeInv(wd));
      const uint2 t = top(sh, loc), g = top(sh, loc);
      bottom = 0;
      gBase = g.x;
      gMask = g.y;
      tNode = t.x;
      tMask = t.y & kHits;
    }
    while (tMask) {
      uint32_t cnt;
      const uint32_t at = takeLeaf(S, cnt);
      if (!cnt) continue;
      const uint32_t inst = __ldg(&S.instIds[at]);
      const InstDev* in = S.inst + inst;
      // the instance's own box against the distance as it is now: the
      // 8-bit box of the top level may be much larger (a cell is up to
      // 1/128 of its node, which may span the scene) and was tested earlier
      const float4 lo = __ldg(reinterpret_cast<const float4*>(in->boxLo)),
                   hi = __ldg(reinterpret_cast<const float4*>(in->boxHi));
      const float x0 = (lo.x - ox) * ix, x1 = (hi.x - ox) * ix, y0 = (lo.y - oy) * iy, y1 = (hi.y - oy) * iy,
                  z0 = (lo.z - oz) * iz, z1 = (hi.z - oz) * iz;
      const float tn = fmax3(fminf(x0, x1), fminf(y0, y1), fmaxf(fminf(z0, z1), src.tmin(idx)));
      const float tf = fmin3(fmaxf(x0, x1), fmaxf(y0, y1), fminf(fmaxf(z0, z1), best)) * kFarScale;
      if (!(tn <= tf)) continue;
      if (sp + 2 > lim) {
        ovf = true;
        continue;
      }
      push(sh, loc, make_uint2(gBase, gMask), lim, ovf);
      push(sh, loc, make_uint2(tNode, kTriGroup | tMask), lim, ovf);
      bottom = sp;
      curInst = inst;
      float3 wo, wd, o, d;
      src.world(idx, wo, wd);
      xformRay(in->w2o, wo, wd, o, d);
      setSpace(o, safeInv(d));
      setShear(wtPre(d));
      enterTree(__float_as_uint(lo.w));
      const uint32_t leaves = __float_as_uint(hi.w);
      if (leaves) {  // a handful of triangles: straight to them
        tNode = gBase;
        tMask = leaves;
        gMask = 0u;
      }
      return false;
    }
    if (idle()) next(sh, loc);
    return idle();
  }
};

// One round of the warp's active lanes (`act`): node steps, one leaf, one
// transition.  True for a lane whose traversal is over; `stop` (for the whole
// warp) when the node loop passed its bound.
template <bool ANY, bool COUNT, class T, class Src>
__device__ __forceinline__ bool traceRound(const SceneDev& S, Src& src, T& tr, uint32_t idx, bool active, unsigned act,
                                           int nodeLanes, bool spec, int lim, uint32_t& events, uint2* sh, uint2* loc,
                                           uint32_t& nNodes, uint32_t& nTris, bool& ovf, bool& stop) {
  // Node steps while enough lanes want one.  Lanes with a leaf group in
  // hand walk on when `spec` (and there is room on the stack).  A pass that stops early leaves lanes at a leaf or a
  // transition, which go on below: some lane advances in every round.
  // Both loops carry a bound far above any real traversal: past it the
  // warp stops and reports the error instead of running on.
  uint32_t spin = 0;
  for (;;) {
    const bool want = active && tr.hasNodes() && tr.tMask == 0u;
    const unsigned wm = __ballot_sync(0xffffffffu, want);
    if (wm == 0u || (__popc(wm) < nodeLanes && wm != act)) break;
    if (++spin > kTraceSpinCap) break;
    // A speculative step pushes two entries, and the ordered steps below it one
    // on each further level (of treeLevels - 1 at most): with room for all of
    // them, speculation never overflows a stack that the ordered walk fits.
    if (want || (spec && active && tr.hasNodes() && tr.bottom != 0 && tr.sp + S.treeLevels < lim))
      tr.template nodeStep<COUNT>(S, src.tmin(idx), sh, loc, lim, nNodes, ovf);
  }
  if (spin > kTraceSpinCap) {
    ovf = true;
    stop = true;
    return false;
  }
  bool done = false;
  if (active && tr.bottom != 0 && tr.tMask != 0u) {
    done = tr.template leafStep<ANY, COUNT>(S, src, idx, sh, loc, nTris);
    ++events;
  }
  __syncwarp();
  if (active && !done && (tr.bottom == 0 ? tr.tMask != 0u || tr.idle() : tr.idle())) {
    done = tr.move(S, src, idx, sh, loc, lim, ovf);
    ++events;
  }
  if (events > kTraceRayCap) {
    ovf = true;
    done = active;
  }
  return done;
}

// Persistent warp over a ray source.  Lanes whose ray is finished take the
// next rays of the source (one fetch per refill, per warp) while the other
// lanes keep traversing.  Src supplies count, warps (that share it), fetch(n) -> first index (called
// by one lane), commit(first, n) (called by every lane), load(i, tr),
// tmin(i), world(i, o, d), store(i, hit), later(i, inst, prim) (the hit stored
// last belongs to a later instance or primitive) and finish(i, found).
template <bool ANY, bool COUNT, int TB, int SHS, class Src>
__device__ __forceinline__ void traceWarp(const SceneDev& S, Src& src, uint2* sh, uint2* loc, uint32_t refill,
                                          bool spec, int lim, uint32_t& nNodes, uint32_t& nTris, bool& ovf) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lanesBelow = (1u << lane) - 1u;
  // Lanes in use: a short queue is spread over all warps of the grid, so that
  // fewer rays share (and serialise) a warp (a 320x180 preview's closest hits
  // 0.65 -> 0.41 ms, a 1280x720 frame's 0.92 -> 0.72).
  const uint32_t use = min(32u, max(1u, (src.count + src.warps - 1u) / src.warps));
  const unsigned usable = 0xffffffffu >> (32u - use);
  const int nodeLanes = int(use) * kNodeLanes / 32;
  bool active = false, drained = false;
  uint32_t idx = 0, events = 0;
  Trav<TB, SHS> tr;
  tr.gMask = tr.tMask = 0u;
  tr.bottom = 0;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !active) & usable;
    if (idle && !drained && (uint32_t(__popc(idle)) >= refill || idle == usable)) {
      const int leader = __ffs(idle) - 1;
      uint32_t base = 0;
      if (int(lane) == leader) base = src.fetch(uint32_t(__popc(idle)));
      base = __shfl_sync(0xffffffffu, base, leader);
      src.commit(base, uint32_t(__popc(idle)));
      drained = base + uint32_t(__popc(idle)) >= src.count;
      if (idle >> lane & 1u) {
        const uint32_t r = base + uint32_t(__popc(idle & lanesBelow));
        if (r < src.count) {
          idx = r;
          active = true;
          events = 0;
          src.load(S, r, tr);
        }
      }
    }
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!act) {
      if (drained) break;
      continue;
    }
    bool stop = false;
    const bool done = traceRound<ANY, COUNT>(S, src, tr, idx, active, act, nodeLanes, spec, lim, events, sh, loc,
                                             nNodes, nTris, ovf, stop);
    if (stop) break;
    if (done) {
      active = false;
      events = 0;
      src.finish(idx, tr.found);
    }
  }
}

// Ray queue of a wavefront pass.  LIVE: the running kernel also writes the
// queue (the path kernel), so its rays are not read through the read-only path.
template <bool ANY, bool LIVE = false>
struct QueueSrc {
  template <class V>
  static __device__ __forceinline__ V get(const V* p) {
    return LIVE ? *p : __ldg(p);
  }
  const WaveDev* W;
  const KParams* P;
  const float4 *rO, *rD;
  uint32_t* fetchCtr;
  uint32_t count, warps;
  uint32_t wave;  // wavefront pass (1-based)
  __device__ __forceinline__ uint32_t fetch(uint32_t n) { return atomicAdd(fetchCtr, n); }
  __device__ __forceinline__ bool stopAtHit() const { return ANY; }
  __device__ __forceinline__ void commit(uint32_t, uint32_t) {}
  template <class T>
  __device__ __forceinline__ void load(const SceneDev& S, uint32_t r, T& tr) {
    const float4 o4 = get(&rO[r]);
    const float4 d4 = get(&rD[r]);
    tr.init(S, make_float3(o4.x, o4.y, o4.z), make_float3(d4.x, d4.y, d4.z), ANY ? o4.w : 10000000000.0f);
  }
  __device__ __forceinline__ float tmin(uint32_t) const { return ANY ? 0.0f : 0.00001f; }
  __device__ __forceinline__ void world(uint32_t r, float3& o, float3& d) const {
    const float4 o4 = get(&rO[r]);
    const float4 d4 = get(&rD[r]);
    o = make_float3(o4.x, o4.y, o4.z);
    d = make_float3(d4.x, d4.y, d4.z);
  }
  __device__ __forceinline__ void store(uint32_t i, float t, float u, float v, uint32_t prim, uint32_t inst) {
    W->hit[i] = make_float4(t, u, v, __uint_as_float(prim));
    W->hitInst[i] = inst;
  }
  __device__ __forceinline__ bool later(uint32_t i, uint32_t inst, uint32_t prim) const {
    const uint32_t h = W->hitInst[i];
    return inst < h || (inst == h && prim < __float_as_uint(W->hit[i].w));
  }
  __device__ __forceinline__ void finish(uint32_t i, bool found) {
    if (ANY) {
      if (!found) {
        const uint32_t p = __float_as_uint(get(&rD[i].w));
        const float4 c = get(&W->shC[i]);
        float4 r = W->rad[p];
        r.x = r.x + c.x;
        r.y = r.y + c.y;
        r.z = r.z + c.z;
        W->rad[p] = r;
        if (P->records) W->rec[p].y |= 1u << (wave - (W->path[p].info.y >> kPassShift) - 1u);
      }
    } else if (!found) {
      W->hit[i] = make_float4(-1.0f, 0.0f, 0.0f, 0.0f);
      W->hitInst[i] = 0xffffffffu;
    }
  }
};

}  // namespace
}  // namespace asuna
