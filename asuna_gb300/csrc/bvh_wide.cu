// bvh_wide.cu — collapses the builders' binary trees into the 8-wide nodes
// that the traversal reads.
//
// The layout and the octant slots follow Ylitie, Karras and Laine, "Efficient
// incoherent ray traversal on GPUs through compressed wide BVHs" (HPG 2017):
// a node holds up to eight child boxes as 8-bit offsets in a per-node frame,
// its inner children are consecutive nodes and its leaf triangles consecutive
// records, and a child sits in the slot whose sign pattern points to its side
// of the node, so a ray visits slots in the order of its direction octant.
//
// One thread makes one wide node, level by level from the roots: it opens
// the child with the largest surface area until there are eight (or only
// leaves are left), reserves the children's nodes and triangles with one
// atomic each, assigns the slots greedily and quantises the boxes outwards.
// The levels are launched without waiting for their sizes (each kernel reads
// its own from the counters).  Bound by the latency of the gathered 64-byte
// binary nodes and by one thread's serial work per node: 3.3 ms for 21M
// triangles, of 39 ms for the whole scene creation.
//
// A box in the frame (p, 2^e per axis) covers its child with 1/32 cell to
// spare on every side: the traversal evaluates plane distances as one fused
// multiply-add whose rounding moves a plane by far less (see trace.cu), so no
// child that the exact box test would keep is lost.  Planes are culling data
// only: triangles and hits stay in 32 bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "bvh_wide.h"
#include "common.h"

namespace asuna {
namespace {

constexpr int kThreads = 128;
constexpr size_t kKeepLoose = 1 << 20;  // node arrays up to this size stay as they were reserved

struct WideItem {
  int32_t ref;    // binary inner node
  uint32_t node;  // the wide node it becomes
  uint32_t top;   // 1: top level (leaves are instances)
};

enum { kWNodes = 0, kWTris = 1, kWInst = 2, kWError = 3, kWLevel0 = 4, kWNum = 4 + 72 };

struct WideCtx {
  const BvhNode* bin;
  const TriDev* tris;
  WideNode* out;
  TriDev* outTris;
  uint32_t* instIds;
  uint32_t* rootLeaves;
  uint32_t* counters;  // [kWLevel0 + l]: items of level l
  WideItem* items[2];
  uint32_t nodeCap, triCap, instCap, itemCap;
};

struct Child {
  float lo[3], hi[3];
  int32_t ref;
};

__device__ __forceinline__ float childArea(const Child& c) {
  const float x = c.hi[0] - c.lo[0], y = c.hi[1] - c.lo[1], z = c.hi[2] - c.lo[2];
  return x * y + y * z + z * x;
}

// Appends the children of binary node `ref` (empty slots left out).
__device__ __forceinline__ int openNode(const BvhNode* bin, int32_t ref, Child* c, int at) {
  const BvhNode n = bin[ref];
  for (int s = 0; s < 2; ++s) {
    const int32_t r = s == 0 ? n.ref.x : n.ref.y;
    if (r == kStackSentinel) continue;
    nodeGetBox(n, s, c[at].lo, c[at].hi);
    for (int a = 0; a < 3; ++a) {  // (NaN: the other operand, so the box stays conservative)
      c[at].lo[a] = fminf(fmaxf(c[at].lo[a], -kWideFar), kWideFar);
      c[at].hi[a] = fmaxf(fminf(c[at].hi[a], kWideFar), -kWideFar);
    }
    c[at].ref = r;
    ++at;
  }
  return at;
}

__global__ void __launch_bounds__(kThreads) k_collapse(WideCtx C, int level) {
  // (an earlier level that ran out of room left items unwritten)
  const uint32_t n = C.counters[kWError] ? 0u : min(C.counters[kWLevel0 + level], C.itemCap);
  const WideItem* in = C.items[level & 1];
  WideItem* next = C.items[(level & 1) ^ 1];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const WideItem it = in[i];
    Child c[8];
    int nc = openNode(C.bin, it.ref, c, 0);
    while (nc < 8) {
      int best = -1;
      float area = -1.0f;
      for (int k = 0; k < nc; ++k)
        if (c[k].ref >= 0) {
          const float a = childArea(c[k]);
          if (best < 0 || a > area) {
            best = k;
            area = a;
          }
        }
      if (best < 0) break;
      const int32_t ref = c[best].ref;
      c[best] = c[nc - 1];
      nc = openNode(C.bin, ref, c, nc - 1);
    }
    // frame: per axis the smallest power-of-two cell whose 8-bit range spans
    // the children with the margins
    float p[3];
    uint32_t ebyte[3];
    float perCell[3];  // cells per unit: 2^-e
    float mid[3];
    for (int a = 0; a < 3; ++a) {
      float lo = nc ? c[0].lo[a] : 0.0f, hi = nc ? c[0].hi[a] : 0.0f;
      for (int k = 1; k < nc; ++k) {
        lo = fminf(lo, c[k].lo[a]);
        hi = fmaxf(hi, c[k].hi[a]);
      }
      mid[a] = 0.5f * lo + 0.5f * hi;
      int e = -125;
      const float ext = __fsub_ru(hi, lo);
      if (ext > 0.0f) e = max(e, ilogbf(ext) - 7);  // 2^e * 255 >= ext within two steps
      // (boxes of at most 2 kWideFar: e stays far below the byte's range)
      for (;; ++e) {
        const float cell = __uint_as_float(uint32_t(e + 127) << 23);
        perCell[a] = __uint_as_float(uint32_t(127 - e) << 23);
        p[a] = __fsub_rd(lo, cell * 0.0625f);
        if (e >= kWideMaxExp || ceilf(__fsub_ru(hi, p[a]) * perCell[a] + 0.03125f) <= 255.0f) break;
      }
      ebyte[a] = uint32_t(e + kWideExpBias);
    }
    // slots: the (child, slot) pair with the largest projection first
    int slotOf[8];
    uint32_t freeSlots = 0xffu, left = (1u << nc) - 1u;
    for (int r = 0; r < nc; ++r) {
      float bestCost = -INFINITY;
      int bc = __ffs(left) - 1, bs = __ffs(freeSlots) - 1;
      for (int k = 0; k < nc; ++k) {
        if (!(left >> k & 1u)) continue;
        const float x = c[k].lo[0] + c[k].hi[0] - 2.0f * mid[0], y = c[k].lo[1] + c[k].hi[1] - 2.0f * mid[1],
                    z = c[k].lo[2] + c[k].hi[2] - 2.0f * mid[2];
        for (int s = 0; s < 8; ++s) {
          if (!(freeSlots >> s & 1u)) continue;
          const float v = (s & 1 ? x : -x) + (s & 2 ? y : -y) + (s & 4 ? z : -z);
          if (v > bestCost) {
            bestCost = v;
            bc = k;
            bs = s;
          }
        }
      }
      slotOf[bc] = bs;
      left &= ~(1u << bc);
      freeSlots &= ~(1u << bs);
    }
    // reservations
    uint32_t inner = 0, leafPrims = 0;
    for (int k = 0; k < nc; ++k) {
      if (c[k].ref >= 0)
        ++inner;
      else
        leafPrims += leafCount(c[k].ref);
    }
    uint32_t childBase = 0, primBase = 0, itemBase = 0;
    if (inner) {
      childBase = atomicAdd(&C.counters[kWNodes], inner);
      itemBase = atomicAdd(&C.counters[kWLevel0 + level + 1], inner);
    }
    if (leafPrims) primBase = atomicAdd(&C.counters[it.top ? kWInst : kWTris], leafPrims);
    if (childBase + inner > C.nodeCap || itemBase + inner > C.itemCap ||
        primBase + leafPrims > (it.top ? C.instCap : C.triCap)) {
      atomicOr(&C.counters[kWError], 1u);
      continue;
    }
    // children in slot order
    uint32_t q[6][2] = {}, meta[2] = {}, imask = 0;
    uint32_t usedInner = 0, usedPrims = 0;
    for (int s = 0; s < 8; ++s) {
      int k = -1;
      for (int j = 0; j < nc; ++j)
        if (slotOf[j] == s) k = j;
      const int sh = 8 * (s & 3), h = s >> 2;
      if (k < 0) {
        for (int a = 0; a < 3; ++a) q[a][h] |= 255u << sh;
        continue;
      }
      for (int a = 0; a < 3; ++a) {
        // (the rounding of the last sum, 2^-16 cell, comes out of the margin)
        const float lo = floorf(__fsub_rd(c[k].lo[a], p[a]) * perCell[a] - 0.03125f);
        const float hi = ceilf(__fsub_ru(c[k].hi[a], p[a]) * perCell[a] + 0.03125f);
        q[a][h] |= uint32_t(fminf(fmaxf(lo, 0.0f), 255.0f)) << sh;
        q[3 + a][h] |= uint32_t(fminf(fmaxf(hi, 0.0f), 255.0f)) << sh;
      }
      if (c[k].ref >= 0) {
        imask |= 1u << s;
        next[itemBase + usedInner] = WideItem{c[k].ref, childBase + usedInner, it.top};
        ++usedInner;
      } else {
        const uint32_t first = leafFirst(c[k].ref), cnt = leafCount(c[k].ref);
        if (cnt > kWideLeaf) atomicOr(&C.counters[kWError], 2u);
        meta[h] |= (cnt << 5 | usedPrims) << sh;
        for (uint32_t j = 0; j < min(cnt, kWideLeaf); ++j) {
          if (it.top)
            C.instIds[primBase + usedPrims + j] = first + j;
          else
            C.outTris[primBase + usedPrims + j] = C.tris[first + j];
        }
        usedPrims += cnt;
      }
    }
    WideNode w;
    w.w[0] = make_uint4(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]),
                        ebyte[0] | ebyte[1] << 8 | ebyte[2] << 16 | imask << 24);
    w.w[1] = make_uint4(childBase, primBase, meta[0], meta[1]);
    w.w[2] = make_uint4(q[0][0], q[0][1], q[1][0], q[1][1]);
    w.w[3] = make_uint4(q[2][0], q[2][1], q[3][0], q[3][1]);
    w.w[4] = make_uint4(q[4][0], q[4][1], q[5][0], q[5][1]);
    C.out[it.node] = w;
    if (level == 0) {
      uint32_t slots = 0;
      for (int s = 0; s < 8; ++s)
        if (meta[s >> 2] >> (8 * (s & 3)) & 0xe0u) slots |= 1u << s;
      C.rootLeaves[i] = !it.top && inner == 0 && leafPrims <= kWideLeaf ? slots : 0u;
    }
  }
}

}  // namespace

int buildWide(const BvhNode* nodes, uint32_t nodeCount, const TriDev* tris, uint32_t triCount, uint32_t instCount,
              const std::vector<int32_t>& roots, uint32_t maxDepth, cudaStream_t st, WideBvh& out) {
  const uint32_t nr = uint32_t(roots.size());
  // a wide node comes from one binary inner node each, and a level's items
  // are distinct binary nodes
  const uint32_t nodeCap = nodeCount + nr;
  const int levels = int(std::min<uint32_t>(maxDepth + 1, kWNum - kWLevel0 - 1));
  // at most half of the binary nodes lie on one level
  const uint32_t itemCap = nodeCount / 2 + nr + 1;
  // one temporary block: the counters, the roots' leaves, the two item lists
  // and the nodes, unless their bound is small enough to keep them in it
  auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t oRoots = pad(kWNum * 4), oA = oRoots + pad(size_t(nr) * 4),
               oB = oA + pad(size_t(itemCap) * sizeof(WideItem)), oNodes = oB + pad(size_t(itemCap) * sizeof(WideItem));
  struct Tmp {
    char* p = nullptr;
    ~Tmp() { cudaFree(p); }
  } tmp;
  const bool keep = size_t(nodeCap) * sizeof(WideNode) <= kKeepLoose;
  ASUNA_CUDA_TRY(
      cudaMalloc(reinterpret_cast<void**>(&tmp.p), oNodes + (keep ? 0 : size_t(nodeCap) * sizeof(WideNode))));
  if (keep) ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&out.nodes), size_t(nodeCap) * sizeof(WideNode)));
  ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&out.tris),
                            size_t(triCount) * sizeof(TriDev) + (size_t(instCount) + 1) * 4));
  out.instIds = reinterpret_cast<uint32_t*>(out.tris + triCount);
  WideCtx C;
  C.bin = nodes;
  C.tris = tris;
  C.out = keep ? out.nodes : reinterpret_cast<WideNode*>(tmp.p + oNodes);
  C.outTris = out.tris;
  C.instIds = out.instIds;
  C.counters = reinterpret_cast<uint32_t*>(tmp.p);
  C.rootLeaves = reinterpret_cast<uint32_t*>(tmp.p + oRoots);
  C.items[0] = reinterpret_cast<WideItem*>(tmp.p + oA);
  C.items[1] = reinterpret_cast<WideItem*>(tmp.p + oB);
  C.nodeCap = nodeCap;
  C.triCap = triCount;
  C.instCap = instCount;
  C.itemCap = itemCap;
  std::vector<WideItem> first(nr);
  for (uint32_t k = 0; k < nr; ++k) first[k] = WideItem{roots[k], k, k + 1 == nr ? 1u : 0u};
  uint32_t ctr[kWNum] = {};
  ctr[kWNodes] = nr;
  ctr[kWLevel0] = nr;
  ASUNA_CUDA_TRY(cudaMemcpyAsync(C.items[0], first.data(), nr * sizeof(WideItem), cudaMemcpyHostToDevice, st));
  ASUNA_CUDA_TRY(cudaMemcpyAsync(tmp.p, ctr, sizeof(ctr), cudaMemcpyHostToDevice, st));
  int dev = 0, sms = 0;
  ASUNA_CUDA_TRY(cudaGetDevice(&dev));
  ASUNA_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (int l = 0; l < levels; ++l) {
    // (a level has at most eight times the items of the one above)
    const uint64_t most = l < 9 ? std::min<uint64_t>(itemCap, uint64_t(nr) << (3 * l)) : itemCap;
    k_collapse<<<unsigned(std::min<uint64_t>((most + kThreads - 1) / kThreads, uint64_t(sms) * 8)), kThreads, 0, st>>>(
        C, l);
  }
  ASUNA_CUDA_TRY(cudaGetLastError());
  out.rootLeaves.resize(nr);
  ASUNA_CUDA_TRY(cudaMemcpyAsync(ctr, tmp.p, sizeof(ctr), cudaMemcpyDeviceToHost, st));
  ASUNA_CUDA_TRY(cudaMemcpyAsync(out.rootLeaves.data(), C.rootLeaves, size_t(nr) * 4, cudaMemcpyDeviceToHost, st));
  ASUNA_CUDA_TRY(cudaStreamSynchronize(st));
  if (ctr[kWError] || ctr[kWLevel0 + levels] || ctr[kWTris] != triCount || ctr[kWInst] != instCount)
    return fail(ASUNA_ERR_INVALID, "wide BVH: collapse failed (error bits %u, %u of %u triangles, %u of %u instances)",
                ctr[kWError], ctr[kWTris], triCount, ctr[kWInst], instCount);
  out.nodeCount = ctr[kWNodes];
  while (out.levels < uint32_t(levels) && ctr[kWLevel0 + out.levels]) ++out.levels;
  if (keep) {
    out.bytes = size_t(nodeCap) * sizeof(WideNode) + triCount * sizeof(TriDev) + (size_t(instCount) + 1) * 4;
    return ASUNA_OK;
  }
  // the node bound is loose (about a fifth is used): an array of the size used
  out.bytes = size_t(out.nodeCount) * sizeof(WideNode) + triCount * sizeof(TriDev) + (size_t(instCount) + 1) * 4;
  ASUNA_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&out.nodes), size_t(out.nodeCount) * sizeof(WideNode)));
  ASUNA_CUDA_TRY(cudaMemcpyAsync(out.nodes, C.out, size_t(out.nodeCount) * sizeof(WideNode),
                                 cudaMemcpyDeviceToDevice, st));
  ASUNA_CUDA_TRY(cudaStreamSynchronize(st));
  return ASUNA_OK;
}

}  // namespace asuna
