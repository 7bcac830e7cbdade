// lbvh_dev.cuh — device-side LBVH box tests and the stackless traversal shared by the query,
// contact-generation and self-contact kernels.
//
// Box tests restate Bounds::Overlap (xrtailor/src/physics/broad_phase/Bounds.cu:115-191);
// the traversal restates QueryDeviceStackless (xrtailor/src/physics/broad_phase/lbvh/BVH.cu:957-1055):
// left-first, escape indices instead of a stack, at most LBVH_MAX_BUFFER_SIZE (256) hits.
// Candidates are handed to a visitor in traversal order instead of a 1 KB per-thread buffer, so
// the narrow phase runs inline with identical first-minimum semantics.
#pragma once
#include "common.cuh"
#include "context.h"

namespace xrt {

__device__ __forceinline__ bool overlap_point(float4 l, float4 h, f3 p) {
  return p.x > l.x && p.x < h.x && p.y > l.y && p.y < h.y && p.z > l.z && p.z < h.z;
}

__device__ __forceinline__ int seg_intersection(float d1, float d2, f3 p1, f3 p2, f3& hit) {
  if ((d1 * d2) >= 0.0f) return 0;
  if (d1 == d2) return 0;
  hit = p1 + (p2 - p1) * (-d1 / (d2 - d1));
  return 1;
}
__device__ __forceinline__ int seg_in_box(f3 q, float4 l, float4 h, int axis) {
  if (axis == 1 && q.z > l.z && q.z < h.z && q.y > l.y && q.y < h.y) return 1;
  if (axis == 2 && q.z > l.z && q.z < h.z && q.x > l.x && q.x < h.x) return 1;
  if (axis == 3 && q.x > l.x && q.x < h.x && q.y > l.y && q.y < h.y) return 1;
  return 0;
}

__device__ __forceinline__ bool overlap_segment(float4 l, float4 h, f3 p1, f3 p2) {
  if (p2.x < l.x && p1.x < l.x) return false;
  if (p2.x > h.x && p1.x > h.x) return false;
  if (p2.y < l.y && p1.y < l.y) return false;
  if (p2.y > h.y && p1.y > h.y) return false;
  if (p2.z < l.z && p1.z < l.z) return false;
  if (p2.z > h.z && p1.z > h.z) return false;
  if (p1.x > l.x && p1.x < h.x && p1.y > l.y && p1.y < h.y && p1.z > l.z && p1.z < h.z) return true;
  f3 hit = mk3(0, 0, 0);
  if ((seg_intersection(p1.x - l.x, p2.x - l.x, p1, p2, hit) && seg_in_box(hit, l, h, 1)) ||
      (seg_intersection(p1.y - l.y, p2.y - l.y, p1, p2, hit) && seg_in_box(hit, l, h, 2)) ||
      (seg_intersection(p1.z - l.z, p2.z - l.z, p1, p2, hit) && seg_in_box(hit, l, h, 3)) ||
      (seg_intersection(p1.x - h.x, p2.x - h.x, p1, p2, hit) && seg_in_box(hit, l, h, 1)) ||
      (seg_intersection(p1.y - h.y, p2.y - h.y, p1, p2, hit) && seg_in_box(hit, l, h, 2)) ||
      (seg_intersection(p1.z - h.z, p2.z - h.z, p1, p2, hit) && seg_in_box(hit, l, h, 3)))
    return true;
  return false;
}

__device__ __forceinline__ bool overlap_box(float4 l, float4 h, f3 qlo, f3 qhi) {
  return !(l.x > qhi.x || h.x < qlo.x || l.y > qhi.y || h.y < qlo.y || l.z > qhi.z || h.z < qlo.z);
}

// ---- instances (InstView) ----------------------------------------------------------------------
__device__ __forceinline__ uint32_t inst_index(const InstView& I, uint32_t v) {
  return I.count == 1 ? 0u : __ldg(&I.of_vertex[v]);
}
__device__ __forceinline__ InstanceRec inst_rec(const InstView& I, uint32_t s) {
  return I.count == 1 ? I.one : I.rec[s];
}

// ---- forests (LbvhForest) ----------------------------------------------------------------------
__device__ __forceinline__ int4 forest_rec(const LbvhForest& F, uint32_t s) {
  return F.nseg == 1 ? F.one : F.seg[s];
}

// Segment owning primitive / sorted leaf position i.  The last segment whose base is <= i: empty
// segments share their base with the next one, so the segment found always owns i.
__device__ __forceinline__ uint32_t forest_find(const LbvhForest& F, uint32_t i) {
  if (F.nseg == 1) return 0;
  uint32_t lo = 0, hi = F.nseg;  // base(lo) <= i < base(hi)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if ((uint32_t)F.seg[mid].x <= i) lo = mid;
    else hi = mid;
  }
  return lo;
}

// ---- bottom-up merge (AssignAABBCAS_Kernel, BVH.cu:515-538) -------------------------------------
// The hierarchy over sorted keys is a radix tree, so it follows from the common prefix of each
// pair of neighbors alone: delta[i] = 1 + common prefix of keys i and i + 1 (0 behind the last key
// of a segment).  A subtree over positions [l, r] is the left child of the split after r when
// delta[r] > delta[l - 1], else the right child of the split after l - 1 (two equal neighbors
// cannot occur: sorted unique keys that differ at one bit do so once).  A left child's node id is
// its last position, a right child's its first (Karras), the root's 0, and the escape of a subtree
// ending at r is the right child of the split after r.  So one walk from the leaves gives boxes,
// links and escapes, and a refit needs nothing but delta.
//
// A block of kTreeBlock threads takes as many consecutive leaves.  Subtrees inside the block meet
// in shared memory; a subtree that finds no partner there when the block is through (its sibling
// reaches into another block) and those at the block's ends go on in global memory: the first
// arrival at a split leaves its outer end in the split's slot and stops, the second takes it, clears
// the slot for the next walk and merges.
// Bounded by the latency of a level, 2,100 cycles through the L2 (slot, then box) against about 250
// in shared memory, and for millions of leaves by the node writes.  Against hierarchy, boxes and
// escapes as four kernels and a merge that met in global memory throughout (ncu, warm cache):
// 2.09 M triangles 354 -> 190 us to build and 237 -> 164 us to refit, the 13,776-triangle body
// 52 -> 22 us and 31 -> 22 us.
constexpr int kTreeBlock = 256;

struct TreeRest {
  float4 a;  // lower corner, upper x
  float2 b;  // upper y, z
  unsigned long long l, r;
};
struct TreeMem {
  LbvhForest F;
  float4 *lo, *hi;                 // nodes
  int4* node;                      // links, written by BUILD walks
  int32_t *iesc, *eesc;            // escape tables, written by BUILD walks
  const uint8_t* delta;            // per sorted position
  unsigned long long* slot;        // per split: the first arrival's outer end (0: none yet)
  // small trees: the subtrees each block leaves, their number, and the blocks done
  TreeRest* rest;
  uint32_t *rest_count, *ticket;
};
inline TreeMem tree_mem(const Lbvh& b) {
  TreeMem t;
  t.F = b.forest();
  t.lo = b.lo.p;
  t.hi = b.hi.p;
  t.node = b.node.p;
  t.iesc = b.iesc.p;
  t.eesc = b.eesc.p;
  t.delta = b.delta.p;
  t.slot = b.slot.p;
  t.rest = reinterpret_cast<TreeRest*>(b.rest.p);
  t.rest_count = b.rest_count.p;
  t.ticket = b.rest_count.p + Lbvh::kSmallBlocks;
  return t;
}

// One end of a subtree: its position, the prefix shared with the neighbor outside (0: none), and
// whether the child that the split there has on the other side is a leaf.  Carried along, so a
// merge reads no prefix.
struct TreeEnd {
  uint32_t pos, d, leaf;
};
__device__ __forceinline__ unsigned long long pack_end(const TreeEnd& e) {
  return ((unsigned long long)(0x10000u | e.d << 1 | e.leaf) << 32) | e.pos;  // never 0
}
__device__ __forceinline__ TreeEnd unpack_end(unsigned long long v) {
  const uint32_t h = (uint32_t)(v >> 32) & 0xFFFFu;  // small_tree keeps an index above bit 48
  return TreeEnd{(uint32_t)v, h >> 1, h & 1u};
}

// The right child of the split after r (the escape of a subtree that ends there), the left child of
// the split before l, the node over [l, r]; `base`, `n`: the segment.
__device__ __forceinline__ int right_of(const TreeEnd& r, uint32_t base, uint32_t n) {
  const uint32_t p = r.pos + 1 - base;
  return r.d == 0 ? -1 : (int)(r.leaf ? n - 1 + p : p);
}
__device__ __forceinline__ int left_of(const TreeEnd& l, uint32_t base, uint32_t n) {
  const uint32_t p = l.pos - 1 - base;
  return (int)(l.leaf ? n - 1 + p : p);
}
__device__ __forceinline__ uint32_t id_of(const TreeEnd& l, const TreeEnd& r, uint32_t base) {
  return (l.d | r.d) == 0 ? 0u : (r.d > l.d ? r.pos : l.pos) - base;
}
// The node over [le, re] of segment `rec`, and its children's parent links; its own is its parent's
// to write.
template <bool BUILD>
__device__ __forceinline__ void write_node(const TreeMem& t, const int4& rec, f3 l, f3 u,
                                           uint32_t left, uint32_t right, const TreeEnd& le,
                                           const TreeEnd& re) {
  const uint32_t id = id_of(le, re, (uint32_t)rec.x);
  const int esc = right_of(re, (uint32_t)rec.x, (uint32_t)rec.y);
  __stcg(&t.lo[rec.z + id], mk4(l, __int_as_float((int)left)));
  __stcg(&t.hi[rec.z + id], mk4(u, __int_as_float(esc)));
  if (BUILD) {
    int4* node = t.node + rec.z;
    int* w = &node[id].x;
    w[1] = (int)left;
    *reinterpret_cast<int2*>(w + 2) = make_int2((int)right, -1);
    if ((le.d | re.d) == 0) w[0] = -1;
    node[left].x = (int)id;
    node[right].x = (int)id;
    t.iesc[(uint32_t)rec.w + id] = esc;
  }
}

// On through global memory from the subtree over [l, r], whose node is written: by this thread, or
// ahead of a barrier of the block.
template <bool BUILD>
__device__ __forceinline__ void tree_walk(const TreeMem& t, const int4& rec, TreeEnd l, TreeEnd r,
                                          f3 bl, f3 bu, uint32_t* err) {
  const uint32_t base = (uint32_t)rec.x, n = (uint32_t)rec.y;
  uint32_t steps = 0;
  while (l.d | r.d) {
    if (++steps > n) {
      raise_error(err, kErrTreeWalk);
      return;
    }
    const bool left = r.d > l.d;
    const uint32_t g = left ? r.pos : l.pos - 1;
    // acq_rel: releases this subtree's box with its end (the thread's own stores and those ordered
    // before it by a barrier); the second arrival acquires the first's
    unsigned long long far;
    asm volatile("atom.acq_rel.gpu.global.exch.b64 %0, [%1], %2;"
                 : "=l"(far)
                 : "l"(t.slot + g), "l"(pack_end(left ? l : r))
                 : "memory");
    if (far == 0) return;  // first arrival
    const uint32_t sid = (uint32_t)(left ? right_of(r, base, n) : left_of(l, base, n));
    const float4 a = __ldcg(&t.lo[rec.z + sid]), b = __ldcg(&t.hi[rec.z + sid]);
    t.slot[g] = 0;
    const f3 al = left ? bl : mk3(a), cl = left ? mk3(a) : bl;  // left child's, right child's
    const f3 au = left ? bu : mk3(b), cu = left ? mk3(b) : bu;
    bl = mk3(fminf(al.x, cl.x), fminf(al.y, cl.y), fminf(al.z, cl.z));
    bu = mk3(fmaxf(au.x, cu.x), fmaxf(au.y, cu.y), fmaxf(au.z, cu.z));
    const TreeEnd e = unpack_end(far);
    const uint32_t me = l.pos == r.pos ? n - 1 + (l.pos - base) : id_of(l, r, base);
    if (left) r = e;
    else l = e;
    write_node<BUILD>(t, rec, bl, bu, left ? me : sid, left ? sid : me, l, r);
  }
}

struct TreeShared {
  float box[2][6][kTreeBlock];             // per split: the boxes of its left and right child
  unsigned long long end[2][kTreeBlock];   // their outer ends
  uint32_t count[kTreeBlock];              // arrivals
};

// One leaf per thread, every thread of the block (`valid`: it has one).  `i` is the leaf's sorted
// position over the forest, [bl, bu] its box, `obj` its segment-local object.
template <bool BUILD>
__device__ __forceinline__ void tree_up(const TreeMem& t, TreeShared& sh, uint32_t i, bool valid,
                                        uint32_t obj, f3 bl, f3 bu, uint32_t* err) {
  sh.count[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t c0 = i - threadIdx.x;  // the block's first position
  const int4 rec = valid ? forest_rec(t.F, forest_find(t.F, i)) : make_int4(0, 0, 0, 0);
  const uint32_t base = (uint32_t)rec.x, n = (uint32_t)rec.y;
  TreeEnd l{i, 0, 0}, r{i, 0, 0};
  if (valid) {
    l.d = i > base ? t.delta[i - 1] : 0u;
    r.d = t.delta[i];
    l.leaf = !(i > base + 1 && t.delta[i - 2] > l.d);
    r.leaf = !(i < base + n - 1 && t.delta[i + 1] > r.d);
  }
  const f3 leaf_l = bl, leaf_u = bu;
  const TreeEnd after = r;  // the leaf's own right end, for its escape
  // Inside the block: shared memory only (a fence with global stores in flight takes 2,000 cycles
  // and more), the nodes are written below.
  uint32_t waiting = kNone;  // the split of the block this thread's subtree arrived at first
  uint32_t steps = 0;
  while (valid && (l.d | r.d)) {
    const bool left = r.d > l.d;
    const uint32_t g = left ? r.pos : l.pos - 1;
    if (g < c0 || g + 1 >= c0 + kTreeBlock) break;  // its sibling lies outside
    if (++steps > n) {
      raise_error(err, kErrTreeWalk);
      valid = false;
      break;
    }
    const uint32_t k = g - c0, side = left ? 0u : 1u;
    sh.box[side][0][k] = bl.x; sh.box[side][1][k] = bl.y; sh.box[side][2][k] = bl.z;
    sh.box[side][3][k] = bu.x; sh.box[side][4][k] = bu.y; sh.box[side][5][k] = bu.z;
    sh.end[side][k] = pack_end(left ? l : r);
    __threadfence_block();
    if (atomicAdd(&sh.count[k], 1u) == 0) {
      waiting = k;
      break;
    }
    __threadfence_block();
    const volatile float(*v)[6][kTreeBlock] = sh.box;
    bl = mk3(fminf(v[0][0][k], v[1][0][k]), fminf(v[0][1][k], v[1][1][k]),
             fminf(v[0][2][k], v[1][2][k]));
    bu = mk3(fmaxf(v[0][3][k], v[1][3][k]), fmaxf(v[0][4][k], v[1][4][k]),
             fmaxf(v[0][5][k], v[1][5][k]));
    const TreeEnd far = unpack_end(*(const volatile unsigned long long*)&sh.end[side ^ 1u][k]);
    if (left) r = far;
    else l = far;
  }
  __syncthreads();
  if (i < base + n && n > 0) {  // this position's leaf, and the node of the split after it
    const uint32_t id = n - 1 + (i - base);
    const int esc = right_of(after, base, n);
    __stcg(&t.lo[rec.z + id], mk4(leaf_l, __int_as_float((int)obj)));
    __stcg(&t.hi[rec.z + id], mk4(leaf_u, __int_as_float(esc)));
    if (BUILD) {
      int* w = &t.node[rec.z + id].x;
      w[1] = w[2] = -1;
      w[3] = (int)obj;
      if (n == 1) w[0] = -1;
      t.eesc[i] = esc;
    }
    const uint32_t k = threadIdx.x;
    if (sh.count[k] == 2) {
      const TreeEnd le = unpack_end(sh.end[0][k]), re = unpack_end(sh.end[1][k]);
      const uint32_t p = i - base;
      write_node<BUILD>(
          t, rec,
          mk3(fminf(sh.box[0][0][k], sh.box[1][0][k]), fminf(sh.box[0][1][k], sh.box[1][1][k]),
              fminf(sh.box[0][2][k], sh.box[1][2][k])),
          mk3(fmaxf(sh.box[0][3][k], sh.box[1][3][k]), fmaxf(sh.box[0][4][k], sh.box[1][4][k]),
              fmaxf(sh.box[0][5][k], sh.box[1][5][k])),
          le.pos == i ? n - 1 + p : p, re.pos == i + 1 ? n + p : p + 1, le, re);
    }
  }
  // A node is written by the thread at its split, its subtree carried on by another: the barrier
  // orders all of the block's nodes before any of its exchanges, so that an exchange releases them.
  __syncthreads();
  if (!valid || (waiting != kNone && sh.count[waiting] != 1u)) return;
  tree_walk<BUILD>(t, rec, l, r, bl, bu, err);
}

// ---- the same for a small single tree -----------------------------------------------------------
// Up to kSmallMax leaves: the blocks list the subtrees that are left (those whose siblings reach
// into another block) in position order, and the block that finishes last merges all of them in its
// shared memory the same way.  A level there costs about 250 cycles against 2,100 through the L2,
// and 13 to 19 levels of a small obstacle's tree lie across blocks.  A block leaves fewer than
// kRestPerBlock: the nodes across one of its two ends are a chain of growing prefix, 63 at most, and
// each has at most one child inside.
constexpr uint32_t kSmallMax = 64 * kTreeBlock;
constexpr uint32_t kRestPerBlock = 128;
constexpr int kRestPerThread = 4;
constexpr uint32_t kRestMax = kRestPerThread * kTreeBlock;  // above (never seen): tree_walk

struct SmallShared {
  float box[2][6][kRestMax];
  unsigned long long end[2][kRestMax];   // bit 49 up: the first / last subtree of the row it covers
  uint32_t count[kRestMax];
  uint32_t sum[kSmallMax / kTreeBlock + 1], warp_count[kTreeBlock / 32], last;
};

// One leaf per thread; arguments as for tree_up.
template <bool BUILD>
__device__ __forceinline__ void small_tree(const TreeMem& t, SmallShared& sh, uint32_t i, bool valid,
                                           uint32_t obj, f3 bl, f3 bu, uint32_t* err) {
  const uint32_t n = t.F.one.y, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t c0 = blockIdx.x * kTreeBlock, m0 = min(n - c0, (uint32_t)kTreeBlock);
  const int4 rec = make_int4(0, (int)n, 0, 0);
  // the parent of the subtree over [l, r], the subtrees first to last of a row of m, if it lies in
  // the row
  auto parent_of = [&](const TreeEnd& l, const TreeEnd& r, uint32_t first, uint32_t last, uint32_t m) {
    const bool left = r.d > l.d;
    if ((l.d | r.d) == 0 || (left ? last + 1 >= m : first == 0)) return -1;
    const uint32_t k = left ? last : first - 1;
    return sh.count[k] == 2
               ? (int)id_of(unpack_end(sh.end[0][k]), unpack_end(sh.end[1][k]), 0)
               : -1;
  };
  // the node over both children of split g, from slot k of a row of m
  auto write_split = [&](uint32_t g, uint32_t k, uint32_t m, bool top) {
    const unsigned long long el = sh.end[0][k], er = sh.end[1][k];
    const TreeEnd l = unpack_end(el), r = unpack_end(er);
    const uint32_t first = (uint32_t)(el >> 49), last = (uint32_t)(er >> 49);
    const uint32_t id = id_of(l, r, 0);
    const uint32_t left = l.pos == g ? n - 1 + g : g, right = r.pos == g + 1 ? n + g : g + 1;
    const int esc = right_of(r, 0, n);
    __stcg(&t.lo[id],
           make_float4(fminf(sh.box[0][0][k], sh.box[1][0][k]), fminf(sh.box[0][1][k], sh.box[1][1][k]),
                       fminf(sh.box[0][2][k], sh.box[1][2][k]), __int_as_float((int)left)));
    __stcg(&t.hi[id],
           make_float4(fmaxf(sh.box[0][3][k], sh.box[1][3][k]), fmaxf(sh.box[0][4][k], sh.box[1][4][k]),
                       fmaxf(sh.box[0][5][k], sh.box[1][5][k]), __int_as_float(esc)));
    if (BUILD) {
      __stcg(&t.node[id], make_int4(parent_of(l, r, first, last, m), (int)left, (int)right, -1));
      t.iesc[id] = esc;
      // children that a block wrote before the list was complete
      if (top && first == k) t.node[left].x = (int)id;
      if (top && last == k + 1) t.node[right].x = (int)id;
    }
  };
  // merges upwards from the first-th of `m` subtrees in a row, slot j being the split after the
  // j-th; returns the slot it waits at, or kNone at the root or at a split outside the row
  auto climb = [&](TreeEnd& l, TreeEnd& r, float b[6], uint32_t first, uint32_t m) {
    uint32_t steps = 0, last = first;  // the subtrees it covers
    while (l.d | r.d) {
      const bool left = r.d > l.d;
      const uint32_t k = left ? last : first - 1;
      if (left ? last + 1 >= m : first == 0) return kNone;
      if (++steps > n) {
        raise_error(err, kErrTreeWalk);
        return kNone;
      }
      const uint32_t side = left ? 0u : 1u;
#pragma unroll
      for (int q = 0; q < 6; ++q) sh.box[side][q][k] = b[q];
      sh.end[side][k] = pack_end(left ? l : r) | (unsigned long long)(left ? first : last) << 49;
      __threadfence_block();
      if (atomicAdd(&sh.count[k], 1u) == 0) return k;
      __threadfence_block();
      const volatile float(*v)[6][kRestMax] = sh.box;
#pragma unroll
      for (int q = 0; q < 6; ++q)
        b[q] = q < 3 ? fminf(v[0][q][k], v[1][q][k]) : fmaxf(v[0][q][k], v[1][q][k]);
      const unsigned long long far = *(const volatile unsigned long long*)&sh.end[side ^ 1u][k];
      if (left) {
        r = unpack_end(far);
        last = (uint32_t)(far >> 49);
      } else {
        l = unpack_end(far);
        first = (uint32_t)(far >> 49);
      }
    }
    return kNone;
  };
  sh.count[tid] = 0;
  __syncthreads();
  TreeEnd l{i, 0, 0}, r{i, 0, 0};
  if (valid) {
    l.d = i > 0 ? t.delta[i - 1] : 0u;
    r.d = t.delta[i];
    l.leaf = !(i > 1 && t.delta[i - 2] > l.d);
    r.leaf = !(i + 1 < n && t.delta[i + 1] > r.d);
  }
  const TreeEnd leaf_l = l, leaf_r = r;
  float b[6] = {bl.x, bl.y, bl.z, bu.x, bu.y, bu.z};
  const uint32_t at = valid ? climb(l, r, b, tid, m0) : kNone;
  __syncthreads();
  const bool left_over = valid && (l.d | r.d) && (at == kNone || sh.count[at] == 1u);
  const unsigned mask = __ballot_sync(0xFFFFFFFFu, left_over);
  if (lane == 0) sh.warp_count[warp] = (uint32_t)__popc(mask);
  __syncthreads();
  if (left_over) {  // a subtree's thread is one of its leaves', so threads are in position order
    uint32_t rank = (uint32_t)__popc(mask & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < warp; ++w) rank += sh.warp_count[w];
    TreeRest& e = t.rest[blockIdx.x * kRestPerBlock + min(rank, kRestPerBlock - 1)];
    e.a = make_float4(b[0], b[1], b[2], b[3]);
    e.b = make_float2(b[4], b[5]);
    e.l = pack_end(l);
    e.r = pack_end(r);
  }
  if (tid == 0) {
    uint32_t all = 0;
    for (uint32_t w = 0; w < kTreeBlock / 32; ++w) all += sh.warp_count[w];
    t.rest_count[blockIdx.x] = all;
  }
  if (valid) {
    const int esc = right_of(leaf_r, 0, n);
    __stcg(&t.lo[n - 1 + i], mk4(bl, __int_as_float((int)obj)));
    __stcg(&t.hi[n - 1 + i], mk4(bu, __int_as_float(esc)));
    if (BUILD) {
      __stcg(&t.node[n - 1 + i], make_int4(parent_of(leaf_l, leaf_r, tid, tid, m0), -1, -1, (int)obj));
      t.eesc[i] = esc;
    }
    if (tid + 1 < m0 && sh.count[tid] == 2) write_split(i, tid, m0, false);
  }
  __syncthreads();
  if (tid == 0) {  // the last block of the grid goes on (a lone block has no subtree left but the root)
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "l"(t.ticket)
                 : "memory");
    sh.last = old + 1 == gridDim.x;
    if (sh.last) *t.ticket = 0;
    __threadfence();
  }
  __syncthreads();
  if (!sh.last) return;
  if (tid <= gridDim.x) {
    uint32_t x = 0;
    for (uint32_t k = 0; k < tid; ++k) x += __ldcg(&t.rest_count[k]);
    sh.sum[tid] = x;
  }
#pragma unroll
  for (int q = 0; q < kRestPerThread; ++q) sh.count[tid + q * kTreeBlock] = 0;
  __syncthreads();
  const uint32_t rest = sh.sum[gridDim.x];
  uint32_t split[kRestPerThread];
  const bool fits = rest <= kRestMax;
  for (uint32_t q = 0, k = tid; k < rest; ++q, k += kTreeBlock) {
    uint32_t lo = 0, hi = gridDim.x;  // its block
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (sh.sum[mid] <= k) lo = mid;
      else hi = mid;
    }
    const TreeRest* e = t.rest + lo * kRestPerBlock + (k - sh.sum[lo]);
    const float4 ea = __ldcg(&e->a);
    const float2 eb = __ldcg(&e->b);
    TreeEnd el = unpack_end(__ldcg(&e->l)), er = unpack_end(__ldcg(&e->r));
    if (fits) {
      float v[6] = {ea.x, ea.y, ea.z, ea.w, eb.x, eb.y};
#pragma unroll
      for (int z = 0; z < kRestPerThread; ++z)
        if (z == (int)q) split[z] = er.pos;
      climb(el, er, v, k, rest);
    } else {
      tree_walk<BUILD>(t, rec, el, er, mk3(ea.x, ea.y, ea.z), mk3(ea.w, eb.x, eb.y), err);
    }
  }
  __syncthreads();
  if (!fits) return;
#pragma unroll
  for (int q = 0; q < kRestPerThread; ++q) {
    const uint32_t k = tid + q * kTreeBlock;
    if (k + 1 < rest && sh.count[k] == 2) write_split(split[q], k, rest, true);
  }
}

// ---- shared by the kernels of one cluster ---------------------------------------------------------
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Stores word `v` at `p` of the block of rank `cta`.
__device__ __forceinline__ void st_cluster(void* p, uint32_t cta, uint32_t v) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// ---- refit: leaves grow, internal boxes follow ----------------------------------------------------
// `grow(prim, lo, hi)` extends the box of global primitive `prim`.
template <bool SMALL, class Grow>
__global__ void __launch_bounds__(kTreeBlock) k_refit(uint32_t n, Grow grow, TreeMem t,
                                                      uint32_t* err) {
  extern __shared__ float4 smem[];
  const uint32_t i = blockIdx.x * kTreeBlock + threadIdx.x;
  uint32_t obj = 0;
  f3 bl = mk3(0, 0, 0), bu = bl;
  if (i < n) {
    const int4 r = forest_rec(t.F, forest_find(t.F, i));
    const uint32_t k = (uint32_t)r.z + (uint32_t)r.y - 1 + (i - (uint32_t)r.x);
    const float4 l = t.lo[k], h = t.hi[k];
    obj = (uint32_t)__float_as_int(l.w);
    bl = mk3(l);
    bu = mk3(h);
    grow((uint32_t)r.x + obj, bl, bu);
  }
  if (SMALL)
    small_tree<false>(t, *reinterpret_cast<SmallShared*>(smem), i, i < n, obj, bl, bu, err);
  else
    tree_up<false>(t, *reinterpret_cast<TreeShared*>(smem), i, i < n, obj, bl, bu, err);
}
template <class Grow>
void launch_refit(const Lbvh& b, const Grow& grow, cudaStream_t s, uint32_t* err) {
  auto k = b.small() ? k_refit<true, Grow> : k_refit<false, Grow>;
  const size_t smem = b.small() ? sizeof(SmallShared) : sizeof(TreeShared);
  if (raise_smem((const void*)k, smem) != cudaSuccess) return;
  k<<<grid_for(b.n, kTreeBlock), kTreeBlock, smem, s>>>(b.n, grow, tree_mem(b), err);
}

// Stackless traversal state; one node visit per lbvh_step.
struct TraverseState {
  int node;        // next node, -1 = done
  uint32_t found;  // leaves visited (capped at kMaxCandidates)
  uint32_t guard;  // node visits (bounded by 2n + 2)
};

__device__ __forceinline__ TraverseState lbvh_begin(const LbvhView& b) {
  return TraverseState{b.n == 0 ? -1 : 0, 0u, 0u};
}

// One node visit; returns false once the traversal has ended (no visit made).
template <class Overlap, class Visit>
__device__ __forceinline__ bool lbvh_step(const LbvhView& b, TraverseState& st, Overlap ov,
                                          Visit visit, uint32_t* err) {
  if (st.node == -1 || st.found >= kMaxCandidates) return false;
  if (++st.guard > 2 * b.n + 2) {
    raise_error(err, kErrTraversal);
    st.node = -1;
    return false;
  }
  const float4 l = b.lo[st.node], h = b.hi[st.node];
  if (ov(l, h)) {
    if ((uint32_t)st.node >= b.n - 1) {
      visit((uint32_t)__float_as_int(l.w));
      ++st.found;
      st.node = __float_as_int(h.w);
    } else {
      st.node = __float_as_int(l.w);
    }
  } else {
    st.node = __float_as_int(h.w);
  }
  return true;
}

// Stackless traversal; `ov(lo, hi)` tests a node box, `visit(object)` receives each hit.
template <class Overlap, class Visit>
__device__ __forceinline__ uint32_t lbvh_traverse(const LbvhView& b, Overlap ov, Visit visit,
                                                  uint32_t* err) {
  TraverseState st = lbvh_begin(b);
  while (lbvh_step(b, st, ov, visit, err)) {
  }
  return st.found;
}

}  // namespace xrt
