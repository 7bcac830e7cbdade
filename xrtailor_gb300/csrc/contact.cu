// contact.cu — obstacle motion within a frame and Swift obstacle-contact generation.
//
//   Interpolate_Kernel .............. xrtailor/src/physics/PhysicsMesh.cu:610-620
//   UpdateNodeMidstepNormals ........ xrtailor/src/physics/PhysicsMeshHelper.cu:212-225, 297-310
//   GenerateVF_DCD_Kernel ........... xrtailor/src/physics/pbd_collision/PBDCollision.cu:17-46
//   GenerateVFCCD_Kernel ............ PBDCollision.cu:236-267
//   GenerateEE_DCD_Kernel ........... PBDCollision.cu:100-151 (R-triangle edge filter RTriangle.cu:12-17)
//   PredictedToPositions/UpdateNormals PhysicsMesh.cu:604-608, PhysicsMeshHelper.cu:196-210
//
// Vertex normals are gathered per vertex over its faces in ascending face order (the reference
// scatters them with float atomics); the interpolated midstep position x1 of a neighbor is
// recomputed from x0 and x inside the gather, so interpolation and normals are one kernel.
#include <algorithm>

#include "common.cuh"
#include "context.h"
#include "lbvh_dev.cuh"
#include "prim_tests.cuh"

namespace xrt {
namespace {

__device__ __forceinline__ f3 lerp_pos(const float4* __restrict__ x0, const float4* __restrict__ x,
                                       int i, float alpha) {
  return (1.0f - alpha) * mk3(x0[i]) + alpha * mk3(x[i]);
}

// The weighted sum of the face normals around each vertex of the warp, in list order.  The warp's
// vertices own consecutive entries of the list: the lanes work out the terms of kFan entries at a
// time, one entry a lane, whichever vertex owns it, and each vertex adds its own up from shared
// memory.  A vertex has six faces as a rule, but a pole of a body of revolution its whole ring, which
// would be one lane's chain.
constexpr int kFanBlock = 64;
constexpr uint32_t kFanRounds = 6, kFan = 32 * kFanRounds;
struct FanShared {
  float x[kFan], y[kFan], z[kFan];
};
template <class Pos>
__device__ __forceinline__ f3 fan_sum(FanShared& w, const int4* __restrict__ tri,
                                      const uint32_t* __restrict__ ptr,
                                      const uint32_t* __restrict__ list, uint32_t i, uint32_t nv,
                                      Pos pos) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t k = 0, end = 0;
  if (i < nv) {
    k = ptr[i];
    end = ptr[i + 1];
  }
  const uint32_t first = __shfl_sync(0xFFFFFFFFu, k, 0);
  const uint32_t last = __reduce_max_sync(0xFFFFFFFFu, end);
  f3 acc = mk3(0, 0, 0);
  for (uint32_t base = first; base < last; base += kFan) {
    const uint32_t n = min(last - base, kFan);
    uint32_t fc[kFanRounds];
    int4 t[kFanRounds];
    f3 xi[kFanRounds], e0[kFanRounds], e1[kFanRounds];
#pragma unroll
    for (uint32_t r = 0; r < kFanRounds; ++r)
      fc[r] = 32 * r + lane < n ? list[base + 32 * r + lane] : 0u;
#pragma unroll
    for (uint32_t r = 0; r < kFanRounds; ++r)
      if (32 * r + lane < n) t[r] = tri[fc[r] >> 2];
#pragma unroll
    for (uint32_t r = 0; r < kFanRounds; ++r) {
      if (32 * r + lane >= n) continue;
      const uint32_t j = fc[r] & 3u;  // the owner's corner
      xi[r] = pos(j == 0 ? t[r].x : j == 1 ? t[r].y : t[r].z);
      e0[r] = pos(j == 0 ? t[r].y : j == 1 ? t[r].z : t[r].x);
      e1[r] = pos(j == 0 ? t[r].z : j == 1 ? t[r].x : t[r].y);
    }
#pragma unroll
    for (uint32_t r = 0; r < kFanRounds; ++r) {
      if (32 * r + lane >= n) continue;
      const f3 a = e0[r] - xi[r], b = e1[r] - xi[r];
      const f3 term = cross(a, b) / (dot(a, a) * dot(b, b));
      w.x[32 * r + lane] = term.x;
      w.y[32 * r + lane] = term.y;
      w.z[32 * r + lane] = term.z;
    }
    __syncwarp();
    for (; k < end && k < base + n; ++k)
      acc = acc + mk3(w.x[k - base], w.y[k - base], w.z[k - base]);
    __syncwarp();
  }
  return acc;
}

// The same with a lane that takes its vertex's faces one after the other, every position once.
template <class Pos>
__device__ __forceinline__ f3 fan_walk(const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
                                       const uint32_t* __restrict__ list, uint32_t i, uint32_t nv,
                                       Pos pos) {
  f3 acc = mk3(0, 0, 0);
  if (i >= nv) return acc;
  const f3 xi = pos((int)i);
  for (uint32_t k = ptr[i]; k < ptr[i + 1]; ++k) {
    const uint32_t fc = list[k];
    const int4 t = tri[fc >> 2];
    const uint32_t j = fc & 3u;
    const f3 a = pos(j == 0 ? t.y : j == 1 ? t.z : t.x) - xi;
    const f3 b = pos(j == 0 ? t.z : j == 1 ? t.x : t.y) - xi;
    acc = acc + cross(a, b) / (dot(a, a) * dot(b, b));
  }
  return acc;
}

// SPREAD: fan_sum, else fan_walk (uses_spread_fans).
template <bool SPREAD>
constexpr int kFanThreads = SPREAD ? kFanBlock : kBlock;
template <bool SPREAD, class Pos>
__device__ __forceinline__ f3 fan(const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
                                  const uint32_t* __restrict__ list, uint32_t i, uint32_t nv,
                                  Pos pos) {
  if constexpr (SPREAD) {
    __shared__ FanShared shared[kFanBlock / 32];
    return fan_sum(shared[threadIdx.x >> 5], tri, ptr, list, i, nv, pos);
  } else {
    return fan_walk(tri, ptr, list, i, nv, pos);
  }
}

template <bool SPREAD>
__global__ void __launch_bounds__(kFanThreads<SPREAD>) k_obstacle_pass(
    const float4* __restrict__ x0, const float4* __restrict__ x, float4* __restrict__ x1,
    float4* __restrict__ n1, const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
    const uint32_t* __restrict__ list, uint32_t nv, float alpha) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const f3 acc =
      fan<SPREAD>(tri, ptr, list, i, nv, [&](int j) { return lerp_pos(x0, x, j, alpha); });
  if (i >= nv) return;
  x1[i] = mk4(lerp_pos(x0, x, i, alpha), 0.0f);
  n1[i] = mk4(normalize(acc), 0.0f);
}

__global__ void __launch_bounds__(kFanBlock) k_vertex_normals(
    const float4* __restrict__ x, const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
    const uint32_t* __restrict__ list, float4* __restrict__ out, uint32_t nv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const f3 acc = fan<true>(tri, ptr, list, i, nv, [&](int j) { return mk3(x[j]); });
  if (i < nv) out[i] = mk4(normalize(acc), 0.0f);
}

// Frame end: x0 = x, then normals of the new x0 (computed from x, which is the same data).
template <bool SPREAD>
__global__ void __launch_bounds__(kFanThreads<SPREAD>) k_obstacle_commit(
    const float4* __restrict__ x, float4* __restrict__ x0, float4* __restrict__ nrm,
    const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
    const uint32_t* __restrict__ list, uint32_t nv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const f3 acc = fan<SPREAD>(tri, ptr, list, i, nv, [&](int j) { return mk3(x[j]); });
  if (i >= nv) return;
  x0[i] = mk4(mk3(x[i]), 0.0f);
  nrm[i] = mk4(normalize(acc), 0.0f);
}

// ---- contact generation: one query per cloth vertex (VF) or edge (EE) ------------------------------
// A warp takes a packet of queries from a counter and works through (query, node) pairs: up to 32
// pairs are taken off a stack in shared memory at a time, one a lane; a pair whose boxes overlap
// puts the node's left child on the stack, and a left child its sibling.  So a query's walk is
// spread over the lanes: walks near the obstacle are hundreds of nodes long and the others end at
// the root, and a lane per query left a warp waiting for its longest.  The tests of the leaves, five
// to ten box tests each, go to queues in shared memory and run 32 at a time as well.  A query's
// result is the smallest distance, and of equal ones that of the first leaf of the walk, kept as the
// minimum of (distance, tree position of the leaf) in one 64-bit word: the distances are not
// negative, so their bits compare as they do, and a walk meets the leaves in the order of their
// positions.  The winner's data are computed again at the end.  Only the cap of 256 leaves depends
// on the order: queries that meet more are walked again, one a lane, in order, up to the cap.
// Contacts record global triangle ids.
// 24 garments on bodies of 13,776 triangles: EE 430 -> 251 us, VF 321 -> 107 against one walk per lane
// with the same queues, and 740 / 340 us with the leaves' tests in the walk; a 256 x 256 cloth: EE 75
// -> 43, VF 72 -> 30; an 11,495-vertex garment: EE 100 -> 33, VF 96 -> 30.  Bound by issue: about 190
// instructions a round, most of them the segment's tests against the six faces.
constexpr int kGenBlock = 128, kGenWarps = kGenBlock / 32;
// Pairs on a warp's stack.  A full round leaves kReserve free; without room for one, pairs are taken
// singly, which deepens the stack by at most one per level of the tree (64-bit keys: 65 levels).
constexpr uint32_t kStack = 512, kReserve = 128;

// A warp's queue of tests: x = element (global), y = place in the walk, z = query that asks.
template <int N>
struct TestQueue {
  uint4 entry[N];
};
// Adds one test per lane with `on`; work(entry, true) runs 32 of them once there are as many.
template <class Work>
__device__ __forceinline__ void queue_push(TestQueue<64>& w, uint32_t& count, bool on,
                                           uint32_t element, uint32_t place, uint32_t slot,
                                           Work work) {
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, on);
  if (m == 0) return;
  if (on) w.entry[count + __popc(m & ((1u << lane) - 1u))] = make_uint4(element, place, slot, 0);
  count += __popc(m);
  __syncwarp();
  if (count >= 32) {
    count -= 32;
    const uint4 e = w.entry[count + lane];
    __syncwarp();
    work(e, true);
  }
}
// Runs what is left; work(entry, the lane has one).
template <int N, class Work>
__device__ __forceinline__ void queue_flush(TestQueue<N>& w, uint32_t& count, Work work) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool on = lane < count;
  const uint4 e = on ? w.entry[lane] : make_uint4(0, 0, 0, 0);
  __syncwarp();
  if (count != 0) work(e, on);
  count = 0;
  __syncwarp();
}
// The key of a result: smaller distances first, then the earlier place.  A distance counts only
// below kScalarMax (no NaN, no infinity), so a key of no_result() stays where none does.
__device__ __forceinline__ unsigned long long no_result() {
  return (unsigned long long)__float_as_uint(kScalarMax) << 32;
}
__device__ __forceinline__ void keep_nearest(unsigned long long& key, float dist, uint32_t place) {
  if (dist < kScalarMax)
    atomicMin(&key, (unsigned long long)__float_as_uint(dist) << 32 | place);
}

struct PairStack {
  uint2 e[kStack];      // node of the query's tree; query | left child << 5 | mask << 6
  int4 tree[32];        // of each query's tree: first primitive, primitives, first node
};
// Takes packets of `packet` queries until none of `nq` is left.  start(i) sets the lane's query up
// and returns its mask of tests (0: none) and its tree's record; within(slot, mask) leaves the tests
// of query `slot` that have not passed the cap, test(l, h, slot, mask) returns the
// tests of query `slot` that overlap the box, leaf(hit, slot, element, place) takes the leaves of
// all lanes (hit 0: none), finish(i, record) writes the lane's result.
template <class Start, class Within, class Test, class Leaf, class Finish>
__device__ __forceinline__ void pair_loop(PairStack& w, const LbvhForest& F, uint32_t* counter,
                                          uint32_t nq, uint32_t packet, uint32_t* err, Start start,
                                          Within within, Test test, Leaf leaf, Finish finish) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  for (;;) {
    uint32_t first = 0;
    if (lane == 0) first = atomicAdd(counter, packet);
    first = __shfl_sync(kAll, first, 0);
    if (first >= nq) return;
    const uint32_t i = first + lane;
    const bool valid = lane < packet && i < nq;
    int4 rec = make_int4(0, 0, 0, 0);
    const uint32_t mask = valid ? start(i, rec) : 0u;
    w.tree[lane] = rec;
    const bool has = mask != 0 && rec.y != 0;
    const unsigned m = __ballot_sync(kAll, has);
    if (has) w.e[__popc(m & below)] = make_uint2(0u, lane | mask << 6);
    uint32_t count = __popc(m);
    __syncwarp();
    for (uint32_t guard = 0; count != 0; ++guard) {
      uint32_t n = count < 32u ? count : 32u;
      const uint32_t room = kStack - kReserve > count ? kStack - kReserve - count : 1u;
      if (room < n) n = room;
      if (guard / 32u > 2 * F.all.n + 2 || count > kStack - 2) {
        raise_error(err, kErrTraversal);
        break;
      }
      count -= n;
      const bool on = lane < n;
      const uint2 e = on ? w.e[count + lane] : make_uint2(0, 0);
      __syncwarp();
      const uint32_t slot = e.y & 31u, tests = on ? within(slot, e.y >> 6) : 0u;
      uint32_t hit = 0, down = 0, esc = 0;
      bool inner = false;
      int4 t = make_int4(0, 0, 0, 0);
      if (tests) {
        t = w.tree[slot];
        const float4 l = F.all.lo[t.z + (int)e.x], h = F.all.hi[t.z + (int)e.x];
        down = (uint32_t)__float_as_int(l.w);
        esc = (uint32_t)__float_as_int(h.w);
        inner = (int)e.x < t.y - 1;
        hit = test(l, h, slot, tests);
      }
      const bool deeper = inner && hit != 0, sibling = tests && (e.y & 32u);
      const unsigned ms = __ballot_sync(kAll, sibling), md = __ballot_sync(kAll, deeper);
      if (sibling) w.e[count + __popc(ms & below)] = make_uint2(esc, slot | tests << 6);
      count += __popc(ms);
      if (deeper) w.e[count + __popc(md & below)] = make_uint2(down, slot | 32u | hit << 6);
      count += __popc(md);
      __syncwarp();
      leaf(inner ? 0u : hit, slot, (uint32_t)t.x + down, e.x - (uint32_t)(t.y - 1));
    }
    finish(valid, i, rec);
    __syncwarp();
  }
}

// VF-DCD (nearest obstacle point of the predicted vertex) and VF-CCD (first obstacle hit of the
// segment x0 -> x) of one vertex, two tests of one query (GenerateVF_DCD_Kernel,
// GenerateVFCCD_Kernel), with the nodes they share fetched once.
struct VfShared {
  PairStack stack;
  TestQueue<64> dq, cq;
  float4 x[32], x0[32], dir[32];  // dir.w = length
  unsigned long long dkey[32], ckey[32];
  uint32_t found[32];  // leaves of the first test | of the second << 16
};
__global__ void __launch_bounds__(kGenBlock) k_generate_vf(LbvhForest F, InstView I,
                                                        const float4* __restrict__ x,
                                                        const float4* __restrict__ x0,
                                                        uint32_t nv, int* __restrict__ vf_idx,
                                                        float4* __restrict__ vf_qs,
                                                        float4* __restrict__ vf_ns,
                                                        int* __restrict__ rt_idx,
                                                        float4* __restrict__ rt_qc,
                                                        float4* __restrict__ rt_nc, uint32_t* err,
                                                        uint32_t* counter, uint32_t packet) {
  __shared__ VfShared shared[kGenWarps];
  VfShared& w = shared[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t dcount = 0, ccount = 0;
  auto nearest = [&](uint4 e, bool on) {
    if (!on) return;
    f3 qs;
    const float4* p = F.all.pred + 3 * (size_t)e.x;
    keep_nearest(w.dkey[e.z], nearest_point(mk3(w.x[e.z]), mk3(p[0]), mk3(p[1]), mk3(p[2]), qs), e.y);
  };
  auto ray = [&](uint4 e, bool on) {
    if (!on) return;
    const float4* p = F.all.pred + 3 * (size_t)e.x;
    const float4 d = w.dir[e.z];
    keep_nearest(w.ckey[e.z],
                 ray_intersect(mk3(w.x0[e.z]), mk3(d), d.w, mk3(p[0]), mk3(p[1]), mk3(p[2])), e.y);
  };
  auto leaves = [&](uint32_t hit, uint32_t slot, uint32_t element, uint32_t place) {
    queue_push(w.dq, dcount, hit & 1u, element, place, slot, nearest);
    queue_push(w.cq, ccount, hit & 2u, element, place, slot, ray);
  };
  auto flush = [&]() {
    queue_flush(w.dq, dcount, nearest);
    queue_flush(w.cq, ccount, ray);
  };
  pair_loop(
      w.stack, F, counter, nv, packet, err,
      [&](uint32_t i, int4& rec) {
        rec = forest_rec(F, inst_index(I, i));
        const f3 p = mk3(x[i]), p0 = mk3(x0[i]);
        f3 dir = p - p0;
        const float len = length(dir);
        const bool still = len < kEps;  // a still vertex casts no ray
        if (!still) dir = dir / len;
        w.x[lane] = mk4(p, 0.0f);
        w.x0[lane] = mk4(p0, 0.0f);
        w.dir[lane] = mk4(dir, len);
        w.dkey[lane] = w.ckey[lane] = no_result();
        w.found[lane] = 0;
        return still ? 1u : 3u;
      },
      [&](uint32_t slot, uint32_t mask) {
        const uint32_t found = w.found[slot];
        if ((found & 0xFFFFu) > kMaxCandidates) mask &= ~1u;
        if (found >> 16 > kMaxCandidates) mask &= ~2u;
        return mask;
      },
      [&](float4 l, float4 h, uint32_t slot, uint32_t mask) {
        const f3 p = mk3(w.x[slot]);
        uint32_t hit = (mask & 1u) && overlap_point(l, h, p) ? 1u : 0u;
        if ((mask & 2u) && overlap_segment(l, h, mk3(w.x0[slot]), p)) hit |= 2u;
        return hit;
      },
      [&](uint32_t hit, uint32_t slot, uint32_t element, uint32_t place) {
        if (hit) atomicAdd(&w.found[slot], (hit & 1u) | (hit & 2u) << 15);
        leaves(hit, slot, element, place);
      },
      [&](bool valid, uint32_t i, int4 rec) {
        flush();
        const LbvhView b{(uint32_t)rec.y, F.all.pred + 3 * (size_t)rec.x, F.all.lo + rec.z,
                         F.all.hi + rec.z};
        const f3 p = mk3(w.x[lane]), p0 = mk3(w.x0[lane]);
        // beyond the cap: again in order, one walk per test
#pragma unroll 1
        for (uint32_t k = 1; k <= 2; ++k) {
          const uint32_t found = k == 1 ? w.found[lane] & 0xFFFFu : w.found[lane] >> 16;
          const bool again = valid && found > kMaxCandidates;
          if (!__any_sync(0xFFFFFFFFu, again)) continue;
          TraverseState st = lbvh_begin(b);
          if (!again) st.node = -1;
          else (k == 1 ? w.dkey[lane] : w.ckey[lane]) = no_result();
          __syncwarp();
          bool walks = true;
          while (__any_sync(0xFFFFFFFFu, walks)) {
            uint32_t f = kNone, place = 0;
            const uint32_t at = (uint32_t)st.node;
            walks = lbvh_step(
                b, st,
                [&](float4 l, float4 h) {
                  return k == 1 ? overlap_point(l, h, p) : overlap_segment(l, h, p0, p);
                },
                [&](uint32_t o) {
                  f = (uint32_t)rec.x + o;
                  place = at - (b.n - 1);
                },
                err);
            __syncwarp();
            leaves(f != kNone ? k : 0u, lane, f, place);
          }
          flush();
        }
        if (!valid) return;
        const unsigned long long d = w.dkey[lane], c = w.ckey[lane];
        f3 dqs = mk3(0, 0, 0), cqc = dqs;
        int didx = -1, cidx = -1;
        if (d != no_result()) {
          const int f = __float_as_int(b.lo[b.n - 1 + (uint32_t)d].w);
          const f3 v0 = mk3(b.pred[3 * f]), v1 = mk3(b.pred[3 * f + 1]), v2 = mk3(b.pred[3 * f + 2]);
          nearest_point(p, v0, v1, v2, dqs);
          didx = rec.x + f;
          vf_ns[i] = mk4(face_normal(v0, v1, v2), 0.0f);
        }
        if (c != no_result()) {
          cqc = p0 + __uint_as_float((uint32_t)(c >> 32)) * mk3(w.dir[lane]);
          const int f = __float_as_int(b.lo[b.n - 1 + (uint32_t)c].w);
          cidx = rec.x + f;
          rt_nc[i] = mk4(face_normal(mk3(b.pred[3 * f]), mk3(b.pred[3 * f + 1]),
                                     mk3(b.pred[3 * f + 2])), 0.0f);
        }
        vf_idx[i] = didx;
        vf_qs[i] = mk4(dqs, 0.0f);
        rt_idx[i] = cidx;
        rt_qc[i] = mk4(cqc, 0.0f);
      });
}

// EE-DCD: closest R-triangle-owned obstacle edge to each cloth edge (GenerateEE_DCD_Kernel).  The
// queued leaves are taken apart 32 at a time into the edges they own (none to three), and those
// are tested 32 at a time; element and place of an edge are three times the leaf's, plus its own.
struct EeShared {
  PairStack stack;
  TestQueue<64> leaves;
  TestQueue<128> edges;
  float4 p[32], q[32];
  unsigned long long key[32];
  uint32_t found[32];
};
__global__ void __launch_bounds__(kGenBlock) k_generate_ee(LbvhForest F, InstView I,
                                                        const float4* __restrict__ x,
                                                        const uint2* __restrict__ edge, uint32_t ne,
                                                        const int4* __restrict__ otri,
                                                        float4* __restrict__ ee_a,
                                                        float4* __restrict__ ee_b,
                                                        float4* __restrict__ ee_c,
                                                        float4* __restrict__ ee_rec,
                                                        uint8_t* __restrict__ vflag, uint32_t* err,
                                                        uint32_t* counter, uint32_t packet) {
  __shared__ EeShared shared[kGenWarps];
  EeShared& w = shared[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t nleaf = 0, nedge = 0;
  auto closest = [&](uint4 e, bool on) {
    if (!on) return;
    const uint32_t a = e.y % 3u;
    const float4* pred = F.all.pred;
    float s, t;
    f3 c1, c2;
    if (closest_seg_seg(mk3(w.p[e.z]), mk3(w.q[e.z]), mk3(pred[e.x]),
                        mk3(pred[a == 2 ? e.x - 2 : e.x + 1]), s, t, c1, c2) != 0.0f)
      keep_nearest(w.key[e.z], length(c1 - c2), e.y);
  };
  auto take_apart = [&](uint4 e, bool on) {
    const uint32_t own = on ? (uint32_t)otri[e.x].w >> 3 & 7u : 0u, k = __popc(own);
    const unsigned below = (1u << lane) - 1u;
    const unsigned m0 = __ballot_sync(0xFFFFFFFFu, k & 1u), m1 = __ballot_sync(0xFFFFFFFFu, k & 2u);
    uint32_t at = nedge + __popc(m0 & below) + 2 * __popc(m1 & below);
#pragma unroll
    for (uint32_t a = 0; a < 3; ++a)
      if (own >> a & 1u) w.edges.entry[at++] = make_uint4(3 * e.x + a, 3 * e.y + a, e.z, 0);
    nedge += __popc(m0) + 2 * __popc(m1);
    __syncwarp();
    while (nedge >= 32) {
      nedge -= 32;
      closest(w.edges.entry[nedge + lane], true);
    }
    __syncwarp();
  };
  auto flush = [&]() {
    queue_flush(w.leaves, nleaf, take_apart);
    queue_flush(w.edges, nedge, closest);
  };
  pair_loop(
      w.stack, F, counter, ne, packet, err,
      [&](uint32_t e, int4& rec) {
        const uint2 ed = edge[e];
        rec = forest_rec(F, inst_index(I, ed.x));
        w.p[lane] = x[ed.x];
        w.q[lane] = x[ed.y];
        w.key[lane] = no_result();
        w.found[lane] = 0;
        return 1u;
      },
      [&](uint32_t slot, uint32_t mask) { return w.found[slot] > kMaxCandidates ? 0u : mask; },
      [&](float4 l, float4 h, uint32_t slot, uint32_t mask) {
        return overlap_segment(l, h, mk3(w.p[slot]), mk3(w.q[slot])) ? 1u : 0u;
      },
      [&](uint32_t hit, uint32_t slot, uint32_t element, uint32_t place) {
        if (hit) atomicAdd(&w.found[slot], 1u);
        queue_push(w.leaves, nleaf, hit != 0, element, place, slot, take_apart);
      },
      [&](bool valid, uint32_t e, int4 rec) {
        flush();
        const LbvhView b{(uint32_t)rec.y, F.all.pred + 3 * (size_t)rec.x, F.all.lo + rec.z,
                         F.all.hi + rec.z};
        const bool again = valid && w.found[lane] > kMaxCandidates;
        if (__any_sync(0xFFFFFFFFu, again)) {  // beyond the cap: again, in order
          const f3 pc = mk3(w.p[lane]), qc = mk3(w.q[lane]);
          TraverseState st = lbvh_begin(b);
          if (!again) st.node = -1;
          else w.key[lane] = no_result();
          __syncwarp();
          bool walks = true;
          while (__any_sync(0xFFFFFFFFu, walks)) {
            uint32_t f = kNone, place = 0;
            const uint32_t at = (uint32_t)st.node;
            walks = lbvh_step(
                b, st, [&](float4 l, float4 h) { return overlap_segment(l, h, pc, qc); },
                [&](uint32_t o) {
                  f = (uint32_t)rec.x + o;
                  place = at - (b.n - 1);
                },
                err);
            __syncwarp();
            queue_push(w.leaves, nleaf, f != kNone, f, place, lane, take_apart);
          }
          flush();
        }
        if (!valid) return;
        const unsigned long long key = w.key[lane];
        float min_dist = kScalarMax, s = 0, t = 0;
        f3 p2 = mk3(0, 0, 0), q2 = p2, fn = p2;
        if (key != no_result()) {
          const uint32_t a = (uint32_t)key % 3u;
          const int f = __float_as_int(b.lo[b.n - 1 + (uint32_t)key / 3u].w);
          const f3 v0 = mk3(b.pred[3 * f]), v1 = mk3(b.pred[3 * f + 1]), v2 = mk3(b.pred[3 * f + 2]);
          p2 = a == 0 ? v0 : a == 1 ? v1 : v2;
          q2 = a == 0 ? v1 : a == 1 ? v2 : v0;
          fn = face_normal(v0, v1, v2);
          f3 c1, c2;
          closest_seg_seg(mk3(w.p[lane]), mk3(w.q[lane]), p2, q2, s, t, c1, c2);
          min_dist = __uint_as_float((uint32_t)(key >> 32));
        }
        ee_a[e] = make_float4(min_dist, p2.x, p2.y, p2.z);
        ee_b[e] = make_float4(q2.x, q2.y, q2.z, s);
        ee_c[e] = make_float4(fn.x, fn.y, fn.z, t);
        const f3 c2 = (1 - t) * p2 + t * q2;
        ee_rec[2 * (size_t)e] = make_float4(c2.x, c2.y, c2.z, s);
        ee_rec[2 * (size_t)e + 1] = make_float4(fn.x, fn.y, fn.z, min_dist);
        if (min_dist <= 1e6f) {  // a contact (the EE solve's test): flag both endpoints
          const uint2 ed = edge[e];
          vflag[ed.x] = 1;
          vflag[ed.y] = 1;
        }
      });
}

}  // namespace

// One wave of spread blocks (512 vertices an SM) is faster for bodies of revolution whatever the ring
// (ring 84, 6,890 vertices 30 -> 5.6 us) and up to 1.5 us either way for meshes without poles.  Beyond it
// a lane per vertex is, until its longest ring, 0.32 us a face, takes longer than the extra waves:
// without poles 78,400 vertices take 12.0 us spread and 7.2 a lane each, 160,000 19.9 and 10.1; ring 24
// 82,680 10.0 and 11.8, 165,000 15.8 and 13.0; ring 48 165,000 17.3 and 27.5, 330,000 33.6 and 32.3; ring
// 84 660,000 62 and 70, 1.4 M 119 and 91.
static bool uses_spread_fans(const Context& c) {
  return c.onv <= 512u * (uint32_t)c.num_sms || c.longest_fan > c.onv / 5000u;
}

void launch_obstacle_pass(Context& c, int step, int num_steps) {
  if (c.onv == 0) return;
  const float alpha = ((float)step + 1.0f) / (float)num_steps;
  const bool spread = uses_spread_fans(c);
  const unsigned block = spread ? kFanThreads<true> : kFanThreads<false>;
  (spread ? k_obstacle_pass<true> : k_obstacle_pass<false>)<<<grid_for(c.onv, block), block, 0,
                                                               c.stream>>>(
      c.ox0.p, c.ox.p, c.ox1.p, c.on1.p, c.otri.p, c.ovf_ptr.p, c.ovf_list.p, c.onv, alpha);
  launch_refit_midstep(c.bvh, c.ox1.p, c.on1.p, c.otri.p, c.params.bvh_tolerance, c.stream, c.err.p);
}

// Persistent warps: at most as many blocks as stay resident (six per SM) take packets until the
// counter passes the end.  A large packet fills its warp's rounds; a small one is done sooner and
// spreads the queries.  The largest with two packets per resident warp: of 11,495 / 33,950 queries
// (VF / EE) packets of 32, 8, 4 take 37, 32, 30 / 57, 39, 33 us, of 65,536 / 195,841 queries packets
// of 32, 16, 8, 4 take 32, 30, 30, 31 / 49, 43, 41, 45, of 0.9 / 2.7 M queries 32, 16, 8 take
// 107, 132, 176 / 251, 317, 432.
struct GenGrid {
  unsigned blocks, packet;
};
static GenGrid gen_grid(const Context& c, uint32_t nq) {
  const unsigned blocks = (unsigned)c.num_sms * 6u;
  unsigned packet = 32;
  while (packet > 4 && nq / packet < 2 * blocks * kGenWarps) packet /= 2;
  return {std::min((nq - 1) / (packet * kGenWarps) + 1, blocks), packet};
}

void launch_generate_contacts(Context& c) {
  if (!c.bvh.active) return;
  const LbvhForest F = c.bvh.forest();
  const InstView I = c.inst_view();
  cudaMemsetAsync(c.gen_counter.p, 0, sizeof(uint32_t) * 3, c.stream);
  cudaMemsetAsync(c.ee_vflag.p, 0, c.nv, c.stream);  // this pass's contacts set it
  const GenGrid v = gen_grid(c, c.nv), e = gen_grid(c, c.ne);
  k_generate_vf<<<v.blocks, kGenBlock, 0, c.stream>>>(F, I, c.x.p, c.x0.p, c.nv, c.vf_idx.p,
                                                      c.vf_qs.p, c.vf_ns.p, c.rt_idx.p, c.rt_qc.p,
                                                      c.rt_nc.p, c.err.p,
                                                      c.gen_counter.p, v.packet);
  k_generate_ee<<<e.blocks, kGenBlock, 0, c.stream>>>(F, I, c.x.p, c.edge.p, c.ne, c.otri.p,
                                                      c.ee_a.p, c.ee_b.p, c.ee_c.p, c.ee_rec.p,
                                                      c.ee_vflag.p,
                                                      c.err.p, c.gen_counter.p + 2, e.packet);
}

void launch_obstacle_commit(Context& c) {
  if (c.onv == 0) return;
  const bool spread = uses_spread_fans(c);
  const unsigned block = spread ? kFanThreads<true> : kFanThreads<false>;
  (spread ? k_obstacle_commit<true> : k_obstacle_commit<false>)<<<grid_for(c.onv, block), block, 0,
                                                                   c.stream>>>(
      c.ox.p, c.ox0.p, c.on.p, c.otri.p, c.ovf_ptr.p, c.ovf_list.p, c.onv);
}

void launch_vertex_normals(const float4* x, const int4* tri, const uint32_t* ptr,
                           const uint32_t* list, float4* out, uint32_t nv, cudaStream_t s) {
  if (nv == 0) return;
  k_vertex_normals<<<grid_for(nv, kFanBlock), kFanBlock, 0, s>>>(x, tri, ptr, list, out, nv);
}

void launch_prims_obstacle(Context& c, float tol) {
  launch_prims_from_mesh(c.bvh, c.ox0.p, c.on.p, c.otri.p, c.onf, tol, c.stream);
}

}  // namespace xrt
