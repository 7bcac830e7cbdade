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

__global__ void k_obstacle_pass(const float4* __restrict__ x0, const float4* __restrict__ x,
                                float4* __restrict__ x1, float4* __restrict__ n1,
                                const int4* __restrict__ tri, const uint32_t* __restrict__ ptr,
                                const uint32_t* __restrict__ list, uint32_t nv, float alpha) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const f3 xi = lerp_pos(x0, x, i, alpha);
  f3 acc = mk3(0, 0, 0);
  for (uint32_t k = ptr[i]; k < ptr[i + 1]; ++k) {
    const uint32_t fc = list[k];
    const int4 t = tri[fc >> 2];
    const int id[3] = {t.x, t.y, t.z};
    const int j = (int)(fc & 3u);
    const f3 e0 = lerp_pos(x0, x, id[(j + 1) % 3], alpha) - xi;
    const f3 e1 = lerp_pos(x0, x, id[(j + 2) % 3], alpha) - xi;
    acc = acc + cross(e0, e1) / (dot(e0, e0) * dot(e1, e1));
  }
  x1[i] = mk4(xi, 0.0f);
  n1[i] = mk4(normalize(acc), 0.0f);
}

__global__ void k_vertex_normals(const float4* __restrict__ x, const int4* __restrict__ tri,
                                 const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ list,
                                 float4* __restrict__ out, uint32_t nv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const f3 xi = mk3(x[i]);
  f3 acc = mk3(0, 0, 0);
  for (uint32_t k = ptr[i]; k < ptr[i + 1]; ++k) {
    const uint32_t fc = list[k];
    const int4 t = tri[fc >> 2];
    const int id[3] = {t.x, t.y, t.z};
    const int j = (int)(fc & 3u);
    const f3 e0 = mk3(x[id[(j + 1) % 3]]) - xi;
    const f3 e1 = mk3(x[id[(j + 2) % 3]]) - xi;
    acc = acc + cross(e0, e1) / (dot(e0, e0) * dot(e1, e1));
  }
  out[i] = mk4(normalize(acc), 0.0f);
}

// Frame end: x0 = x, then normals of the new x0 (computed from x, which is the same data).
__global__ void k_obstacle_commit(const float4* __restrict__ x, float4* __restrict__ x0,
                                  float4* __restrict__ nrm, const int4* __restrict__ tri,
                                  const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ list,
                                  uint32_t nv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const f3 xi = mk3(x[i]);
  f3 acc = mk3(0, 0, 0);
  for (uint32_t k = ptr[i]; k < ptr[i + 1]; ++k) {
    const uint32_t fc = list[k];
    const int4 t = tri[fc >> 2];
    const int id[3] = {t.x, t.y, t.z};
    const int j = (int)(fc & 3u);
    const f3 e0 = mk3(x[id[(j + 1) % 3]]) - xi;
    const f3 e1 = mk3(x[id[(j + 2) % 3]]) - xi;
    acc = acc + cross(e0, e1) / (dot(e0, e0) * dot(e1, e1));
  }
  x0[i] = mk4(xi, 0.0f);
  nrm[i] = mk4(normalize(acc), 0.0f);
}

// ---- contact generation: one query per cloth vertex (VF) or edge (EE) ------------------------------
// Persistent warps whose lanes each walk the tree of their query's instance; lanes that are done
// take new queries from a counter together, once kRefill of them are idle (walks near the obstacle
// are hundreds of nodes long, the others end at the root).  A leaf's test is five to ten times a
// box test and meets few lanes at a time, so the lanes only walk: the leaves go to a queue in
// shared memory, and their tests run 32 at a time on full warps.  A query's result is the smallest
// distance, and of equal ones that of the first leaf, kept as the minimum of (distance, place in
// the walk) in one 64-bit word: the distances are not negative, so their bits compare as they do,
// and a walk meets the leaves in the order of their tree positions.  The winner's data are computed
// again at the end.  So each query tests the same nodes and leaves as in a walk by itself, with the
// same cap, and the results are the same.  Contacts record global triangle ids.
// Against walks that ran each leaf's test in place (7.7 of 32 lanes busy): 24 garments on bodies of
// 13,776 triangles EE 740 -> 430 us, VF 340 -> 300 us; a 256 x 256 cloth EE 155 -> 75, VF 105 -> 72.
// A warp walking the union of its lanes' nodes instead: 1,000 and 410 us, 95 and 78 us.
constexpr int kGenWarps = kBlock / 32;
constexpr int kRefill = 8;

// A warp's queue of tests: x = element (global), y = place in the walk, z = lane that asks.
template <int N>
struct TestQueue {
  uint4 entry[N];
};
// Adds one test per lane with `on`; work(entry) runs 32 of them once there are as many.
template <class Work>
__device__ __forceinline__ void queue_push(TestQueue<64>& w, uint32_t& count, bool on,
                                           uint32_t element, uint32_t place, Work work) {
  const uint32_t lane = threadIdx.x & 31u;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, on);
  if (m == 0) return;
  if (on) w.entry[count + __popc(m & ((1u << lane) - 1u))] = make_uint4(element, place, lane, 0);
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
  if (count == 0) return;
  const uint32_t lane = threadIdx.x & 31u;
  const bool on = lane < count;
  const uint4 e = on ? w.entry[lane] : make_uint4(0, 0, 0, 0);
  count = 0;
  __syncwarp();
  work(e, on);
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

// The loop of a warp: start(query) sets a lane's query up, step() visits one node on all lanes and
// returns whether the lane's walk goes on, flush() runs the tests still queued, finish(query)
// writes the result.
template <class Start, class Step, class Flush, class Finish>
__device__ __forceinline__ void query_loop(uint32_t* counter, uint32_t nq, Start start, Step step,
                                           Flush flush, Finish finish) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t q = kNone;
  bool walks = false, drained = false;  // drained: the counter has passed nq
  for (;;) {
    const unsigned idle = __ballot_sync(kAll, !walks);
    if (idle == kAll || (!drained && __popc(idle) >= kRefill)) {
      flush();
      __syncwarp();
      if (!walks && q != kNone) {
        finish(q);
        q = kNone;
      }
      if (drained) return;
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(counter, (uint32_t)__popc(idle));
      base = __shfl_sync(kAll, base, 0);
      drained = base + (uint32_t)__popc(idle) >= nq;
      const uint32_t cand = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
      if (!walks && cand < nq) {
        q = cand;
        walks = start(q);
      }
      __syncwarp();
    }
    walks = step(walks);
  }
}

// VF-DCD (nearest obstacle point of the predicted vertex) and VF-CCD (first obstacle hit of the
// segment x0 -> x) of one vertex, in one walk of its instance's tree.  Each query keeps the state
// of its own stackless traversal: where its box test fails at an internal node that the other
// query enters, it stays off until the walk reaches that node's escape index (the first node
// after the subtree), and it stops after its own 256th leaf.  So each query tests the same nodes
// in the same order as alone, visits the same leaves in the same order and ends at the same cap:
// both results are those of the two separate traversals (GenerateVF_DCD_Kernel,
// GenerateVFCCD_Kernel), with the nodes they share fetched once.
struct VfShared {
  TestQueue<64> dq, cq;
  float4 x[32], x0[32], dir[32];  // dir.w = length
  unsigned long long dkey[32], ckey[32];
};
__global__ void __launch_bounds__(kBlock, 4) k_generate_vf(LbvhForest F, InstView I,
                                                        const float4* __restrict__ x,
                                                        const float4* __restrict__ x0,
                                                        uint32_t nv, int* __restrict__ vf_idx,
                                                        float4* __restrict__ vf_qs,
                                                        int* __restrict__ rt_idx,
                                                        float4* __restrict__ rt_qc, uint32_t* err,
                                                        uint32_t* counter) {
  constexpr int kOn = -1, kDone = -2;  // a query's state; >= 0: off until the walk reaches it
  __shared__ VfShared shared[kGenWarps];
  VfShared& w = shared[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  LbvhView b{};
  uint32_t base = 0, guard = 0, dfound = 0, cfound = 0, dcount = 0, ccount = 0;
  int node = -1, dstate = kDone, cstate = kDone;
  f3 px = mk3(0, 0, 0), p0 = px;
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
  query_loop(
      counter, nv,
      [&](uint32_t i) {
        const uint32_t sg = inst_index(I, i);
        b = forest_view(F, sg);
        base = (uint32_t)forest_rec(F, sg).x;
        px = mk3(x[i]);
        p0 = mk3(x0[i]);
        f3 dir = px - p0;
        const float len = length(dir);
        const bool still = len < kEps;  // a still vertex casts no ray
        if (!still) dir = dir / len;
        w.x[lane] = mk4(px, 0.0f);
        w.x0[lane] = mk4(p0, 0.0f);
        w.dir[lane] = mk4(dir, len);
        w.dkey[lane] = w.ckey[lane] = no_result();
        node = b.n == 0 ? -1 : 0;
        guard = dfound = cfound = 0;
        dstate = kOn;
        cstate = still ? kDone : kOn;
        return node != -1;
      },
      [&](bool on) {
        bool od = false, oc = false, leaf = false;
        uint32_t f = 0, place = 0;
        if (on) {
          if (dstate == node) dstate = kOn;  // the walk left the subtree the query skipped
          if (cstate == node) cstate = kOn;
          const bool don = dstate == kOn, con = cstate == kOn;
          const float4 l = b.lo[node], h = b.hi[node];
          od = don && overlap_point(l, h, px);
          oc = con && overlap_segment(l, h, p0, px);
          const int esc = __float_as_int(h.w), down = __float_as_int(l.w);
          leaf = (uint32_t)node >= b.n - 1;
          if (leaf) {
            f = base + (uint32_t)down;
            place = (uint32_t)node - (b.n - 1);
            if (od && ++dfound >= kMaxCandidates) dstate = kDone;
            if (oc && ++cfound >= kMaxCandidates) cstate = kDone;
            node = esc;
          } else if (od || oc) {
            // off for the subtree (an escape of -1: for the rest of the walk)
            if (don && !od) dstate = esc >= 0 ? esc : kDone;
            if (con && !oc) cstate = esc >= 0 ? esc : kDone;
            node = down;
          } else {
            node = esc;
          }
          if (dstate == kDone && cstate == kDone) node = -1;
          if (++guard > 2 * b.n + 2 && node != -1) {
            raise_error(err, kErrTraversal);
            node = -1;
          }
        }
        __syncwarp();
        queue_push(w.dq, dcount, leaf && od, f, place, nearest);
        queue_push(w.cq, ccount, leaf && oc, f, place, ray);
        return on && node != -1;
      },
      [&]() {
        queue_flush(w.dq, dcount, nearest);
        queue_flush(w.cq, ccount, ray);
      },
      [&](uint32_t i) {
        const unsigned long long d = w.dkey[lane], c = w.ckey[lane];
        f3 dqs = mk3(0, 0, 0), cqc = dqs;
        int didx = -1, cidx = -1;
        if (d != no_result()) {
          const int f = __float_as_int(b.lo[b.n - 1 + (uint32_t)d].w);
          nearest_point(px, mk3(b.pred[3 * f]), mk3(b.pred[3 * f + 1]), mk3(b.pred[3 * f + 2]), dqs);
          didx = (int)base + f;
        }
        if (c != no_result()) {
          cqc = p0 + __uint_as_float((uint32_t)(c >> 32)) * mk3(w.dir[lane]);
          cidx = (int)base + __float_as_int(b.lo[b.n - 1 + (uint32_t)c].w);
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
  TestQueue<64> leaves;
  TestQueue<128> edges;
  float4 p[32], q[32];
  unsigned long long key[32];
};
__global__ void __launch_bounds__(kBlock, 4) k_generate_ee(LbvhForest F, InstView I,
                                                        const float4* __restrict__ x,
                                                        const uint2* __restrict__ edge, uint32_t ne,
                                                        const int4* __restrict__ otri,
                                                        float4* __restrict__ ee_a,
                                                        float4* __restrict__ ee_b,
                                                        float4* __restrict__ ee_c,
                                                        uint8_t* __restrict__ vflag, uint32_t* err,
                                                        uint32_t* counter) {
  __shared__ EeShared shared[kGenWarps];
  EeShared& w = shared[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u;
  LbvhView b{};
  uint32_t base = 0, guard = 0, found = 0, nleaf = 0, nedge = 0;
  int node = -1;
  f3 pc = mk3(0, 0, 0), qc = pc;
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
  query_loop(
      counter, ne,
      [&](uint32_t e) {
        const uint2 ed = edge[e];
        const uint32_t sg = inst_index(I, ed.x);
        b = forest_view(F, sg);
        base = (uint32_t)forest_rec(F, sg).x;
        pc = mk3(x[ed.x]);
        qc = mk3(x[ed.y]);
        w.p[lane] = mk4(pc, 0.0f);
        w.q[lane] = mk4(qc, 0.0f);
        w.key[lane] = no_result();
        node = b.n == 0 ? -1 : 0;
        guard = found = 0;
        return node != -1;
      },
      [&](bool on) {
        bool hit = false;
        uint32_t f = 0, place = 0;
        if (on) {
          const float4 l = b.lo[node], h = b.hi[node];
          const bool ov = overlap_segment(l, h, pc, qc);
          const int esc = __float_as_int(h.w), down = __float_as_int(l.w);
          const bool leaf = (uint32_t)node >= b.n - 1;
          if (ov && leaf) {
            hit = true;
            f = base + (uint32_t)down;
            place = (uint32_t)node - (b.n - 1);
          }
          node = ov && !leaf ? down : esc;
          if (hit && ++found >= kMaxCandidates) node = -1;
          if (++guard > 2 * b.n + 2 && node != -1) {
            raise_error(err, kErrTraversal);
            node = -1;
          }
        }
        __syncwarp();
        queue_push(w.leaves, nleaf, hit, f, place, take_apart);
        return on && node != -1;
      },
      [&]() {
        queue_flush(w.leaves, nleaf, take_apart);
        queue_flush(w.edges, nedge, closest);
      },
      [&](uint32_t e) {
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
          closest_seg_seg(pc, qc, p2, q2, s, t, c1, c2);
          min_dist = __uint_as_float((uint32_t)(key >> 32));
        }
        ee_a[e] = make_float4(min_dist, p2.x, p2.y, p2.z);
        ee_b[e] = make_float4(q2.x, q2.y, q2.z, s);
        ee_c[e] = make_float4(fn.x, fn.y, fn.z, t);
        if (min_dist <= 1e6f) {  // a contact (the EE solve's test): flag both endpoints
          const uint2 ed = edge[e];
          vflag[ed.x] = 1;
          vflag[ed.y] = 1;
        }
      });
}

}  // namespace

void launch_obstacle_pass(Context& c, int step, int num_steps) {
  if (c.onv == 0) return;
  const float alpha = ((float)step + 1.0f) / (float)num_steps;
  k_obstacle_pass<<<grid_for(c.onv), kBlock, 0, c.stream>>>(c.ox0.p, c.ox.p, c.ox1.p, c.on1.p,
                                                            c.otri.p, c.ovf_ptr.p, c.ovf_list.p,
                                                            c.onv, alpha);
  launch_refit_midstep(c.bvh, c.ox1.p, c.on1.p, c.otri.p, c.params.bvh_tolerance, c.stream, c.err.p);
}

void launch_generate_contacts(Context& c) {
  if (!c.bvh.active) return;
  const LbvhForest F = c.bvh.forest();
  const InstView I = c.inst_view();
  // persistent work queues: a few resident waves of blocks fetch queries until the counters
  // pass the end
  const unsigned cap = (unsigned)c.num_sms * 8u;
  cudaMemsetAsync(c.gen_counter.p, 0, sizeof(uint32_t) * 3, c.stream);
  cudaMemsetAsync(c.ee_vflag.p, 0, c.nv, c.stream);  // this pass's contacts set it
  k_generate_vf<<<std::min(grid_for(c.nv), cap), kBlock, 0, c.stream>>>(
      F, I, c.x.p, c.x0.p, c.nv, c.vf_idx.p, c.vf_qs.p, c.rt_idx.p, c.rt_qc.p, c.err.p,
      c.gen_counter.p);
  k_generate_ee<<<std::min(grid_for(c.ne), cap), kBlock, 0, c.stream>>>(
      F, I, c.x.p, c.edge.p, c.ne, c.otri.p, c.ee_a.p, c.ee_b.p, c.ee_c.p, c.ee_vflag.p, c.err.p,
      c.gen_counter.p + 2);
}

void launch_obstacle_commit(Context& c) {
  if (c.onv == 0) return;
  k_obstacle_commit<<<grid_for(c.onv), kBlock, 0, c.stream>>>(c.ox.p, c.ox0.p, c.on.p, c.otri.p,
                                                              c.ovf_ptr.p, c.ovf_list.p, c.onv);
}

void launch_vertex_normals(const float4* x, const int4* tri, const uint32_t* ptr,
                           const uint32_t* list, float4* out, uint32_t nv, cudaStream_t s) {
  if (nv == 0) return;
  k_vertex_normals<<<grid_for(nv), kBlock, 0, s>>>(x, tri, ptr, list, out, nv);
}

void launch_prims_obstacle(Context& c, float tol) {
  launch_prims_from_mesh(c.bvh, c.ox0.p, c.on.p, c.otri.p, c.onf, tol, c.stream);
}

}  // namespace xrt
