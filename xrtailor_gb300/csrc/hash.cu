// hash.cu — Swift particle self-collision: uniform-grid hash, stable sort, cell ranges,
// neighbor cache and the Jacobi push-out with friction.
//
//   ComputeIntCoord/HashCoords ...... xrtailor/src/physics/broad_phase/spatial_hash/SpatialHashGPU.cu:9-25
//   FindCellStart_Kernel ............ SpatialHashGPU.cu:27-54
//   CacheNeighbors_Kernel ........... SpatialHashGPU.cu:56-99
//   HashObjects ..................... SpatialHashGPU.cu:128-160 (cub radix sort -> radix.cu)
//   CollideParticles_Kernel ......... xrtailor/src/physics/ClothSolverHelper.cu:171-219
//   ComputeFriction / ApplyDeltas ... ClothSolverHelper.cu:139-169
//
// The push-out reads positions from one buffer and writes the relaxed result to the other (the
// caller swaps them), which is the reference's deltas + ApplyDeltas pair in one launch.
#include "common.cuh"
#include "context.h"
#include "lbvh_dev.cuh"
#include "project_dev.cuh"

namespace xrt {
namespace {

__device__ __forceinline__ int int_coord(float value, float spacing) {
  return (int)floorf(value / spacing);
}
__device__ __forceinline__ int hash_coords(int x, int y, int z, int table) {
  const int h = (int)(((uint32_t)x * 92837111u) ^ ((uint32_t)y * 689287499u) ^
                      ((uint32_t)z * 283923481u));
  return abs(h % table);
}

// Keys of instance s lie in [table_base, table_base + table_size): each instance hashes into its
// own table of 2 V_s cells (the reference's 2V for that cloth alone), laid end to end.
__global__ void k_hash(const float4* __restrict__ x, uint32_t nv, InstView I,
                       uint32_t* __restrict__ key, uint32_t* __restrict__ val) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  const InstanceRec r = inst_rec(I, inst_index(I, i));
  const float4 p = x[i];
  key[i] = r.table_base + (uint32_t)hash_coords(int_coord(p.x, r.spacing), int_coord(p.y, r.spacing),
                                                int_coord(p.z, r.spacing), (int)r.table_size);
  val[i] = i;
}

__global__ void k_cell_bounds(const uint32_t* __restrict__ skey, uint32_t nv,
                              uint32_t* __restrict__ cell_start, uint32_t* __restrict__ cell_end) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= nv) return;
  const uint32_t h = skey[id];
  if (id == 0 || h != skey[id - 1]) {
    cell_start[h] = id;
    if (id > 0) cell_end[skey[id - 1]] = id;
  }
  if (id == nv - 1) cell_end[h] = id + 1;
}

// A lane per vertex, cell by cell.
__global__ void k_cache_neighbors_lane(const uint32_t* __restrict__ sidx,
                                       const uint32_t* __restrict__ cell_start,
                                       const uint32_t* __restrict__ cell_end,
                                       const float4* __restrict__ x,
                                       const float4* __restrict__ x_init, uint32_t nv, InstView I,
                                       uint32_t maxnb, uint32_t* __restrict__ neighbors) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nv) return;
  const uint32_t id = sidx[tid];
  const InstanceRec r = inst_rec(I, inst_index(I, id));
  const float spacing = r.spacing, spacing2 = r.spacing2, d2 = r.d2;
  const int table = (int)r.table_size;
  const f3 pos = mk3(x[id]);
  const f3 orig = mk3(x_init[id]);
  const int ix = int_coord(pos.x, spacing), iy = int_coord(pos.y, spacing),
            iz = int_coord(pos.z, spacing);
  uint64_t ni = id;
  const uint64_t limit = (uint64_t)nv * maxnb;
  for (int xx = ix - 1; xx <= ix + 1; ++xx)
    for (int yy = iy - 1; yy <= iy + 1; ++yy)
      for (int zz = iz - 1; zz <= iz + 1; ++zz) {
        const uint32_t h = r.table_base + (uint32_t)hash_coords(xx, yy, zz, table);
        const uint32_t start = cell_start[h];
        if (start == kNone) continue;
        const uint32_t end = min(cell_end[h], start + maxnb);
        for (uint32_t k = start; k < end; ++k) {
          const uint32_t nb = sidx[k];
          const f3 dp = pos - mk3(x[nb]);
          const f3 d0 = orig - mk3(x_init[nb]);
          if (nb != id && dot(dp, dp) < spacing2 && dot(d0, d0) > d2) {
            neighbors[ni] = nb;
            ni += nv;
            if (ni >= limit) return;
          }
        }
      }
  if (ni < limit) neighbors[ni] = kNone;
}

// A warp per vertex: 27 lanes look up the cells around it, the cells' entries are numbered through in
// cell order, and 32 entries at a time are tested and appended in that order.  The same lists.
constexpr int kCells = 27;
__global__ void k_cache_neighbors(const uint32_t* __restrict__ sidx,
                                  const uint32_t* __restrict__ cell_start,
                                  const uint32_t* __restrict__ cell_end,
                                  const float4* __restrict__ x, const float4* __restrict__ x_init,
                                  uint32_t nv, InstView I, uint32_t maxnb,
                                  uint32_t* __restrict__ neighbors) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31u;
  if (warp >= nv) return;
  const uint32_t id = sidx[warp];
  const InstanceRec r = inst_rec(I, inst_index(I, id));
  const f3 pos = mk3(x[id]), orig = mk3(x_init[id]);
  // cell `lane`: z runs fastest, then y
  const int cx = (int)lane / 9, cy = (int)lane / 3 % 3, cz = (int)lane % 3;
  uint32_t start = 0, size = 0;
  if (lane < kCells) {
    const uint32_t h = r.table_base +
                       (uint32_t)hash_coords(int_coord(pos.x, r.spacing) - 1 + cx,
                                             int_coord(pos.y, r.spacing) - 1 + cy,
                                             int_coord(pos.z, r.spacing) - 1 + cz,
                                             (int)r.table_size);
    start = cell_start[h];
    const uint32_t end = cell_end[h];
    if (start != kNone) size = min(end, start + maxnb) - start;
  }
  uint32_t upto = size;  // entries of the cells up to this lane's
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const uint32_t o = __shfl_up_sync(kAll, upto, d);
    if (lane >= (uint32_t)d) upto += o;
  }
  const uint32_t total = __shfl_sync(kAll, upto, 31);
  start -= upto - size;  // entry e of the numbering is start + e of its cell
  uint32_t found = 0;
  for (uint32_t base = 0; base < total && found < maxnb; base += 32) {
    const uint32_t e = base + lane;
    uint32_t cell = 0;  // the first cell with upto > e
#pragma unroll
    for (int d = 16; d > 0; d /= 2)
      if (__shfl_sync(kAll, upto, (int)cell + d - 1) <= e) cell += d;
    const uint32_t first = __shfl_sync(kAll, start, (int)(cell & 31u));
    uint32_t nb = id;
    bool near = false;
    if (e < total) {
      nb = sidx[first + e];
      const f3 dp = pos - mk3(x[nb]);
      const f3 d0 = orig - mk3(x_init[nb]);
      near = nb != id && dot(dp, dp) < r.spacing2 && dot(d0, d0) > r.d2;
    }
    const unsigned m = __ballot_sync(kAll, near);
    const uint32_t at = found + __popc(m & ((1u << lane) - 1u));
    if (near && at < maxnb) neighbors[id + (size_t)nv * at] = nb;
    found += __popc(m);
  }
  if (lane == 0 && found < maxnb) neighbors[id + (size_t)nv * found] = kNone;
}

__device__ __forceinline__ f3 friction_of(float mu, f3 correction, f3 rel_vel) {
  f3 fr = mk3(0, 0, 0);
  const float cl = length(correction);
  if (mu > 0.0f && cl > 0.0f) {
    const f3 nrm = correction / cl;
    const f3 tan_vel = rel_vel - nrm * dot(rel_vel, nrm);
    const float tl = length(tan_vel);
    const float max_tl = cl * mu;
    fr = -tan_vel * tmin(max_tl / tl, 1.0f);
  }
  return fr;
}

// The two terms of a pair within reach, w_i * common and w_i * friction (CollideParticles_Kernel), in
// straight-line correctly rounded operations where the operands are in range (project_dev.cuh), and
// by the operators otherwise: the same bits.
struct PairTerm {
  f3 push, drag;
};
__device__ __noinline__ PairTerm pair_term_any(f3 diff, float distance, float diameter, float denom,
                                               float w_i, f3 rel, float mu) {
  const f3 gradient = diff / (distance + kEps);
  const float lambda = (distance - diameter) / denom;
  const f3 common = lambda * gradient;
  return PairTerm{w_i * common, w_i * friction_of(mu, common, rel)};
}
__device__ __forceinline__ bool quotient_range(float a) { return a == 0.0f || in_range(fabsf(a)); }
__device__ __forceinline__ bool quotient_range(f3 a) {
  return quotient_range(a.x) && quotient_range(a.y) && quotient_range(a.z);
}
// a / b with y = recip(b); a zero keeps its sign
__device__ __forceinline__ float div_by(float a, float b, float y) {
  float q = a * y;
  q = fmaf(fmaf(-b, q, a), y, q);
  q = fmaf(fmaf(-b, q, a), y, q);
  return a == 0.0f ? a : q;
}
__device__ __forceinline__ f3 div_by(f3 a, float b, float y) {
  return mk3(div_by(a.x, b, y), div_by(a.y, b, y), div_by(a.z, b, y));
}
__device__ __forceinline__ PairTerm pair_term(f3 diff, float dd, float distance, float diameter,
                                              float denom, float w_i, f3 rel, float mu) {
  const float reach = distance + kEps;
  const f3 gradient = div_by(diff, reach, recip(reach));
  const float depth = distance - diameter;  // < 0
  const float lambda = div_rn(depth, denom);
  const f3 common = lambda * gradient;
  const float cc = dot(common, common);
  const float cl = sqrt_rn(cc);
  const f3 nrm = div_by(common, cl, recip(cl));
  const f3 tan_vel = rel - nrm * dot(rel, nrm);
  const float tt = dot(tan_vel, tan_vel);
  const float tl = sqrt_rn(tt);
  const float max_tl = cl * mu;
  const float k = div_rn(max_tl, tl);
  const bool fine = in_range(dd) && in_range(-depth) && in_range(denom) && quotient_range(diff) &&
                    in_range(cc) && quotient_range(common) && mu > 0.0f && in_range(tt) &&
                    in_range(max_tl);
  if (!fine) return pair_term_any(diff, distance, diameter, denom, w_i, rel, mu);
  return PairTerm{w_i * common, w_i * (-tan_vel * tmin(k, 1.0f))};
}

// Particle push-out with friction for many vertices: a warp takes 32, one per lane.  Its lanes test
// their listed neighbors eight slots at a time (ids, then positions, all loads of a batch in flight)
// and push the pairs within reach, slot by slot, into a queue in shared memory; every 32 of them run
// on the whole warp, one pair per lane, and add their terms to the owners' sums.  The queue keeps
// each vertex's pairs in slot order, and of several pairs of one owner in a turn the earlier
// commits first, so the sums are the reference's.  Bounded by instructions: with the pair's 130
// in the lane that found it, a warp ran them for its longest list (20 slots where the mean is 8, of
// which 40% lie within reach).
constexpr uint32_t kQueue = 512;  // a batch of slots adds at most 256 to at most 31
struct CollideShared {
  float own[8][32];  // predicted position, weight, velocity, diameter
  float sum[3][32];
  uint32_t other[kQueue];
  uint8_t owner[kQueue];
};

__global__ void k_collide_queue(const float4* __restrict__ x_in, float4* __restrict__ x_out,
                                const float4* __restrict__ x0,
                                const uint32_t* __restrict__ neighbors, uint32_t nv,
                                uint32_t maxnb, InstView I, float mu, float relaxation) {
  extern __shared__ float4 smem[];
  pdl_release();
  pdl_wait();
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  CollideShared& sh = reinterpret_cast<CollideShared*>(smem)[threadIdx.x >> 5];
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  const bool has = id < nv;
  float4 pi = make_float4(0, 0, 0, 0);
  float reach2 = 0.0f;
  if (has) {
    const InstanceRec rec = inst_rec(I, inst_index(I, id));
    reach2 = rec.reach2;
    pi = x_in[id];
    const f3 v = mk3(pi) - mk3(x0[id]);
    const float own[8] = {pi.x, pi.y, pi.z, pi.w, v.x, v.y, v.z, rec.diameter};
#pragma unroll
    for (int k = 0; k < 8; ++k) sh.own[k][lane] = own[k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) sh.sum[k][lane] = 0.0f;
  __syncwarp();
  const f3 pred_i = mk3(pi);
  const float w_i = pi.w;
  uint32_t head = 0, queued = 0;  // the queue, the same in every lane
  int cnt = 0;
  auto run = [&](uint32_t n) {  // the queue's first n pairs (n <= 32)
    const bool on = lane < n;
    const uint32_t at = (head + lane) % kQueue;
    uint32_t o = 0;
    PairTerm t{mk3(0, 0, 0), mk3(0, 0, 0)};
    if (on) {
      o = sh.owner[at];
      const uint32_t j = sh.other[at];
      const float4 pj = x_in[j];
      const f3 oj = mk3(x0[j]);
      const f3 po = mk3(sh.own[0][o], sh.own[1][o], sh.own[2][o]);
      const f3 vo = mk3(sh.own[4][o], sh.own[5][o], sh.own[6][o]);
      const float wo = sh.own[3][o], diameter = sh.own[7][o];
      const f3 diff = po - mk3(pj);
      const float dd = dot(diff, diff);
      const float distance = in_range(dd) ? sqrt_rn(dd) : sqrtf(dd);
      t = pair_term(diff, dd, distance, diameter, wo + pj.w, wo, vo - (mk3(pj) - oj), mu);
    }
    unsigned peers = __ballot_sync(0xFFFFFFFFu, on);  // the pairs of this lane's owner
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const unsigned one = __ballot_sync(0xFFFFFFFFu, o >> b & 1u);
      peers &= o >> b & 1u ? one : ~one;
    }
    const uint32_t rank = (uint32_t)__popc(peers & below);
    for (uint32_t turn = 0; __any_sync(0xFFFFFFFFu, on && rank >= turn); ++turn) {
      if (on && rank == turn) {
        const f3 s = mk3(sh.sum[0][o], sh.sum[1][o], sh.sum[2][o]) - t.push + t.drag;
        sh.sum[0][o] = s.x;
        sh.sum[1][o] = s.y;
        sh.sum[2][o] = s.z;
      }
      __syncwarp();
    }
    head = (head + n) % kQueue;
    queued -= n;
  };
  constexpr uint32_t kBatch = 8;
  bool open = has;  // no id >= nv so far (reference: j > num_particles; j == nv never occurs)
  for (uint32_t base = 0; base < maxnb && __any_sync(0xFFFFFFFFu, open); base += kBatch) {
    uint32_t nb[kBatch];
#pragma unroll
    for (uint32_t r = 0; r < kBatch; ++r)
      nb[r] = open && base + r < maxnb ? neighbors[(uint64_t)(base + r) * nv + id] : nv;
    float4 pj[kBatch];
    uint32_t listed = 0;
#pragma unroll
    for (uint32_t r = 0; r < kBatch; ++r) {
      open = open && nb[r] < nv;
      pj[r] = open ? x_in[nb[r]] : make_float4(0, 0, 0, 0);
      if (open) listed |= 1u << r;
    }
#pragma unroll
    for (uint32_t r = 0; r < kBatch; ++r) {
      const f3 diff = pred_i - mk3(pj[r]);
      // distance >= diameter, without the root (reach2: the smallest square whose root reaches it)
      const bool hit = (listed >> r & 1u) && !(w_i + pj[r].w <= 0) && !(dot(diff, diff) >= reach2);
      const unsigned hits = __ballot_sync(0xFFFFFFFFu, hit);
      if (hits == 0) continue;
      if (hit) {
        const uint32_t at = (head + queued + (uint32_t)__popc(hits & below)) % kQueue;
        sh.other[at] = nb[r];
        sh.owner[at] = (uint8_t)lane;
        ++cnt;
      }
      queued += (uint32_t)__popc(hits);
    }
    __syncwarp();
    const bool last = base + kBatch >= maxnb || !__any_sync(0xFFFFFFFFu, open);
    while (queued >= 32 || (last && queued)) run(min(queued, 32u));
  }
  if (!has) return;
  const f3 pd = mk3(sh.sum[0][lane], sh.sum[1][lane], sh.sum[2][lane]);
  f3 q = pred_i;
  const float count = (float)cnt;
  if (count > 0.0f) q = q + pd / count * relaxation;
  x_out[id] = mk4(q, w_i);
}

// Particle push-out with friction, four lanes per vertex.  A lane takes neighbor slots q, q + 4, so
// eight slots' ids, positions and previous positions each arrive in one round trip; the terms
// go through shared memory and lane q adds component q of them in slot order, which is the
// reference's order.
constexpr int kCollideLanes = 4;
constexpr int kCollideRows = 2;  // slots per lane and turn
constexpr int kTermStride = 32 * kCollideRows + 1;  // keeps the four lanes' reads on distinct banks

__global__ void k_collide(const float4* __restrict__ x_in,
                          float* __restrict__ x_out, const float4* __restrict__ x0,
                          const uint32_t* __restrict__ neighbors, uint32_t nv, uint32_t maxnb,
                          InstView I, float mu, float relaxation) {
  extern __shared__ float s_term[];  // 6 kTermStride per warp
  pdl_release();
  pdl_wait();
  const uint32_t lane = threadIdx.x & 31u, q = lane & 3u;
  const uint32_t id = (blockIdx.x * blockDim.x + threadIdx.x) / kCollideLanes;
  float* term = s_term + (threadIdx.x >> 5) * (6 * kTermStride);
  const bool has = id < nv;
  uint32_t nb[kCollideRows];
#pragma unroll
  for (int r = 0; r < kCollideRows; ++r) {
    const uint32_t slot = kCollideLanes * r + q;
    nb[r] = has && slot < maxnb ? neighbors[(uint64_t)slot * nv + id] : nv;
  }
  float4 pi = make_float4(0, 0, 0, 0);
  f3 vel_i = mk3(0, 0, 0);
  float diameter = 0.0f;
  if (has) {
    diameter = inst_rec(I, inst_index(I, id)).diameter;
    pi = x_in[id];
    vel_i = mk3(pi) - mk3(x0[id]);
  }
  const f3 pred_i = mk3(pi);
  const float w_i = pi.w;
  float pd = 0.0f;  // component q
  int cnt = 0;
  for (uint32_t base = 0;; base += kCollideLanes * kCollideRows) {
    // the list ends at the first id >= nv (reference: j > num_particles; j == nv never occurs)
    bool on[kCollideRows];
    bool open = has;
#pragma unroll
    for (int r = 0; r < kCollideRows; ++r) {
      const unsigned ends = __ballot_sync(0xFFFFFFFFu, nb[r] >= nv) >> (lane & ~3u) & 0xFu;
      on[r] = open && (ends & ((2u << q) - 1u)) == 0;
      open = open && ends == 0;
    }
    float4 pj[kCollideRows], oj[kCollideRows];
#pragma unroll
    for (int r = 0; r < kCollideRows; ++r) {
      pj[r] = oj[r] = make_float4(0, 0, 0, 0);
      if (on[r]) {
        pj[r] = x_in[nb[r]];
        oj[r] = x0[nb[r]];
      }
    }
    const bool more = __any_sync(0xFFFFFFFFu, open);
    if (more) {  // the next turn's ids
#pragma unroll
      for (int r = 0; r < kCollideRows; ++r) {
        const uint32_t slot = base + kCollideLanes * (kCollideRows + r) + q;
        nb[r] = open && slot < maxnb ? neighbors[(uint64_t)slot * nv + id] : nv;
      }
    }
#pragma unroll
    for (int r = 0; r < kCollideRows; ++r) {
      const float denom = w_i + pj[r].w;
      const f3 diff = pred_i - mk3(pj[r]);
      const float dd = dot(diff, diff);
      bool hit = on[r] && !(denom <= 0);
      const float distance = in_range(dd) ? sqrt_rn(dd) : sqrtf(dd);
      hit = hit && !(distance >= diameter);
      const unsigned hits = __ballot_sync(0xFFFFFFFFu, hit);
      if (hits == 0) continue;
      if (hit) {
        const f3 rel = vel_i - (mk3(pj[r]) - mk3(oj[r]));
        const PairTerm t = pair_term(diff, dd, distance, diameter, denom, w_i, rel, mu);
        float* o = term + 32 * r + lane;
        o[0] = t.push.x;
        o[kTermStride] = t.push.y;
        o[2 * kTermStride] = t.push.z;
        o[3 * kTermStride] = t.drag.x;
        o[4 * kTermStride] = t.drag.y;
        o[5 * kTermStride] = t.drag.z;
      }
      __syncwarp();
      const unsigned mine = hits >> (lane & ~3u) & 0xFu;
      cnt += __popc(mine);
      const float* o = term + min(q, 2u) * kTermStride + 32 * r + (lane & ~3u);
#pragma unroll
      for (int k = 0; k < kCollideLanes; ++k)
        if (mine >> k & 1u) {
          pd = pd - o[k];
          pd = pd + o[3 * kTermStride + k];
        }
      __syncwarp();
    }
    if (!more) break;
  }
  if (!has) return;
  const float count = (float)cnt;
  float v = q == 0 ? pi.x : (q == 1 ? pi.y : (q == 2 ? pi.z : pi.w));
  if (q < 3 && count > 0.0f) v = v + pd / count * relaxation;
  x_out[4 * (size_t)id + q] = v;
}

}  // namespace

void launch_hash(Context& c) {
  const uint32_t nv = c.nv;
  if (nv == 0) return;
  const uint32_t table = 2 * nv;  // the instances' tables end to end
  int bits = 0;
  while ((1u << bits) < table) ++bits;
  const InstView I = c.inst_view();
  k_hash<<<grid_for(nv), kBlock, 0, c.stream>>>(c.x.p, nv, I, c.hash_key.p, c.hash_val.p);
  uint32_t *skey = nullptr, *sidx = nullptr;
  c.hash_sorter.sort(c.hash_key.p, c.hash_val.p, nv, bits, c.stream, &skey, &sidx);
  cudaMemsetAsync(c.cell_start.p, 0xFF, sizeof(uint32_t) * table, c.stream);
  k_cell_bounds<<<grid_for(nv), kBlock, 0, c.stream>>>(skey, nv, c.cell_start.p, c.cell_end.p);
  // A lane's walk of its cells is a chain of about 100 us whatever the number of vertices; a warp per
  // vertex has no chain but issues more: 65,536 vertices 108 us by lanes and 39 by warps, 917 k 372 and
  // 483.  A hash's kernels take 11.6 and 10.7 us on average at 193,600 vertices, 12.5 and 12.4 at 243,049,
  // 12.9 and 13.2 at 270,400, 18.5 and 20.3 at 490,000.
  if (nv <= 1600u * (uint32_t)c.num_sms)
    k_cache_neighbors<<<grid_for(nv, kBlock / 32), kBlock, 0, c.stream>>>(
        sidx, c.cell_start.p, c.cell_end.p, c.x.p, c.x_init.p, nv, I,
        (uint32_t)c.params.max_neighbor_size, c.neighbors.p);
  else
    k_cache_neighbors_lane<<<grid_for(nv), kBlock, 0, c.stream>>>(
        sidx, c.cell_start.p, c.cell_end.p, c.x.p, c.x_init.p, nv, I,
        (uint32_t)c.params.max_neighbor_size, c.neighbors.p);
}

void launch_collide(Context& c, const FrameConst& k) {
  const uint32_t block = c.vertex_block;
  // Four lanes per vertex shorten a launch that is bound by its lists' round trips; with many vertices
  // the instructions count, of which the queue issues half as many.  Frames of a folded sheet, four
  // lanes and queue: 65,536 vertices 2.18 and 2.25 ms, 108,900 2.82 and 2.83, 129,600 3.02 and 3.00,
  // 160,000 3.41 and 3.34; a launch on 917 k vertices 118 and 68 us.
  if (c.nv > 720u * (uint32_t)c.num_sms) {
    const size_t smem = sizeof(CollideShared) * (block / 32);
    if (raise_smem((const void*)k_collide_queue, smem) != cudaSuccess) return;
    launch_k(c.pdl, k_collide_queue, grid_for(c.nv, block), block, smem, c.stream, c.x.p, c.x_alt.p,
             c.x0.p, c.neighbors.p, c.nv, (uint32_t)c.params.max_neighbor_size, c.inst_view(),
             k.friction, k.relaxation);
    return;
  }
  launch_k(c.pdl, k_collide, grid_for(c.nv, block / kCollideLanes), block,
           sizeof(float) * 6 * kTermStride * (block / 32), c.stream, c.x.p,
           reinterpret_cast<float*>(c.x_alt.p), c.x0.p, c.neighbors.p, c.nv,
           (uint32_t)c.params.max_neighbor_size, c.inst_view(), k.friction, k.relaxation);
}

}  // namespace xrt
