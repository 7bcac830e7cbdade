// lbvh.cu — linear BVH over triangles: Morton codes, stable radix sort, Karras hierarchy,
// bottom-up boxes, escape tables, refit and stackless queries.
//
// Reference: xrtailor/src/physics/broad_phase/lbvh/BVH.cu — expand_bits/morton_code :22-46,
// determine_range/find_split :57-210, escape tables :212-273, Karras nodes :275-329,
// UpdateObjects :382-421, InitAABBs :423-462, ComputeMortons :465-479, AssignAABBCAS :515-538,
// Construct :618-722, RefitMidstep :770-818, QueryDeviceStackless :957-1055; box tests
// xrtailor/src/physics/broad_phase/Bounds.cu.
//
// Layout: node k keeps its box and its traversal links in two float4s (32 B, one sector):
//   lo = {lower.xyz, left child (internal) | object (leaf)}, hi = {upper.xyz, escape index}.
// A leaf is node >= n-1.  Stackless traversal therefore reads 32 contiguous bytes per visit.
// The hierarchy is that of 64-bit keys (code << 32 | object): for unique codes this is exactly the
// tree the reference builds on 32-bit codes (every common-prefix length is decided in the high
// word), and for duplicate codes it is the reference's own 64-bit fallback.
#include "common.cuh"
#include "context.h"
#include "lbvh_dev.cuh"

namespace xrt {
namespace {

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__device__ __forceinline__ uint32_t morton_code(f3 p) {
  const float res = 1024.0f;
  float x = tmin(tmax(p.x * res, 0.0f), res - 1.0f);
  float y = tmin(tmax(p.y * res, 0.0f), res - 1.0f);
  float z = tmin(tmax(p.z * res, 0.0f), res - 1.0f);
  return expand_bits((uint32_t)x) * 4 + expand_bits((uint32_t)y) * 2 + expand_bits((uint32_t)z);
}

// Order-preserving float <-> uint mapping for atomic min / max of the root box.  A NaN (the box of a
// triangle shrunk to a point) counts as -0.
__device__ __forceinline__ uint32_t f2o(float f) {
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7FFFFFFFu) > 0x7F800000u) return 0x7FFFFFFFu;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// A primitive's six vertices (v, then pred): float4 arrays, or 9 packed floats each.
struct Prims {
  const float4 *v, *pred;
  const float *v9, *p9;
};
struct Box {
  f3 lo, hi;
};
// InitAABBs_Kernel: bounds of v and pred, corners moved outwards by scr.
template <bool PACKED>
__device__ __forceinline__ Box leaf_box(const Prims& P, uint32_t i, float scr) {
  f3 v[3], q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (PACKED) {
      const float *a = P.v9 + 9 * (size_t)i + 3 * k, *b = P.p9 + 9 * (size_t)i + 3 * k;
      v[k] = mk3(a[0], a[1], a[2]);
      q[k] = P.p9 == P.v9 ? v[k] : mk3(b[0], b[1], b[2]);
    } else {
      v[k] = mk3(P.v[3 * (size_t)i + k]);
      q[k] = mk3(P.pred[3 * (size_t)i + k]);
    }
  }
  f3 bl = mk3(tmin(tmin(v[0].x, tmin(v[1].x, v[2].x)), tmin(q[0].x, tmin(q[1].x, q[2].x))),
              tmin(tmin(v[0].y, tmin(v[1].y, v[2].y)), tmin(q[0].y, tmin(q[1].y, q[2].y))),
              tmin(tmin(v[0].z, tmin(v[1].z, v[2].z)), tmin(q[0].z, tmin(q[1].z, q[2].z))));
  f3 bu = mk3(tmax(tmax(v[0].x, tmax(v[1].x, v[2].x)), tmax(q[0].x, tmax(q[1].x, q[2].x))),
              tmax(tmax(v[0].y, tmax(v[1].y, v[2].y)), tmax(q[0].y, tmax(q[1].y, q[2].y))),
              tmax(tmax(v[0].z, tmax(v[1].z, v[2].z)), tmax(q[0].z, tmax(q[1].z, q[2].z))));
  const f3 center = (bl + bu) * 0.5f;
  const f3 n1 = normalize(bl - center);
  const f3 n2 = normalize(bu - center);
  return Box{bl + scr * n1, bu + scr * n2};
}

// Root boxes are kept as integers that order like the floats, the lower corners complemented, so
// that 0 is neutral and every extremum is an atomicMax.  Extrema are exact, so the order of the
// reduction does not matter; a warp reduces floats, everything above integers.
// lane_extrema: one leaf's own.  In a warp of fewer than 32 leaves of a segment each lane commits, as
// ever (a box with a NaN, of a triangle shrunk to a point, counts there and not in fminf).
__device__ __forceinline__ void lane_extrema(const Box& b, uint32_t out[6]) {
  out[0] = ~f2o(b.lo.x); out[1] = ~f2o(b.lo.y); out[2] = ~f2o(b.lo.z);
  out[3] = f2o(b.hi.x); out[4] = f2o(b.hi.y); out[5] = f2o(b.hi.z);
}
__device__ __forceinline__ void warp_extrema(const Box& b, uint32_t out[6]) {
  const float sum = (b.lo.x + b.lo.y) + (b.lo.z + b.hi.x) + (b.hi.y + b.hi.z);
  if (!__any_sync(0xFFFFFFFFu, sum != sum)) {  // no NaN: the integers order alike
    lane_extrema(b, out);
#pragma unroll
    for (int k = 0; k < 6; ++k) out[k] = __reduce_max_sync(0xFFFFFFFFu, out[k]);
    return;
  }
  float lo[3] = {b.lo.x, b.lo.y, b.lo.z}, hi[3] = {b.hi.x, b.hi.y, b.hi.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[k] = fminf(lo[k], __shfl_xor_sync(0xFFFFFFFFu, lo[k], off));
      hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xFFFFFFFFu, hi[k], off));
    }
    out[k] = ~f2o(lo[k]);
    out[3 + k] = f2o(hi[k]);
  }
}
__device__ __forceinline__ Box empty_box() {
  const float inf = __int_as_float(0x7f800000);
  return Box{mk3(inf, inf, inf), mk3(-inf, -inf, -inf)};
}

// InitAABBs_Kernel + the root reduction (thrust::reduce of Bounds::Merge), per segment; clears the
// merge's slots.  A block whose leaves share a segment commits six extrema (one atomic each per
// warp put 392,000 on six words for 2.09 M triangles: 269 us against 32), a warp that straddles a
// segment boundary commits lane by lane.
template <bool PACKED>
__global__ void __launch_bounds__(kBlock) k_leaf_boxes(Prims P, uint32_t n, float scr,
                                                       float4* __restrict__ leaf_lo,
                                                       float4* __restrict__ leaf_hi,
                                                       unsigned long long* __restrict__ slot,
                                                       uint32_t* __restrict__ root, LbvhForest F) {
  __shared__ uint32_t s_ext[6], s_seg;
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  Box b = empty_box();
  const uint32_t seg = i < n ? forest_find(F, i) : 0xFFFFFFFFu;
  if (threadIdx.x < 6) s_ext[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_seg = seg;
  if (i < n) {
    b = leaf_box<PACKED>(P, i, scr);
    leaf_lo[i] = mk4(b.lo, 0.0f);
    leaf_hi[i] = mk4(b.hi, 0.0f);
    slot[i] = 0;
  }
  __syncthreads();
  const bool whole = __syncthreads_and(seg == s_seg || i >= n);
  const unsigned peers = __match_any_sync(0xFFFFFFFFu, seg);
  if (seg != 0xFFFFFFFFu) {
    uint32_t e[6];
    const bool full = peers == 0xFFFFFFFFu;
    full ? warp_extrema(b, e) : lane_extrema(b, e);
    if (!full || (threadIdx.x & 31) == 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) atomicMax(whole ? &s_ext[k] : &root[6 * (size_t)seg + k], e[k]);
    }
  }
  if (!whole) return;
  __syncthreads();
  if (threadIdx.x < 6) atomicMax(&root[6 * (size_t)s_seg + threadIdx.x], s_ext[threadIdx.x]);
}

__device__ __forceinline__ uint32_t morton_of(const Box& b, const uint32_t root[6]) {
  const f3 wl = mk3(o2f(~root[0]), o2f(~root[1]), o2f(~root[2]));
  const f3 wu = mk3(o2f(root[3]), o2f(root[4]), o2f(root[5]));
  f3 p = 0.5f * (b.lo + b.hi);
  p.x = p.x - wl.x;
  p.y = p.y - wl.y;
  p.z = p.z - wl.z;
  p.x = p.x / (wu.x - wl.x);
  p.y = p.y / (wu.y - wl.y);
  p.z = p.z / (wu.z - wl.z);
  return morton_code(p);
}

// ComputeMortons_Kernel: centre of the leaf box normalised by its segment's root box.
__global__ void k_morton(const float4* __restrict__ leaf_lo, const float4* __restrict__ leaf_hi,
                         const uint32_t* __restrict__ root_all, uint32_t n,
                         uint32_t* __restrict__ morton, uint32_t* __restrict__ index, LbvhForest F) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  morton[i] = morton_of(Box{mk3(leaf_lo[i]), mk3(leaf_hi[i])},
                        root_all + 6 * (size_t)forest_find(F, i));
  index[i] = i;
}

// Segment pass of the sort: after the Morton pass, a stable sort by segment groups each
// segment's primitives in (code, index) order, the order the segment alone would have.
__global__ void k_seg_keys(const uint32_t* __restrict__ sindex, uint32_t n, uint32_t* __restrict__ key,
                           uint32_t* __restrict__ val, LbvhForest F) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  key[i] = forest_find(F, sindex[i]);
  val[i] = i;
}
__global__ void k_seg_gather(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ m_in,
                             const uint32_t* __restrict__ i_in, uint32_t n,
                             uint32_t* __restrict__ m_out, uint32_t* __restrict__ i_out) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const uint32_t q = perm[p];
  m_out[p] = m_in[q];
  i_out[p] = i_in[q];
}

// Common prefix of sorted positions i and i + 1 of one segment plus one, on keys (code << 32 |
// segment-local object); objects of a segment compare as their global ids do.
__device__ __forceinline__ uint8_t prefix_of(uint32_t m0, uint32_t o0, uint32_t m1, uint32_t o1,
                                             uint32_t base) {
  return (uint8_t)(m0 != m1 ? 1 + __clz(m0 ^ m1) : 33 + __clz((o0 - base) ^ (o1 - base)));
}
__global__ void __launch_bounds__(kBlock) k_deltas(const uint32_t* __restrict__ smorton,
                                                   const uint32_t* __restrict__ sindex, uint32_t n,
                                                   uint8_t* __restrict__ delta,
                                                   uint32_t* __restrict__ dup, LbvhForest F) {
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  bool same = false;
  if (i < n) {
    const int4 r = forest_rec(F, forest_find(F, i));
    uint8_t d = 0;
    if (i + 1 < (uint32_t)(r.x + r.y)) {
      const uint32_t m0 = smorton[i], m1 = smorton[i + 1];
      d = prefix_of(m0, sindex[i], m1, sindex[i + 1], (uint32_t)r.x);
      same = m0 == m1;
    }
    delta[i] = d;
  }
  const unsigned eq = __ballot_sync(0xFFFFFFFFu, same);
  if (eq && (threadIdx.x & 31) == 0) atomicAdd(dup, (uint32_t)__popc(eq));
}

// ConstructLeafNodes_Kernel, ConstructInternalNodes64Bits_Kernel, the escape tables and the boxes
// in one bottom-up walk (tree_up).
template <bool SMALL>
__global__ void __launch_bounds__(kTreeBlock) k_tree(const uint32_t* __restrict__ sindex,
                                                     const float4* __restrict__ leaf_lo,
                                                     const float4* __restrict__ leaf_hi, uint32_t n,
                                                     TreeMem t, uint32_t* err) {
  extern __shared__ float4 smem[];
  const uint32_t i = blockIdx.x * kTreeBlock + threadIdx.x;
  f3 bl = mk3(0, 0, 0), bu = bl;
  uint32_t obj = 0;
  if (i < n) {
    obj = sindex[i];
    bl = mk3(leaf_lo[obj]);
    bu = mk3(leaf_hi[obj]);
    obj -= (uint32_t)forest_rec(t.F, forest_find(t.F, i)).x;
  }
  if (SMALL)
    small_tree<true>(t, *reinterpret_cast<SmallShared*>(smem), i, i < n, obj, bl, bu, err);
  else
    tree_up<true>(t, *reinterpret_cast<TreeShared*>(smem), i, i < n, obj, bl, bu, err);
}

// ---- small single trees -------------------------------------------------------------------------
// Everything ahead of k_tree in one launch of one cluster: leaf boxes, root box, Morton codes, the
// stable radix sort (four 8-bit digits) and the neighbors' prefixes.  As 17 launches of a few blocks
// it was bound by the latency of launches and single-block scans (13,776 triangles: 78 us of kernels,
// now 28; with k_tree a whole build 129 -> 50 us); the phases here are a cluster barrier apart
// (0.2 us) and the digit counts cross the blocks through distributed shared memory.
// A warp owns R x 32 consecutive primitives (sorted positions in later passes), so ranking them round
// by round with one running count per warp and digit is stable; the blocks share the warps evenly.
// A lane finds its equals by eight ballots (match.any took 3,000 cycles a pass with 64 groups on an
// SM).
constexpr int kSortCtas = 8;  // the portable cluster size
constexpr int kSortThreads = 1024;
constexpr int kSortWarps = kSortThreads / 32;
static_assert(kSmallMax <= 2 * kSortCtas * kSortThreads, "two primitives a thread");

struct SortShared {
  uint32_t cnt[kSortWarps][256];  // per warp: digit counts, then offsets
  uint32_t total[kSortCtas][256], base[256], part[4][256], warp[8];  // total: every block's
  uint32_t ext[6], exts[kSortCtas][6], root[6];
};

template <bool PACKED, int R>
__global__ void __cluster_dims__(kSortCtas, 1, 1) __launch_bounds__(kSortThreads)
    k_small_sort(Prims P, uint32_t n, float scr, float4* __restrict__ leaf_lo,
                 float4* __restrict__ leaf_hi, uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp,
                 uint32_t* vals_tmp, uint8_t* __restrict__ delta, uint32_t* __restrict__ dup,
                 TreeMem t) {
  __shared__ SortShared sh;
  uint32_t(*s_cnt)[256] = sh.cnt;
  uint32_t(*s_part)[256] = sh.part;
  uint32_t(*s_total)[256] = sh.total;
  uint32_t *s_base = sh.base, *s_warp = sh.warp, *s_ext = sh.ext, *s_root = sh.root;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, cta = blockIdx.x;
  // warps with primitives per block
  const uint32_t warps = ((n + 32 * R - 1) / (32 * R) + kSortCtas - 1) / kSortCtas;
  const uint32_t first = warp < warps ? (cta * warps + warp) * (R * 32) + lane : n + lane;
  if (tid < 6) s_ext[tid] = 0;
  if (cta == 0 && tid == 0) *dup = *t.ticket = 0;
  cluster_sync();  // every block runs before the first write into another's memory
  Box box[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = first + 32 * r;
    box[r] = empty_box();
    if (i < n) {
      box[r] = leaf_box<PACKED>(P, i, scr);
      leaf_lo[i] = mk4(box[r].lo, 0.0f);
      leaf_hi[i] = mk4(box[r].hi, 0.0f);
      t.slot[i] = 0;
    }
    if (i - lane >= n) continue;  // uniform in the warp
    const bool full = i - lane + 32 <= n;
    uint32_t e[6];
    full ? warp_extrema(box[r], e) : lane_extrema(box[r], e);
    if (full ? lane == 0 : i < n) {
#pragma unroll
      for (int k = 0; k < 6; ++k) atomicMax(&s_ext[k], e[k]);
    }
  }
  __syncthreads();
  if (tid < 6 * kSortCtas) st_cluster(&sh.exts[cta][tid % 6], tid / 6, s_ext[tid % 6]);
  cluster_sync();
  if (tid < 6) {
    uint32_t m = 0;
#pragma unroll
    for (int c = 0; c < kSortCtas; ++c) m = max(m, sh.exts[c][tid]);
    s_root[tid] = m;
  }
  __syncthreads();
  uint32_t key[R], val[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = first + 32 * r;
    key[r] = i < n ? morton_of(box[r], s_root) : 0u;
    val[r] = i;
  }
#pragma unroll 1
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 8 * pass;
    uint32_t* ko = pass & 1 ? keys : keys_tmp;
    uint32_t* vo = pass & 1 ? vals : vals_tmp;
    if (pass) {
      const uint32_t* ki = pass & 1 ? keys_tmp : keys;
      const uint32_t* vi = pass & 1 ? vals_tmp : vals;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t i = first + 32 * r;
        key[r] = i < n ? __ldcg(&ki[i]) : 0u;
        val[r] = i < n ? __ldcg(&vi[i]) : 0u;
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) s_cnt[warp][lane + 32 * k] = 0;
    __syncwarp();
    uint32_t rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool has = first + 32 * r < n;
      const uint32_t d = (key[r] >> shift) & 0xFFu;
      unsigned peers = __ballot_sync(0xFFFFFFFFu, has);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const unsigned one = __ballot_sync(0xFFFFFFFFu, (d >> b) & 1u);
        peers &= (d >> b) & 1u ? one : ~one;
      }
      const uint32_t before = has ? s_cnt[warp][d] : 0u;
      rank[r] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (has && (int)lane == __ffs(peers) - 1) s_cnt[warp][d] = before + (uint32_t)__popc(peers);
      __syncwarp();
    }
    __syncthreads();
    {  // offsets of the warps inside the block: a quarter of the warps per thread, then the quarters
      const uint32_t d = tid & 255u, q = tid >> 8;
      uint32_t run = 0;
#pragma unroll
      for (int w = 0; w < kSortWarps / 4; ++w) {
        const uint32_t c = s_cnt[q * (kSortWarps / 4) + w][d];
        s_cnt[q * (kSortWarps / 4) + w][d] = run;
        run += c;
      }
      s_part[q][d] = run;
      __syncthreads();
      // every block gets every block's totals (two blocks per quarter), so that the sums after the
      // barrier read its own memory
      const uint32_t sum = s_part[0][d] + s_part[1][d] + s_part[2][d] + s_part[3][d];
      st_cluster(&s_total[cta][d], 2 * q, sum);
      st_cluster(&s_total[cta][d], 2 * q + 1, sum);
    }
    cluster_sync();
    if (tid < 256) {  // the digit's first position: smaller digits, then earlier blocks
      uint32_t all = 0, mine = 0;
#pragma unroll
      for (uint32_t c = 0; c < kSortCtas; ++c) {
        const uint32_t v = s_total[c][tid];
        mine += c < cta ? v : 0u;
        all += v;
      }
      uint32_t x = all;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= (uint32_t)off) x += y;
      }
      if (lane == 31) s_warp[warp] = x;
      s_base[tid] = x - all + mine;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t before = 0;
      for (uint32_t w = 0; w < warp; ++w) before += s_warp[w];
      s_base[tid] += before;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (first + 32 * r >= n) continue;
      const uint32_t d = (key[r] >> shift) & 0xFFu, q = warp / (kSortWarps / 4);
      uint32_t dst = s_base[d] + s_cnt[warp][d] + rank[r];
      for (uint32_t k = 0; k < q; ++k) dst += s_part[k][d];
      __stcg(&ko[dst], key[r]);
      __stcg(&vo[dst], val[r]);
    }
    cluster_sync();  // the pass's output is visible, and every block has read the totals
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t i = first + 32 * r;
    bool same = false;
    if (i < n) {
      uint8_t d = 0;
      if (i + 1 < n) {
        const uint32_t m0 = __ldcg(&keys[i]), m1 = __ldcg(&keys[i + 1]);
        d = prefix_of(m0, __ldcg(&vals[i]), m1, __ldcg(&vals[i + 1]), 0);
        same = m0 == m1;
      }
      delta[i] = d;
    }
    const unsigned eq = __ballot_sync(0xFFFFFFFFu, same);
    if (eq && lane == 0) atomicAdd(dup, (uint32_t)__popc(eq));
  }
}

__global__ void k_prims_mesh(const float4* __restrict__ x, const float4* __restrict__ nrm,
                             const int4* __restrict__ tri, uint32_t nf, float tol,
                             float4* __restrict__ v, float4* __restrict__ pred) {
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  const int4 t = tri[f];
  const int id[3] = {t.x, t.y, t.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f3 q = mk3(x[id[k]]) + tol * mk3(nrm[id[k]]);
    v[3 * f + k] = mk4(q, 0.0f);
    pred[3 * f + k] = mk4(q, 0.0f);
  }
}

// UpdateObjects_Kernel with ccd = true (BVH.cu:382-418): v from x0, pred from x.
__global__ void k_prims_ccd(const float4* __restrict__ x, const float4* __restrict__ x0,
                            const float4* __restrict__ nrm, const int4* __restrict__ tri,
                            uint32_t nf, float tol, float4* __restrict__ v,
                            float4* __restrict__ pred) {
  const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  const int4 t = tri[f];
  const int id[3] = {t.x, t.y, t.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const f3 n = mk3(nrm[id[k]]);
    v[3 * f + k] = mk4(mk3(x0[id[k]]) + tol * n, 0.0f);
    pred[3 * f + k] = mk4(mk3(x[id[k]]) + tol * n, 0.0f);
  }
}

// RefitExternalNodeMidstep_Kernel: the leaf at node k grows by its triangle's midstep vertices moved
// along their normals, which become its primitive.
struct GrowMidstep {
  const float4 *x1, *n1;
  const int4* tri;
  float tol;
  float4* pred;
  __device__ __forceinline__ void operator()(uint32_t prim, f3& l, f3& h) const {
    const int4 v = tri[prim];
    const int id[3] = {v.x, v.y, v.z};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const f3 q = mk3(x1[id[c]]) + tol * mk3(n1[id[c]]);
      pred[3 * (size_t)prim + c] = mk4(q, 0.0f);
      l = mk3(tmin(l.x, q.x), tmin(l.y, q.y), tmin(l.z, q.z));
      h = mk3(tmax(h.x, q.x), tmax(h.y, q.y), tmax(h.z, q.z));
    }
  }
};
// RefitExternalNode_Kernel(predicted), 9 floats per primitive.
struct GrowPred {
  const float* p9;
  __device__ __forceinline__ void operator()(uint32_t prim, f3& l, f3& h) const {
    const float* q = p9 + 9 * (size_t)prim;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      l = mk3(tmin(l.x, q[3 * c]), tmin(l.y, q[3 * c + 1]), tmin(l.z, q[3 * c + 2]));
      h = mk3(tmax(h.x, q[3 * c]), tmax(h.y, q[3 * c + 1]), tmax(h.z, q[3 * c + 2]));
    }
  }
};

}  // namespace

namespace {

// One query: a point (KIND 0), a segment (1) or a box (2).
template <int KIND>
struct TreeQuery {
  f3 a, c;
  __device__ __forceinline__ TreeQuery(const float* __restrict__ q, uint32_t i) {
    const float* v = q + (KIND == 0 ? 3 : 6) * (size_t)i;
    a = mk3(v[0], v[1], v[2]);
    c = KIND == 0 ? a : mk3(v[3], v[4], v[5]);
  }
  __device__ __forceinline__ bool operator()(float4 l, float4 h) const {
    return KIND == 0 ? overlap_point(l, h, a)
           : KIND == 1 ? overlap_segment(l, h, a, c)
                       : overlap_box(l, h, a, c);
  }
};

// A lane per query.
template <int KIND>
__global__ void k_query(LbvhView b, const float* __restrict__ q, uint32_t nq,
                        uint32_t* __restrict__ counts, uint32_t* __restrict__ cands, uint32_t* err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const TreeQuery<KIND> test(q, i);
  uint32_t* out = cands + (size_t)i * kMaxCandidates;
  uint32_t found = 0;
  lbvh_traverse(b, test, [&](uint32_t obj) { out[found++] = obj; }, err);
  counts[i] = found;
}

// G lanes per query (8 or 32).  What follows in the walk is a stack in shared memory, the next on top:
// nodes to be tested and, behind one of those, leaves known to overlap.  A round takes up to G
// entries, one a lane, and puts in the place of each what follows from it: an overlapping leaf
// itself, below an overlapping inner node its left child, and after a left child its sibling.  The
// leaves ahead of the first node left are the walk's next candidates and leave the stack; at
// kMaxCandidates the walk ends.  A full round leaves kReserve entries free; without room for one,
// entries are taken singly, which deepens the stack by at most one per level of the tree (64-bit
// keys: 65 levels).
constexpr uint32_t kQueryBlock = 128, kReserve = 72;
// An entry: node, or object of a leaf, with its kind in the two top bits.
constexpr uint32_t kLeft = 1u << 30, kDone = 2u << 30, kEntryIds = kLeft;
template <int KIND, int G>
__global__ void __launch_bounds__(kQueryBlock) k_query_group(
    LbvhView b, const float* __restrict__ q, uint32_t nq, uint32_t* __restrict__ counts,
    uint32_t* __restrict__ cands, uint32_t* err) {
  constexpr unsigned kAll = 0xFFFFFFFFu, kGroup = G == 32 ? kAll : (1u << G % 32) - 1u;
  constexpr uint32_t kStack = G == 32 ? 640 : 176;
  static_assert(kReserve >= 65 + 2, "singly taken entries fit");
  __shared__ uint32_t stacks[kQueryBlock / G][kStack];
  const uint32_t lane = threadIdx.x % G, shift = (threadIdx.x & 31u) - lane;
  const unsigned below = (1u << lane) - 1u;
  const uint32_t i = blockIdx.x * (kQueryBlock / G) + threadIdx.x / G;
  const bool valid = i < nq;
  const TreeQuery<KIND> test(q, valid ? i : 0u);
  uint32_t* out = cands + (size_t)i * kMaxCandidates;
  uint32_t* stack = stacks[threadIdx.x / G];
  auto ballot = [&](bool p) { return __ballot_sync(kAll, p) >> shift & kGroup; };
  if (lane == 0) stack[0] = 0u;  // the root
  uint32_t count = valid && b.n ? 1u : 0u, found = 0;
  __syncwarp();
  for (uint32_t round = 0; __any_sync(kAll, count != 0); ++round) {
    if (round > 2 * b.n + 2 || __any_sync(kAll, count > kStack - 2)) {
      if (count != 0 && lane == 0) raise_error(err, kErrTraversal);
      break;
    }
    const uint32_t room = kStack - kReserve > count ? kStack - kReserve - count : 1u;
    const uint32_t n = min(min(count, (uint32_t)G), room);
    const uint32_t e = lane < n ? stack[count - 1 - lane] : 0u;
    count -= n;
    __syncwarp();
    uint32_t first = 0, second = 0, made = 0;  // what follows from the entry, in order
    if (lane < n) {
      if (e & kDone) {
        first = e;
        made = 1;
      } else {
        const uint32_t node = e & (kEntryIds - 1);
        const float4 l = b.lo[node], h = b.hi[node];
        if (test(l, h)) {
          first = (uint32_t)__float_as_int(l.w) | (node >= b.n - 1 ? kDone : kLeft);
          made = 1;
        }
        if (e & kLeft) {
          const uint32_t sibling = (uint32_t)__float_as_int(h.w);
          if (made++) second = sibling;
          else first = sibling;
        }
      }
    }
    const bool leaf = first & kDone;
    const unsigned nodes = ballot(made > (leaf ? 1u : 0u));  // lanes with nodes left
    // candidates: the leaves up to the first such lane's
    const bool take = leaf && (nodes & below) == 0;
    const unsigned taken = ballot(take);
    const uint32_t at = found + __popc(taken & below);
    if (take && at < kMaxCandidates) out[at] = first & (kEntryIds - 1);
    found += __popc(taken);
    const uint32_t keep = made - (take ? 1u : 0u);
    const unsigned m1 = ballot(keep & 1u), m2 = ballot(keep & 2u);
    uint32_t top = count + __popc(m1) + 2 * __popc(m2);  // one above the whole round's
    count = found < kMaxCandidates ? top : 0u;
    top -= __popc(m1 & below) + 2 * __popc(m2 & below);  // one above this lane's
    if (keep > 0) stack[top - 1] = take ? second : first;
    if (keep > 1) stack[top - 2] = second;
    __syncwarp();
  }
  if (valid && lane == 0) counts[i] = min(found, kMaxCandidates);
}

}  // namespace

cudaError_t Lbvh::set_segments(const std::vector<uint32_t>& counts, cudaStream_t s) {
  h_seg.clear();
  if (counts.size() <= 1) return cudaSuccess;
  uint32_t pb = 0, nb = 0, ib = 0;
  for (uint32_t c : counts) {
    h_seg.push_back(make_int4((int)pb, (int)c, (int)nb, (int)ib));
    pb += c;
    nb += c ? 2 * c - 1 : 0;
    ib += c ? c - 1 : 0;
  }
  cudaError_t e = seg.reserve(h_seg.size());
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(seg.p, h_seg.data(), sizeof(int4) * h_seg.size(), cudaMemcpyHostToDevice, s);
  return e;
}

cudaError_t Lbvh::reserve(uint32_t np, bool packed) {
  const size_t nn = np ? 2 * (size_t)np - 1 : 1;
  cudaError_t e = cudaSuccess;
  if (nseg() > 1) {
    if (e == cudaSuccess) e = skey.reserve(np);
    if (e == cudaSuccess) e = sval.reserve(np);
  }
  if (!packed) {
    if (e == cudaSuccess) e = v.reserve(3 * (size_t)np);
    if (e == cudaSuccess) e = pred.reserve(3 * (size_t)np);
  }
  if (e == cudaSuccess) e = leaf_lo.reserve(np);
  if (e == cudaSuccess) e = leaf_hi.reserve(np);
  if (e == cudaSuccess) e = lo.reserve(nn);
  if (e == cudaSuccess) e = hi.reserve(nn);
  if (e == cudaSuccess) e = node.reserve(nn);
  if (e == cudaSuccess) e = morton.reserve(np);
  if (e == cudaSuccess) e = index.reserve(np);
  if (e == cudaSuccess) e = slot.reserve(np);
  if (e == cudaSuccess) e = rest.reserve(rest_words(np));
  if (e == cudaSuccess) e = rest_count.reserve(kSmallBlocks + 1);
  if (e == cudaSuccess) e = delta.reserve(np);
  if (e == cudaSuccess) e = iesc.reserve(np);
  if (e == cudaSuccess) e = eesc.reserve(np);
  if (e == cudaSuccess) e = root.reserve(6 * (size_t)nseg());
  if (e == cudaSuccess) e = dup.reserve(1);
  if (e == cudaSuccess) e = sorter.reserve(np);
  return e;
}

template <bool PACKED>
static void launch_small_sort(const Lbvh& b, const Prims& P, float scr, cudaStream_t s) {
  auto k = b.n <= kSmallMax / 2 ? k_small_sort<PACKED, 1> : k_small_sort<PACKED, 2>;
  k<<<kSortCtas, kSortThreads, 0, s>>>(P, b.n, scr, b.leaf_lo.p, b.leaf_hi.p, b.morton.p,
                                       b.index.p, b.sorter.keys_tmp.p, b.sorter.vals_tmp.p,
                                       b.delta.p, b.dup.p, tree_mem(b));
}

void Lbvh::construct(float scr, cudaStream_t s, uint32_t* d_err, const float* v9,
                     const float* p9) {
  active = n > 0;
  if (n == 0) return;
  const LbvhForest F = forest();
  const uint32_t S = nseg();
  nodes = 0;
  internal = 0;
  if (S == 1) {
    nodes = 2 * n - 1;
    internal = n - 1;
  } else {
    for (const int4& r : h_seg) {
      nodes += r.y ? 2 * (uint32_t)r.y - 1 : 0;
      internal += r.y ? (uint32_t)r.y - 1 : 0;
    }
  }
  const Prims P{v.p, pred.p, v9, p9};
  if (small()) {
    v9 ? launch_small_sort<true>(*this, P, scr, s) : launch_small_sort<false>(*this, P, scr, s);
    sorted_morton = morton.p;
    sorted_index = index.p;
  } else {
    uint32_t* rootu = reinterpret_cast<uint32_t*>(root.p);
    cudaMemsetAsync(rootu, 0, sizeof(uint32_t) * 6 * S, s);
    cudaMemsetAsync(dup.p, 0, sizeof(uint32_t), s);
    auto boxes = v9 ? k_leaf_boxes<true> : k_leaf_boxes<false>;
    boxes<<<grid_for(n), kBlock, 0, s>>>(P, n, scr, leaf_lo.p, leaf_hi.p, slot.p, rootu, F);
    k_morton<<<grid_for(n), kBlock, 0, s>>>(leaf_lo.p, leaf_hi.p, rootu, n, morton.p, index.p, F);
    // Morton codes have 30 bits: four 8-bit passes leave the result in (morton, index)
    sorter.sort(morton.p, index.p, n, 30, s, &sorted_morton, &sorted_index);
    if (S > 1) {
      int bits = 0;
      while ((1u << bits) < S) ++bits;
      k_seg_keys<<<grid_for(n), kBlock, 0, s>>>(sorted_index, n, skey.p, sval.p, F);
      uint32_t *k2 = nullptr, *perm = nullptr;
      sorter.sort(skey.p, sval.p, n, bits, s, &k2, &perm);
      // gather into whichever key / value pair the segment pass's result does not occupy
      const bool in_own = perm == sval.p;
      uint32_t* m_out = in_own ? sorter.keys_tmp.p : skey.p;
      uint32_t* i_out = in_own ? sorter.vals_tmp.p : sval.p;
      k_seg_gather<<<grid_for(n), kBlock, 0, s>>>(perm, sorted_morton, sorted_index, n, m_out, i_out);
      sorted_morton = m_out;
      sorted_index = i_out;
    }
    k_deltas<<<grid_for(n), kBlock, 0, s>>>(sorted_morton, sorted_index, n, delta.p, dup.p, F);
  }
  auto tree = small() ? k_tree<true> : k_tree<false>;
  const size_t smem = small() ? sizeof(SmallShared) : sizeof(TreeShared);
  if (raise_smem((const void*)tree, smem) != cudaSuccess) return;
  tree<<<grid_for(n, kTreeBlock), kTreeBlock, smem, s>>>(sorted_index, leaf_lo.p, leaf_hi.p, n,
                                                         tree_mem(*this), d_err);
}

static_assert(kSmallMax == Lbvh::kSmallBlocks * kTreeBlock &&
                  sizeof(TreeRest) == 16 * Lbvh::kRestWords && kRestPerBlock == Lbvh::kRestPerBlock,
              "small trees: blocks and lists as reserved");
bool Lbvh::small() const { return nseg() == 1 && n <= kSmallMax; }

uint32_t Lbvh::build_launches() const {
  if (small()) return 2;
  const uint32_t pass = RadixSort::hist_entries(n) <= RadixSort::kSingleBlockScan ? 3 : 5;
  uint32_t bits = 0;
  while ((1u << bits) < nseg()) ++bits;
  return 4 + pass * (4 + (bits + 7) / 8) + (nseg() > 1 ? 2 : 0);
}

void Lbvh::refit_from_pred(const float* p9, cudaStream_t s, uint32_t* d_err) {
  if (!active) return;
  launch_refit(*this, GrowPred{p9}, s, d_err);
}

void Lbvh::release() {
  v.release(); pred.release(); leaf_lo.release(); leaf_hi.release(); lo.release(); hi.release();
  node.release(); morton.release(); index.release(); slot.release(); delta.release();
  rest.release(); rest_count.release();
  iesc.release(); eesc.release(); root.release(); dup.release(); skey.release(); sval.release();
  seg.release();
  sorter.keys_tmp.release(); sorter.vals_tmp.release(); sorter.hist.release(); sorter.sums.release();
}

void launch_prims_from_mesh(Lbvh& b, const float4* x, const float4* nrm, const int4* tri,
                            uint32_t nf, float tol, cudaStream_t s) {
  if (nf == 0) return;
  k_prims_mesh<<<grid_for(nf), kBlock, 0, s>>>(x, nrm, tri, nf, tol, b.v.p, b.pred.p);
}

void launch_prims_ccd(Lbvh& b, const float4* x, const float4* x0, const float4* nrm,
                      const int4* tri, uint32_t nf, float tol, cudaStream_t s) {
  if (nf == 0) return;
  k_prims_ccd<<<grid_for(nf), kBlock, 0, s>>>(x, x0, nrm, tri, nf, tol, b.v.p, b.pred.p);
}

void launch_refit_midstep(Lbvh& b, const float4* x1, const float4* n1, const int4* tri, float tol,
                          cudaStream_t s, uint32_t* d_err) {
  if (!b.active) return;
  launch_refit(b, GrowMidstep{x1, n1, tri, tol, b.pred.p}, s, d_err);
}

// Lanes per query.  Few queries are bound by the chain of a walk (2.09 M triangles, boxes of about 29
// leaves, 1,000 queries: one lane 73 us, 8 lanes 29, 32 lanes 21; of 256 and more leaves 240, 77 and
// 35), many by issue: 6,000 queries that end near the root take 21, 20 and 28 us, 20,000 of them 24, 33
// and 70 (but 20,000 of 29 leaves 112, 55 and 104).
constexpr uint32_t kWarpQueries = 3000, kGroupQueries = 20000;
template <int KIND, int G>
static void launch_query_group(const Lbvh& b, const float* q, uint32_t nq, uint32_t* counts,
                               uint32_t* cands, cudaStream_t s, uint32_t* err) {
  k_query_group<KIND, G><<<grid_for(nq, kQueryBlock / G), kQueryBlock, 0, s>>>(b.view(), q, nq, counts,
                                                                             cands, err);
}
template <int KIND>
static void launch_query(const Lbvh& b, const float* q, uint32_t nq, uint32_t* counts,
                         uint32_t* cands, cudaStream_t s, uint32_t* err) {
  if (nq <= kWarpQueries)
    launch_query_group<KIND, 32>(b, q, nq, counts, cands, s, err);
  else if (nq <= kGroupQueries)
    launch_query_group<KIND, 8>(b, q, nq, counts, cands, s, err);
  else
    k_query<KIND><<<grid_for(nq), kBlock, 0, s>>>(b.view(), q, nq, counts, cands, err);
}
void launch_lbvh_query(const Lbvh& b, int kind, const float* d_q, uint32_t nq, uint32_t* d_counts,
                       uint32_t* d_cands, cudaStream_t s, uint32_t* d_err) {
  if (nq == 0 || !b.active) return;
  if (kind == 0) launch_query<0>(b, d_q, nq, d_counts, d_cands, s, d_err);
  else if (kind == 1) launch_query<1>(b, d_q, nq, d_counts, d_cands, s, d_err);
  else launch_query<2>(b, d_q, nq, d_counts, d_cands, s, d_err);
}

}  // namespace xrt
