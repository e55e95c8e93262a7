// GPU BVH construction.
//
// Two builders share the same front end (primitive bounds, centroid bounds,
// 30-bit Morton codes, a stable LSD radix sort written here):
//
//  * build_reference: the reference's Morton build
//    (rendering/taichi/bvh_builder.py:412-478).  Splitting the Morton order
//    at the count median makes the topology depend only on the primitive
//    count, so it is laid out level by level on the device and node bounds
//    are reduced bottom-up.  Node numbering is the reference's DFS pre-order
//    and the output equals GPUBVHBuilder's `nodes` / `ordered_tris` bit for
//    bit.
//  * build_lbvh: Karras' parallel LBVH ("Maximizing parallelism in the
//    construction of BVHs, octrees, and k-d trees", HPG 2012) over the same
//    codes, a bottom-up pass computing bounds and SAH costs, and an SAH
//    collapse of subtrees into leaves of up to `max_leaf` primitives, laid
//    out in Morton order (the root first), and a 4-wide copy.
//
// Both emit the traversal layout described in rx_internal.cuh.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <vector>

#include "rx_internal.cuh"
#include "rx_runtime.h"

namespace rx {

// L2-coherent load of a float3 written by another thread before a fence.
__device__ __forceinline__ float3 ldcg3(const float3* p) {
  const float* f = reinterpret_cast<const float*>(p);
  return f3(__ldcg(f), __ldcg(f + 1), __ldcg(f + 2));
}

// ----------------------------------------------------------------------------
// front end
// ----------------------------------------------------------------------------
// Primitive i < n_tris is a triangle, else analytic object i - n_tris
// (sphere or cube: obj_a = (centre, kind), obj_b = (radius, 0, 0, 0) or
// (half extents, 0)).  Triangle bounds are padded by 1e-4 and centroids are
// (v0 + v1 + v2) / 3 with the reference's float32 order
// (bvh_builder.py:363-368); an object's centroid is its centre.  box_centre
// != 0 (the LBVH): a triangle's key point is the centre of its bounding box
// instead, which on the benchmark scene's rays gives a tree with 2-4 % fewer
// node visits than the centroid.
__global__ void k_prim_bounds(int n_tris, const float* __restrict__ v0, const float* __restrict__ v1,
                              const float* __restrict__ v2, int n_obj, const float4* __restrict__ obj_a,
                              const float4* __restrict__ obj_b, int box_centre, float3* __restrict__ bmin,
                              float3* __restrict__ bmax, float3* __restrict__ cen) {
  int n = n_tris + n_obj;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < n_tris) {
      float3 a = f3(v0[3 * i], v0[3 * i + 1], v0[3 * i + 2]);
      float3 b = f3(v1[3 * i], v1[3 * i + 1], v1[3 * i + 2]);
      float3 c = f3(v2[3 * i], v2[3 * i + 1], v2[3 * i + 2]);
      const float3 lo = vmin(a, vmin(b, c)), hi = vmax(a, vmax(b, c));
      bmin[i] = lo - f3(1e-4f, 1e-4f, 1e-4f);
      bmax[i] = hi + f3(1e-4f, 1e-4f, 1e-4f);
      cen[i] = box_centre ? f3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z))
                          : f3(((a.x + b.x) + c.x) / 3.0f, ((a.y + b.y) + c.y) / 3.0f, ((a.z + b.z) + c.z) / 3.0f);
    } else {
      float4 a = obj_a[i - n_tris], b = obj_b[i - n_tris];
      float3 e = __float_as_int(a.w) == PRIM_SPHERE ? f3(b.x, b.x, b.x) : f3(b.x, b.y, b.z);
      bmin[i] = f3(a.x - e.x, a.y - e.y, a.z - e.z) - f3(1e-4f, 1e-4f, 1e-4f);
      bmax[i] = f3(a.x + e.x, a.y + e.y, a.z + e.z) + f3(1e-4f, 1e-4f, 1e-4f);
      cen[i] = f3(a.x, a.y, a.z);
    }
  }
}

// Two-stage exact min/max reduction of the centroids.
__global__ void k_reduce_bounds(int n, const float3* __restrict__ p, float3* __restrict__ part_min,
                                float3* __restrict__ part_max) {
  chain_wait(p, part_min, part_max);
  chain_go();
  __shared__ float smin[3][256], smax[3][256];
  float3 lo = f3(INFINITY, INFINITY, INFINITY), hi = f3(-INFINITY, -INFINITY, -INFINITY);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    lo = vmin(lo, p[i]);
    hi = vmax(hi, p[i]);
  }
  int t = threadIdx.x;
  smin[0][t] = lo.x; smin[1][t] = lo.y; smin[2][t] = lo.z;
  smax[0][t] = hi.x; smax[1][t] = hi.y; smax[2][t] = hi.z;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (t < s) {
      for (int k = 0; k < 3; ++k) {
        smin[k][t] = fminf(smin[k][t], smin[k][t + s]);
        smax[k][t] = fmaxf(smax[k][t], smax[k][t + s]);
      }
    }
    __syncthreads();
  }
  if (t == 0) {
    part_min[blockIdx.x] = f3(smin[0][0], smin[1][0], smin[2][0]);
    part_max[blockIdx.x] = f3(smax[0][0], smax[1][0], smax[2][0]);
  }
}

// Second stage: one block of kBoundsThreads reduces the parts' boxes --
// the minimum over mins[] and the maximum over maxs[] -- into out[0],
// out[1].  Min and max are exact, so the result does not depend on the
// order.
constexpr int kBoundsThreads = 1024;
__global__ void __launch_bounds__(kBoundsThreads) k_bounds_final(int parts, const float3* __restrict__ mins,
                                                                 const float3* __restrict__ maxs,
                                                                 float3* __restrict__ out) {
  chain_wait(mins, maxs, out);
  chain_go();
  __shared__ float3 slo[kBoundsThreads], shi[kBoundsThreads];
  float3 lo = f3(INFINITY, INFINITY, INFINITY), hi = f3(-INFINITY, -INFINITY, -INFINITY);
  for (int k = threadIdx.x; k < parts; k += kBoundsThreads) {
    lo = vmin(lo, mins[k]);
    hi = vmax(hi, maxs[k]);
  }
  const int t = threadIdx.x;
  slo[t] = lo;
  shi[t] = hi;
  __syncthreads();
  for (int s = kBoundsThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
      slo[t] = vmin(slo[t], slo[t + s]);
      shi[t] = vmax(shi[t], shi[t + s]);
    }
    __syncthreads();
  }
  if (t == 0) {
    out[0] = slo[0];
    out[1] = shi[0];
  }
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  v &= 0x000003ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// 30-bit Morton code of each centroid, normalised over the centroid bounds
// exactly as bvh_builder.py:416-443 (extent <= 1e-12 replaced by 1).
// cubic != 0 (the LBVH): all three axes are normalised by the largest
// extent, so the grid's cells are cubes rather than the bounds' shape; on the
// benchmark scene's rays that tree visits 1.5-5 % fewer nodes.
// `bounds`: the centroid bounds (k_bounds_final).
__global__ void k_morton(int n, const float3* __restrict__ cen, const float3* __restrict__ bounds, int cubic,
                         uint32_t* __restrict__ codes, int* __restrict__ idx) {
  chain_wait(cen, bounds, codes, idx);
  chain_go();
  __shared__ float3 s_lo, s_ext;
  if (threadIdx.x == 0) {
    const float3 lo = bounds[0], hi = bounds[1];
    float3 e = hi - lo;
    if (e.x <= 1e-12f) e.x = 1.0f;
    if (e.y <= 1e-12f) e.y = 1.0f;
    if (e.z <= 1e-12f) e.z = 1.0f;
    if (cubic) {
      const float m = fmaxf(e.x, fmaxf(e.y, e.z));
      e = f3(m, m, m);
    }
    s_lo = lo;
    s_ext = e;
  }
  __syncthreads();
  float3 lo = s_lo, ext = s_ext;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float3 c = cen[i];
    float x = fminf(fmaxf((c.x - lo.x) / ext.x, 0.0f), 1.0f);
    float y = fminf(fmaxf((c.y - lo.y) / ext.y, 0.0f), 1.0f);
    float z = fminf(fmaxf((c.z - lo.z) / ext.z, 0.0f), 1.0f);
    uint32_t qx = (uint32_t)(x * 1023.0f), qy = (uint32_t)(y * 1023.0f), qz = (uint32_t)(z * 1023.0f);
    codes[i] = (expand10(qx) << 2) | (expand10(qy) << 1) | expand10(qz);
    idx[i] = i;
  }
}

// ----------------------------------------------------------------------------
// stable LSD radix sort, 8-bit digits, (key, value) pairs
// tile = 8 warps x CHUNKS x 32 keys per block: 1,024 keys (CHUNKS 4) up to
// 2^20 keys, which fills the device at 150 k keys, else 4,096 with a quarter
// of the histogram.  Four passes over 327 k keys 200 -> 82 us: scatter 22 ->
// 11 us with smaller tiles and all loads ahead of the ranking, the counters'
// scan 21 -> 4 with a block per digit.
// ----------------------------------------------------------------------------
constexpr int kSortWarps = 8;
__host__ __device__ constexpr int sort_tile(int chunks) { return kSortWarps * chunks * 32; }

__global__ void k_sort_hist(int n, const uint32_t* __restrict__ keys, int shift, int tile, uint32_t* __restrict__ hist,
                            int nblocks) {
  chain_wait(keys, hist);
  chain_go();
  __shared__ uint32_t h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  int base = blockIdx.x * tile;
  int end = min(base + tile, n);
  for (int i = base + threadIdx.x; i < end; i += blockDim.x) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[d * nblocks + blockIdx.x] = h[d];
}

// Exclusive sums of 256 values, one per thread of a 256-thread block;
// *total: their sum.  Ends with a barrier.
__device__ __forceinline__ uint32_t block_exclusive_256(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const uint32_t y = warp_sums[w];
    if (w < wid) before += y;
    all += y;
  }
  *total = all;
  __syncthreads();
  return before + x - v;
}

// Exclusive sums along each digit's row of hist[256][nblocks] and the rows'
// totals, one block per digit.  (One block over all 256 x nblocks counters
// took 21 us per pass at 80 blocks; a row each takes 3.)
__global__ void __launch_bounds__(256) k_sort_rows(uint32_t* __restrict__ hist, uint32_t* __restrict__ totals,
                                                   int nblocks) {
  chain_wait(hist, totals);
  chain_go();
  __shared__ uint32_t warp_sums[8];
  uint32_t* row = hist + (size_t)blockIdx.x * nblocks;
  uint32_t carry = 0;
  for (int base = 0; base < nblocks; base += 256) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < nblocks ? row[i] : 0u;
    uint32_t total;
    const uint32_t e = block_exclusive_256(v, warp_sums, &total);
    if (i < nblocks) row[i] = carry + e;
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template <int CHUNKS>
__global__ void __launch_bounds__(kSortWarps * 32)
    k_sort_scatter(int n, const uint32_t* __restrict__ keys_in, const int* __restrict__ vals_in,
                   uint32_t* __restrict__ keys_out, int* __restrict__ vals_out, int shift,
                   const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals, int nblocks) {
  chain_wait(keys_in, vals_in, keys_out, vals_out, hist, totals);
  chain_go();
  static_assert(kSortWarps * 32 == 256, "one thread per digit");
  __shared__ uint32_t wcount[kSortWarps][256];
  __shared__ uint32_t warp_sums[8];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int wbase = blockIdx.x * sort_tile(CHUNKS) + w * CHUNKS * 32 + lane;
  // every load in flight before the first use
  uint32_t key[CHUNKS];
  int val[CHUNKS];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int i = wbase + c * 32;
    key[c] = i < n ? keys_in[i] : 0u;
    val[c] = i < n ? vals_in[i] : 0;
  }
  const uint32_t row = hist[threadIdx.x * nblocks + blockIdx.x];
  for (int i = threadIdx.x; i < kSortWarps * 256; i += blockDim.x) (&wcount[0][0])[i] = 0;
  uint32_t all;
  const uint32_t start = block_exclusive_256(totals[threadIdx.x], warp_sums, &all) + row;
  // pass 1: per-warp digit counts
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    bool ok = wbase + c * 32 < n;
    uint32_t dgt = ok ? (key[c] >> shift) & 255u : 256u;
    unsigned peers = __match_any_sync(0xffffffffu, dgt);
    int leader = __ffs(peers) - 1;
    if (ok && lane == leader) wcount[w][dgt] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per-warp starting offsets: the digit's start, the earlier blocks', the
  // earlier warps'
  uint32_t run = start;
  for (int ww = 0; ww < kSortWarps; ++ww) {
    uint32_t c = wcount[ww][threadIdx.x];
    wcount[ww][threadIdx.x] = run;
    run += c;
  }
  __syncthreads();
  // pass 2: stable scatter in key order
  unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    bool ok = wbase + c * 32 < n;
    uint32_t dgt = ok ? (key[c] >> shift) & 255u : 256u;
    unsigned peers = __match_any_sync(0xffffffffu, dgt);
    int leader = __ffs(peers) - 1;
    if (ok) {
      uint32_t pos = wcount[w][dgt] + __popc(peers & lt);
      keys_out[pos] = key[c];
      vals_out[pos] = val[c];
    }
    __syncwarp();
    if (ok && lane == leader) wcount[w][dgt] += __popc(peers);
    __syncwarp();
  }
}

// Sorts (codes, idx) in place by the low `bits` bits of the key; stable.
static int radix_sort(Ctx* ctx, int n, uint32_t* keys, int* vals, int bits) {
  if (n <= 1) return RX_OK;
  cudaStream_t st = ctx->stream;
  const int chunks = n <= (1 << 20) ? 4 : 16, tile = sort_tile(chunks);
  int nblocks = (n + tile - 1) / tile;
  DevBuf<uint32_t> k2(ctx, n), hist(ctx, (size_t)256 * nblocks), totals(ctx, 256);
  DevBuf<int> v2(ctx, n);
  if (!all_ok(k2, hist, totals, v2)) return set_error(ctx, "BVH sort: out of device memory"), RX_ERR_CAPACITY;
  uint32_t* ka = keys;
  uint32_t* kb = k2.p;
  int* va = vals;
  int* vb = v2.p;
  int passes = (bits + 7) / 8;
  for (int p = 0; p < passes; ++p) {
    int shift = 8 * p;
    launch_chained(st, true, dim3(nblocks), 256, 0, k_sort_hist, n, ka, shift, tile, hist.p, nblocks);
    launch_chained(st, true, dim3(256), 256, 0, k_sort_rows, hist.p, totals.p, nblocks);
    auto scatter = chunks == 4 ? k_sort_scatter<4> : k_sort_scatter<16>;
    launch_chained(st, true, dim3(nblocks), kSortWarps * 32, 0, scatter, n, ka, va, kb, vb, shift, hist.p, totals.p,
                   nblocks);
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    cudaMemcpyAsync(keys, ka, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(vals, va, sizeof(int) * n, cudaMemcpyDeviceToDevice, st);
  }
  // k2, v2, hist, totals are released after the stream drains (DevBuf defers frees)
  return RX_OK;
}

// ----------------------------------------------------------------------------
// reference topology: median-by-count split of the sorted order
// ----------------------------------------------------------------------------
// Number of leaves of the count-median tree over m primitives, leaf <= L.
// At every depth the subtree sizes are s or s + 1, so two counters suffice.
__host__ __device__ inline long long median_tree_leaves(long long m, int L) {
  if (m <= L) return 1;
  long long leaves = 0, s = m, cs = 1, cs1 = 0;
  while (cs + cs1 > 0) {
    if (s + 1 <= L) {
      leaves += cs + cs1;
      break;
    }
    if (s <= L) {
      leaves += cs;
      cs = 0;
    }
    long long h = s / 2, ncs = 0, ncs1 = 0;
    if ((s & 1) == 0) ncs += 2 * cs; else { ncs += cs; ncs1 += cs; }
    if (((s + 1) & 1) == 0) ncs1 += 2 * cs1; else { ncs += cs1; ncs1 += cs1; }
    s = h;
    cs = ncs;
    cs1 = ncs1;
  }
  return leaves;
}

struct RefNodeItem {
  int idx, start, count, parent;
};

__global__ void k_ref_level(const RefNodeItem* __restrict__ cur, int ncur, RefNodeItem* __restrict__ next,
                            int* __restrict__ next_count, int leaf, int* __restrict__ left, int* __restrict__ right,
                            int* __restrict__ tstart, int* __restrict__ tcount, int* __restrict__ parent) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncur; i += gridDim.x * blockDim.x) {
    RefNodeItem it = cur[i];
    parent[it.idx] = it.parent;
    if (it.count <= leaf) {
      left[it.idx] = -1;
      right[it.idx] = -1;
      tstart[it.idx] = it.start;
      tcount[it.idx] = it.count;
    } else {
      int nl = it.count / 2;
      int li = it.idx + 1;
      int ri = it.idx + 1 + (int)(2 * median_tree_leaves(nl, leaf) - 1);
      left[it.idx] = li;
      right[it.idx] = ri;
      tstart[it.idx] = -1;
      tcount[it.idx] = 0;
      int o = atomicAdd(next_count, 2);
      next[o] = RefNodeItem{li, it.start, nl, it.idx};
      next[o + 1] = RefNodeItem{ri, it.start + nl, it.count - nl, it.idx};
    }
  }
}

// Leaves reduce their primitives' bounds, then walk up: the second child to
// arrive at a parent combines both (min / max are exact, order-free).
__global__ void k_ref_bounds(int n_nodes, const int* __restrict__ left, const int* __restrict__ right,
                             const int* __restrict__ tstart, const int* __restrict__ tcount,
                             const int* __restrict__ parent, const int* __restrict__ order,
                             const float3* __restrict__ pmin, const float3* __restrict__ pmax,
                             float3* __restrict__ nmin, float3* __restrict__ nmax, int* __restrict__ flags) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
    if (left[i] != -1) continue;
    float3 lo = f3(INFINITY, INFINITY, INFINITY), hi = f3(-INFINITY, -INFINITY, -INFINITY);
    for (int k = tstart[i]; k < tstart[i] + tcount[i]; ++k) {
      int t = order[k];
      lo = vmin(lo, pmin[t]);
      hi = vmax(hi, pmax[t]);
    }
    nmin[i] = lo;
    nmax[i] = hi;
    int node = parent[i];
    while (node >= 0) {
      __threadfence();
      if (atomicAdd(&flags[node], 1) == 0) break;  // first arrival: sibling finishes
      __threadfence();
      int l = left[node], r = right[node];
      float3 a0 = ldcg3(nmin + l), a1 = ldcg3(nmax + l);
      float3 b0 = ldcg3(nmin + r), b1 = ldcg3(nmax + r);
      nmin[node] = vmin(a0, b0);
      nmax[node] = vmax(a1, b1);
      node = parent[node];
    }
  }
}

// Reference-format nodes -> traversal layout (node index preserved, so the
// root stays 0).  A root leaf gets a wrapper node whose right child is an
// empty leaf.
__global__ void k_ref_to_layout(int n_nodes, const int* __restrict__ left, const int* __restrict__ right,
                                const int* __restrict__ tstart, const int* __restrict__ tcount,
                                const float3* __restrict__ nmin, const float3* __restrict__ nmax,
                                float4* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
    int l, r;
    float3 l0, l1, r0, r1;
    int lw, rw, lc, rc;
    if (left[i] == -1) {
      if (i != 0) continue;  // leaves live inside their parent's record
      l0 = nmin[0]; l1 = nmax[0];
      lw = pack_leaf(tstart[0], tcount[0]); lc = tcount[0];
      r0 = f3(1e30f, 1e30f, 1e30f); r1 = r0;
      rw = pack_leaf(0, 0); rc = 0;
    } else {
      l = left[i];
      r = right[i];
      l0 = nmin[l]; l1 = nmax[l];
      r0 = nmin[r]; r1 = nmax[r];
      lw = left[l] == -1 ? pack_leaf(tstart[l], tcount[l]) : l;
      lc = left[l] == -1 ? tcount[l] : 0;
      rw = left[r] == -1 ? pack_leaf(tstart[r], tcount[r]) : r;
      rc = left[r] == -1 ? tcount[r] : 0;
    }
    float4* o = out + 4 * (size_t)i;
    o[0] = make_float4(l0.x, l1.x, l0.y, l1.y);
    o[1] = make_float4(l0.z, l1.z, r0.x, r1.x);
    o[2] = make_float4(r0.y, r1.y, r0.z, r1.z);
    o[3] = make_float4(__int_as_float(lw), __int_as_float(rw), __int_as_float(lc), __int_as_float(rc));
  }
}

// Primitives and shading records gathered into leaf order.
__global__ void k_gather_prims(int n, const int* __restrict__ order, int n_tris, const float* __restrict__ v0,
                               const float* __restrict__ v1, const float* __restrict__ v2,
                               const float* __restrict__ n0, const float* __restrict__ n1,
                               const float* __restrict__ n2, const int* __restrict__ tri_mat,
                               const float4* __restrict__ obj_a, const float4* __restrict__ obj_b,
                               const int* __restrict__ obj_mat, const int* __restrict__ obj_slot,
                               float4* __restrict__ prims, float4* __restrict__ shade) {
  chain_wait(order, v0, v1, v2, n0, n1, n2, tri_mat, obj_a, obj_b, obj_mat, obj_slot, prims, shade);
  chain_go();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    int i = order[k];
    float4* P = prims + kPrimQuads * (size_t)k;
    float4* S = shade + 3 * (size_t)k;
    if (i < n_tris) {
      float3 a = f3(v0[3 * i], v0[3 * i + 1], v0[3 * i + 2]);
      float3 b = f3(v1[3 * i], v1[3 * i + 1], v1[3 * i + 2]);
      float3 c = f3(v2[3 * i], v2[3 * i + 1], v2[3 * i + 2]);
      float3 e1 = b - a, e2 = c - a;
      P[0] = make_float4(a.x, a.y, a.z, __int_as_float(PRIM_TRI));
      P[1] = make_float4(e1.x, e1.y, e1.z, e2.x);
      P[2] = make_float4(e2.y, e2.z, 0.0f, 0.0f);
      S[0] = make_float4(n0[3 * i], n0[3 * i + 1], n0[3 * i + 2], __int_as_float(tri_mat ? tri_mat[i] : 0));
      S[1] = make_float4(n1[3 * i], n1[3 * i + 1], n1[3 * i + 2], __int_as_float(i));
      S[2] = make_float4(n2[3 * i], n2[3 * i + 1], n2[3 * i + 2], 0.0f);
    } else {
      int s = i - n_tris;
      P[0] = obj_a[s];
      P[1] = obj_b[s];
      P[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      S[0] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(obj_mat[s]));
      S[1] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(obj_slot[s]));
      S[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
}

// ----------------------------------------------------------------------------
// Karras LBVH + SAH collapse
// ----------------------------------------------------------------------------
__device__ __forceinline__ int lcp(const uint32_t* codes, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  uint32_t a = codes[i], b = codes[j];
  if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
  return __clz(a ^ b);
}

// Children are encoded as c >= 0 internal, c < 0 leaf ~prim (sorted position).
__device__ __forceinline__ int left_child(int lo, int gamma) { return lo == gamma ? ~gamma : gamma; }
__device__ __forceinline__ int right_child(int hi, int gamma) { return hi == gamma + 1 ? ~(gamma + 1) : gamma + 1; }

// Internal node i of n - 1 covers the sorted positions [lo, hi], split after
// gamma: record (lo, hi, gamma, -).  Also clears the bottom-up flags and the
// mask counts of the passes that follow.
__global__ void k_karras(int n, const uint32_t* __restrict__ codes, int4* __restrict__ range,
                         int* __restrict__ parent_int, int* __restrict__ parent_leaf, int* __restrict__ flags,
                         int* __restrict__ counts, int n_counts) {
  chain_wait(codes, range, parent_int, parent_leaf, flags, counts);
  chain_go();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
    int d = (lcp(codes, n, i, i + 1) - lcp(codes, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = lcp(codes, n, i, i - d);
    int lmax = 2;
    while (lcp(codes, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
      if (lcp(codes, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = lcp(codes, n, i, j);
    int s = 0;
    int t = l;
    do {
      t = (t + 1) >> 1;
      if (lcp(codes, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    range[i] = make_int4(lo, hi, gamma, 0);
    flags[i] = 0;
    if (i < n_counts) counts[i] = 0;
    if (i == 0) parent_int[0] = -1;  // the root; every other node has a parent that writes it
    const int lc = left_child(lo, gamma), rc = right_child(hi, gamma);
    if (lc >= 0) parent_int[lc] = i; else parent_leaf[~lc] = i;
    if (rc >= 0) parent_int[rc] = i; else parent_leaf[~rc] = i;
  }
}

__device__ __forceinline__ float half_area(float3 lo, float3 hi) {
  float3 e = hi - lo;
  return e.x * e.y + e.y * e.z + e.z * e.x;
}

// Bottom-up bounds and SAH cost.  cost(node) = min(C_i * count (if count <=
// max_leaf), C_t + (A_l cost_l + A_r cost_r) / A).  Node record: a = (min,
// cost), b = (max, height bits), height = levels of the tree under the node,
// 0 where it collapses into a leaf.
//
// The second thread to reach a node computes it.  A block owns kUpLeaves
// consecutive sorted positions: a node that covers none outside them (9 of
// ~20 levels, all but some thousand nodes of a 327 k mesh) is counted and
// its record handed on in shared memory, the rest by device-scope fences and
// atomics; that chain of ~2 us per level was the pass's time.
constexpr int kUpLeaves = 512;

// Adds 1 to a node's counter; what the other thread wrote before its own call
// is visible to the second caller.  (An atomicAdd between two __threadfence,
// which order more: 76 us for the pass, 69 with this.)
__device__ __forceinline__ int arrive(int* flag) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(flag) : "memory");
  return old;
}
__device__ __forceinline__ int arrive_shared(int* flag) {
  int old;
  asm volatile("atom.acq_rel.cta.shared.add.s32 %0, [%1], 1;"
               : "=r"(old)
               : "r"((uint32_t)__cvta_generic_to_shared(flag))
               : "memory");
  return old;
}

struct UpBox {
  float3 lo, hi;
  float cost;
  int height;
};

__device__ __forceinline__ UpBox up_box(float4 a, float4 b) {
  return {f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), a.w, __float_as_int(b.w)};
}

__global__ void __launch_bounds__(kUpLeaves)
    k_lbvh_bottom_up(int n, const int* __restrict__ order, const int4* __restrict__ range,
                     const int* __restrict__ parent_int, const int* __restrict__ parent_leaf,
                     const float3* __restrict__ pmin, const float3* __restrict__ pmax, float4* __restrict__ rec,
                     int* __restrict__ flags, int max_leaf, float c_t, float c_i) {
  chain_wait(order, range, parent_int, parent_leaf, pmin, pmax, rec, flags);
  chain_go();
  __shared__ float4 s_a[kUpLeaves], s_b[kUpLeaves];  // records of this block's nodes, by node - base
  __shared__ float3 s_lo[kUpLeaves], s_hi[kUpLeaves];
  __shared__ int4 s_range[kUpLeaves];  // (lo, hi, gamma, parent)
  __shared__ int s_flag[kUpLeaves];
  const int base = blockIdx.x * kUpLeaves, end = min(base + kUpLeaves, n), k = base + threadIdx.x;
  int node = -1;
  s_flag[threadIdx.x] = 0;
  if (k < end) {
    const int p = order[k];
    node = parent_leaf[k];
    s_lo[threadIdx.x] = pmin[p];
    s_hi[threadIdx.x] = pmax[p];
    if (k < n - 1) {
      int4 q = range[k];
      q.w = parent_int[k];
      s_range[threadIdx.x] = q;
    }
  }
  __syncthreads();
  if (k >= end) return;
  // a node's index lies inside its range, so one that is not here is no
  // block's own
  auto node_range = [&](int i) {
    if (i >= base && i < end) return s_range[i - base];
    int4 q = range[i];
    q.w = parent_int[i];
    return q;
  };
  auto compute = [&](const int4 q, const UpBox& l, const UpBox& r, float4& a, float4& b) {
    const float3 lo = vmin(l.lo, r.lo), hi = vmax(l.hi, r.hi);
    const float area = fmaxf(half_area(lo, hi), 1e-30f);
    const float split = c_t + (half_area(l.lo, l.hi) * l.cost + half_area(r.lo, r.hi) * r.cost) / area;
    const int cnt = q.y - q.x + 1;
    const float leafc = c_i * (float)cnt;
    const bool col = cnt <= max_leaf && leafc <= split;
    a = make_float4(lo.x, lo.y, lo.z, col ? leafc : split);
    b = make_float4(hi.x, hi.y, hi.z, __int_as_float(col ? 0 : 1 + max(l.height, r.height)));
  };
  int4 q = node_range(node);
  while (q.x >= base && q.y < end) {
    if (arrive_shared(&s_flag[node - base]) == 0) return;
    auto child = [&](int c) {
      if (c < 0) return UpBox{s_lo[~c - base], s_hi[~c - base], c_i, 0};
      return up_box(s_a[c - base], s_b[c - base]);
    };
    float4 a, b;
    compute(q, child(left_child(q.x, q.z)), child(right_child(q.y, q.z)), a, b);
    s_a[node - base] = a;
    s_b[node - base] = b;
    rec[2 * (size_t)node] = a;
    rec[2 * (size_t)node + 1] = b;
    if (q.w < 0) return;
    node = q.w;
    q = node_range(node);
  }
  while (true) {
    if (arrive(flags + node) == 0) return;
    const int4 up = q.w < 0 ? q : node_range(q.w);  // in flight with the children's records
    auto child = [&](int c) {
      if (c >= 0) return up_box(__ldcg(rec + 2 * (size_t)c), __ldcg(rec + 2 * (size_t)c + 1));
      const int p = order[~c];
      return UpBox{pmin[p], pmax[p], c_i, 0};
    };
    float4 a, b;
    compute(q, child(left_child(q.x, q.z)), child(right_child(q.y, q.z)), a, b);
    rec[2 * (size_t)node] = a;
    rec[2 * (size_t)node + 1] = b;
    if (q.w < 0) return;
    node = q.w;
    q = up;
  }
}

// Compaction of marked nodes: a bit mask, the marked nodes per kRankWords
// mask words (added up while marking), and the rank of every mask word.
constexpr int kRankWords = 256;

struct NodeMask {
  uint32_t* mask;  // a multiple of kRankWords words
  int* rank;       // marked nodes before each word
  int* counts;     // marked nodes per kRankWords words; zero before marking
  __device__ __forceinline__ int index(int i) const {
    return rank[i >> 5] + __popc(mask[i >> 5] & ((1u << (i & 31)) - 1u));
  }
  __device__ __forceinline__ bool has(int i) const { return mask[i >> 5] >> (i & 31) & 1u; }
  // one word per warp, called by whole warps
  __device__ __forceinline__ void mark(int i, bool keep) const {
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if ((i & 31) == 0) {
      mask[i >> 5] = m;
      if (m) atomicAdd(counts + (i >> 5) / kRankWords, __popc(m));
    }
  }
};

// One block per kRankWords words; the last one writes *total.
__global__ void __launch_bounds__(kRankWords) k_rank(NodeMask m, int n, int* __restrict__ total) {
  chain_wait(m.mask, m.rank, m.counts, total);
  chain_go();
  __shared__ uint32_t warp_sums[8];
  uint32_t before = 0, part = 0, here = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kRankWords) part += m.counts[b];
  block_exclusive_256(part, warp_sums, &before);
  const int w = blockIdx.x * kRankWords + threadIdx.x;
  // words beyond the last node are never written
  const uint32_t e = block_exclusive_256(w * 32LL < n ? __popc(m.mask[w]) : 0, warp_sums, &here);
  m.rank[w] = (int)(before + e);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = (int)(before + here);
}

// Layout of the collapsed tree: a node stays when neither it nor an ancestor
// collapses, and its index is the number of nodes before it that stay (the
// root is node 0).  Only nodes of up to max_leaf primitives have ancestors
// that can collapse.  (One launch per level, breadth first, was 26 to 32
// launches of 3-12 us, 265 us for the 327 k mesh; these three take 34.)
__device__ __forceinline__ int rec_height(const float4* rec, int node) {
  return __float_as_int(rec[2 * (size_t)node + 1].w);
}

__global__ void __launch_bounds__(256)
    k_lbvh_keep(int n_int, const int4* __restrict__ range, const int* __restrict__ parent_int,
                const float4* __restrict__ rec, int max_leaf, NodeMask m, int* __restrict__ levels) {
  chain_wait(range, parent_int, rec, m.mask, m.rank, m.counts, levels);
  chain_go();
  const int i = blockIdx.x * 256 + threadIdx.x;
  bool keep = i < n_int && rec_height(rec, i) > 0;
  for (int p = i; keep;) {
    const int4 q = range[p];
    if (q.y - q.x + 1 > max_leaf) break;
    p = parent_int[p];
    if (p < 0) break;
    keep = rec_height(rec, p) > 0;
  }
  m.mark(i, keep);
  if (i == 0) *levels = rec_height(rec, 0);
}

// at_lo: first sorted position under each laid-out node.
__global__ void k_lbvh_layout(int n_int, const int4* __restrict__ range, const int* __restrict__ order,
                              const float3* __restrict__ pmin, const float3* __restrict__ pmax,
                              const float4* __restrict__ rec, NodeMask m, float4* __restrict__ out,
                              int* __restrict__ at_lo) {
  chain_wait(range, order, pmin, pmax, rec, m.mask, m.rank, m.counts, out, at_lo);
  chain_go();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_int; i += gridDim.x * blockDim.x) {
    if (!m.has(i)) continue;
    const int4 q = range[i];
    const int ch[2] = {left_child(q.x, q.z), right_child(q.y, q.z)};
    int words[2], counts[2];
    float3 b0[2], b1[2];
    for (int s = 0; s < 2; ++s) {
      const int c = ch[s];
      if (c < 0) {
        const int p = order[~c];
        b0[s] = pmin[p];
        b1[s] = pmax[p];
        words[s] = pack_leaf(~c, 1);  // one primitive at sorted position ~c
        counts[s] = 1;
        continue;
      }
      const UpBox u = up_box(rec[2 * (size_t)c], rec[2 * (size_t)c + 1]);
      b0[s] = u.lo;
      b1[s] = u.hi;
      if (u.height == 0) {  // the left child covers [lo, gamma], the right one [gamma + 1, hi]
        const int lo = s ? q.z + 1 : q.x, hi = s ? q.y : q.z;
        words[s] = pack_leaf(lo, hi - lo + 1);
        counts[s] = hi - lo + 1;
      } else {
        words[s] = m.index(c);
        counts[s] = 0;
      }
    }
    const size_t at = m.index(i);
    at_lo[at] = q.x;
    float4* o = out + 4 * at;
    o[0] = make_float4(b0[0].x, b1[0].x, b0[0].y, b1[0].y);
    o[1] = make_float4(b0[0].z, b1[0].z, b0[1].x, b1[1].x);
    o[2] = make_float4(b0[1].y, b1[1].y, b0[1].z, b1[1].z);
    o[3] = make_float4(__int_as_float(words[0]), __int_as_float(words[1]), __int_as_float(counts[0]),
                       __int_as_float(counts[1]));
  }
}

// 4-wide nodes from the laid-out binary tree.  The 4-wide node of binary
// node b starts from b's two children and, while it has fewer than four,
// opens the internal child of largest surface area (replacing it by its own
// two children): the children that the most rays enter are expanded first,
// which removes more node visits than always taking both grandchildren
// (6-8 % fewer visits per ray on the displaced icosphere).  Leaf children
// stay leaves; internal children that remain are 4-wide nodes themselves.
// Empty binary slots (count 0 leaves) are dropped; unused slots get a box at
// 1e30 and count 0.
//
// Which children b would have depends on b's subtree alone, so every binary
// node works them out at once (k_wide_kids); a node then follows those lists
// from the root towards itself to see whether it is reached (k_wide_roots),
// and the reached ones write their records (k_wide_write).  Four short
// launches, whatever the depth: 150 -> 45 us for the 327 k mesh against a
// launch per level of the 4-wide tree (and 184 us with one cooperative
// launch and a grid barrier per level).
struct WideNode {
  float mn[4][3], mx[4][3];
  int wd[4], ct[4];
  int k;
};

// All slots are registers: every index below is a constant after unrolling.
__device__ __forceinline__ void wide_add(WideNode& v, const float4* __restrict__ nb, bool second, int* err) {
  const float4 n0 = nb[0], n1 = nb[1], n2 = nb[2], n3 = nb[3];
  const int w = __float_as_int(second ? n3.y : n3.x), c = __float_as_int(second ? n3.w : n3.z);
  if (w < 0 && c == 0) return;  // empty slot
  if (v.k >= 4) {               // cannot happen: a node is opened only while k < 4
    atomicOr(err, ERR_BAD_NODE);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i != v.k) continue;
    v.mn[i][0] = second ? n1.z : n0.x, v.mx[i][0] = second ? n1.w : n0.y;
    v.mn[i][1] = second ? n2.x : n0.z, v.mx[i][1] = second ? n2.y : n0.w;
    v.mn[i][2] = second ? n2.z : n1.x, v.mx[i][2] = second ? n2.w : n1.y;
    v.wd[i] = w;
    v.ct[i] = w >= 0 ? 0 : c;
  }
  ++v.k;
}

__device__ __forceinline__ void wide_open(WideNode& v, const float4* __restrict__ bin, int n_bin, int b, int* err) {
  v.k = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v.mn[i][0] = v.mn[i][1] = v.mn[i][2] = 1e30f;
    v.mx[i][0] = v.mx[i][1] = v.mx[i][2] = 1e30f;
    v.wd[i] = pack_leaf(0, 0);
    v.ct[i] = 0;
  }
  wide_add(v, bin + 4 * (size_t)b, false, err);
  wide_add(v, bin + 4 * (size_t)b, true, err);
  while (v.k < 4) {
    int bi = -1, open = 0;
    float ba = -1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i >= v.k || v.wd[i] < 0) continue;
      if (v.wd[i] >= n_bin) {  // never entered: flagged and turned into an empty leaf
        atomicOr(err, ERR_BAD_NODE);
        v.wd[i] = pack_leaf(0, 0);
        v.ct[i] = 0;
        continue;
      }
      const float ex = v.mx[i][0] - v.mn[i][0], ey = v.mx[i][1] - v.mn[i][1], ez = v.mx[i][2] - v.mn[i][2];
      const float a = ex * ey + ey * ez + ez * ex;
      if (a > ba) {
        ba = a;
        bi = i;
        open = v.wd[i];
      }
    }
    if (bi < 0) break;
    // remove entry bi (the last entry moves into its place), then append its
    // two children
    --v.k;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = i + 1; j < 4; ++j) {
        if (i != bi || j != v.k) continue;
#pragma unroll
        for (int a = 0; a < 3; ++a) v.mn[i][a] = v.mn[j][a], v.mx[i][a] = v.mx[j][a];
        v.wd[i] = v.wd[j];
        v.ct[i] = v.ct[j];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i != v.k) continue;  // the freed slot, should both children be empty
      v.mn[i][0] = v.mn[i][1] = v.mn[i][2] = 1e30f;
      v.mx[i][0] = v.mx[i][1] = v.mx[i][2] = 1e30f;
      v.wd[i] = pack_leaf(0, 0);
      v.ct[i] = 0;
    }
    wide_add(v, bin + 4 * (size_t)open, false, err);
    wide_add(v, bin + 4 * (size_t)open, true, err);
  }
}

// kids[2b]: the internal children of b's 4-wide node (-1: none), kids[2b + 1]:
// the first sorted position under each.  Also clears the mask counts.
__global__ void __launch_bounds__(128) k_wide_kids(const float4* __restrict__ bin, int n_bin,
                                                   const int* __restrict__ at_lo, int4* __restrict__ kids,
                                                   int* __restrict__ counts, int n_counts, int* err) {
  chain_wait(bin, at_lo, kids, counts);
  chain_go();
  const int b = blockIdx.x * 128 + threadIdx.x;
  if (b >= n_bin) return;
  if (b < n_counts) counts[b] = 0;
  WideNode v;
  wide_open(v, bin, n_bin, b, err);
  int id[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool in = v.wd[i] >= 0 && v.wd[i] < n_bin;
    id[i] = in ? v.wd[i] : -1;
    lo[i] = in ? at_lo[v.wd[i]] : INT_MAX;
  }
  kids[2 * (size_t)b] = make_int4(id[0], id[1], id[2], id[3]);
  kids[2 * (size_t)b + 1] = make_int4(lo[0], lo[1], lo[2], lo[3]);
}

// Marks the binary nodes that are 4-wide nodes: from the root, the child
// that holds b's first position is the one of largest first position not
// beyond it.  A node that an ancestor opened is passed by and the walk ends
// below it.
__global__ void __launch_bounds__(256) k_wide_roots(int n_bin, const int4* __restrict__ kids,
                                                    const int* __restrict__ at_lo, NodeMask m) {
  chain_wait(kids, at_lo, m.mask, m.rank, m.counts);
  chain_go();
  const int b = blockIdx.x * 256 + threadIdx.x;
  int cur = b < n_bin ? 0 : -1;
  const int p = b < n_bin ? at_lo[b] : 0;
  for (int s = 0; s < 64 && cur >= 0 && cur != b; ++s) {  // a tree of 62-bit keys has fewer levels
    const int4 id = kids[2 * (size_t)cur], lo = kids[2 * (size_t)cur + 1];
    int best = -1;
    cur = -1;
    if (lo.x <= p && lo.x > best) best = lo.x, cur = id.x;
    if (lo.y <= p && lo.y > best) best = lo.y, cur = id.y;
    if (lo.z <= p && lo.z > best) best = lo.z, cur = id.z;
    if (lo.w <= p && lo.w > best) best = lo.w, cur = id.w;
  }
  m.mark(b, b < n_bin && cur == b);
}

__global__ void __launch_bounds__(128) k_wide_write(const float4* __restrict__ bin, int n_bin, NodeMask m,
                                                    float4* __restrict__ out4, int* err) {
  chain_wait(bin, m.mask, m.rank, m.counts, out4);
  chain_go();
  const int b = blockIdx.x * 128 + threadIdx.x;
  if (b >= n_bin || !m.has(b)) return;
  WideNode v;
  wide_open(v, bin, n_bin, b, err);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (v.wd[i] >= 0 && v.wd[i] < n_bin) v.wd[i] = m.index(v.wd[i]);
  float4* o = out4 + 8 * (size_t)m.index(b);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o[2 * a] = make_float4(v.mn[0][a], v.mn[1][a], v.mn[2][a], v.mn[3][a]);
    o[2 * a + 1] = make_float4(v.mx[0][a], v.mx[1][a], v.mx[2][a], v.mx[3][a]);
  }
  o[6] = make_float4(__int_as_float(v.wd[0]), __int_as_float(v.wd[1]), __int_as_float(v.wd[2]),
                     __int_as_float(v.wd[3]));
  o[7] = make_float4(__int_as_float(v.ct[0]), __int_as_float(v.ct[1]), __int_as_float(v.ct[2]),
                     __int_as_float(v.ct[3]));
}

// Root record for a tree that is a single leaf of `cnt` primitives.
__global__ void k_single_leaf_root(const float3* __restrict__ bmin, const float3* __restrict__ bmax, int cnt,
                                   float4* __restrict__ out) {
  float3 l0 = bmin[0], l1 = bmax[0];
  float3 r0 = f3(1e30f, 1e30f, 1e30f);
  out[0] = make_float4(l0.x, l1.x, l0.y, l1.y);
  out[1] = make_float4(l0.z, l1.z, r0.x, r0.x);
  out[2] = make_float4(r0.y, r0.y, r0.z, r0.z);
  out[3] = make_float4(__int_as_float(pack_leaf(0, cnt)), __int_as_float(pack_leaf(0, 0)), __int_as_float(cnt),
  __int_as_float(0));
}

static int grid_for(Ctx* ctx, long long n, int block = 256) {
  long long g = (n + block - 1) / block;
  long long cap = (long long)ctx->num_sms * 32;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

// Shared front end: bounds, centroids, Morton codes, stable sort.
// lbvh_keys != 0: Morton keys of box centres on cubic cells (the LBVH); 0:
// the reference's centroids and per-axis normalisation.
static int front_end(Ctx* ctx, Scene* sc, int n_obj, const float4* d_obj_a, const float4* d_obj_b, int lbvh_keys,
                     DevBuf<float3>& pmin, DevBuf<float3>& pmax, DevBuf<int>& order) {
  int n = sc->n_tris + n_obj;
  cudaStream_t st = ctx->stream;
  DevBuf<float3> cen(ctx, n);
  const int parts = std::min(grid_for(ctx, n), 1024);
  DevBuf<float3> part_min(ctx, parts), part_max(ctx, parts);
  DevBuf<uint32_t> codes(ctx, n);
  DevBuf<float3> cbox(ctx, 2);
  if (!all_ok(pmin, pmax, order, cen, part_min, part_max, codes, cbox))
    return set_error(ctx, "BVH build: out of device memory"), RX_ERR_CAPACITY;
  k_prim_bounds<<<grid_for(ctx, n), 256, 0, st>>>(sc->n_tris, sc->d_v0, sc->d_v1, sc->d_v2, n_obj, d_obj_a, d_obj_b,
                                                   lbvh_keys, pmin.p, pmax.p, cen.p);
  launch_chained(st, true, dim3(parts), 256, 0, k_reduce_bounds, n, cen.p, part_min.p, part_max.p);
  launch_chained(st, true, dim3(1), kBoundsThreads, 0, k_bounds_final, parts, part_min.p, part_max.p, cbox.p);
  launch_chained(st, true, dim3(grid_for(ctx, n)), 256, 0, k_morton, n, cen.p, cbox.p, lbvh_keys, codes.p, order.p);
  if (int rc = radix_sort(ctx, n, codes.p, order.p, 30)) return rc;
  sc->tmp_codes.swap(codes);
  return RX_OK;
}

int build_reference(Ctx* ctx, Scene* sc, int leaf) {
  cudaStream_t st = ctx->stream;
  int n = sc->n_tris;
  sc->clear_bvh();
  if (n <= 0) return RX_OK;
  DevBuf<float3> pmin(ctx, n), pmax(ctx, n);
  DevBuf<int> order(ctx, n);
  if (int rc = front_end(ctx, sc, 0, nullptr, nullptr, 0, pmin, pmax, order)) return rc;
  long long n_nodes_ll = 2 * median_tree_leaves(n, leaf) - 1;
  int n_nodes = (int)n_nodes_ll;
  DevBuf<int> left(ctx, n_nodes), right(ctx, n_nodes), tstart(ctx, n_nodes), tcount(ctx, n_nodes);
  DevBuf<int> parent(ctx, n_nodes), flags(ctx, n_nodes);
  DevBuf<float3> nmin(ctx, n_nodes), nmax(ctx, n_nodes);
  DevBuf<RefNodeItem> la(ctx, n_nodes), lb(ctx, n_nodes);
  DevBuf<int> cnt(ctx, 1);
  if (!all_ok(left, right, tstart, tcount, parent, flags, nmin, nmax, la, lb, cnt))
    return set_error(ctx, "reference build: out of device memory"), RX_ERR_CAPACITY;
  RefNodeItem root{0, 0, n, -1};
  cudaMemcpyAsync(la.p, &root, sizeof(root), cudaMemcpyHostToDevice, st);
  int ncur = 1;
  RefNodeItem* cur = la.p;
  RefNodeItem* nxt = lb.p;
  int levels = 0;
  while (ncur > 0) {
    if (++levels > 256 || ncur > n_nodes)
      return set_error(ctx, "reference build: level walk did not terminate"), RX_ERR_DEVICE;
    cudaMemsetAsync(cnt.p, 0, sizeof(int), st);
    k_ref_level<<<grid_for(ctx, ncur), 256, 0, st>>>(cur, ncur, nxt, cnt.p, leaf, left.p, right.p, tstart.p,
                                                      tcount.p, parent.p);
    int h = 0;
    cudaMemcpyAsync(&h, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    ncur = h;
    std::swap(cur, nxt);
  }
  cudaMemsetAsync(flags.p, 0, sizeof(int) * n_nodes, st);
  k_ref_bounds<<<grid_for(ctx, n_nodes), 256, 0, st>>>(n_nodes, left.p, right.p, tstart.p, tcount.p, parent.p,
                                                        order.p, pmin.p, pmax.p, nmin.p, nmax.p, flags.p);
  sc->d_nodes.alloc(ctx, (size_t)4 * n_nodes);
  sc->d_prims.alloc(ctx, (size_t)kPrimQuads * n);
  sc->d_shade.alloc(ctx, (size_t)3 * n);
  if (!all_ok(sc->d_nodes, sc->d_prims, sc->d_shade)) {
    sc->clear_bvh();
    return set_error(ctx, "reference build: out of device memory"), RX_ERR_CAPACITY;
  }
  k_ref_to_layout<<<grid_for(ctx, n_nodes), 256, 0, st>>>(n_nodes, left.p, right.p, tstart.p, tcount.p, nmin.p,
                                                           nmax.p, sc->d_nodes.p);
  launch_chained(st, true, dim3(grid_for(ctx, n)), 256, 0, k_gather_prims, n, order.p, sc->n_tris, sc->d_v0, sc->d_v1,
                 sc->d_v2, sc->d_n0, sc->d_n1, sc->d_n2, sc->d_tri_mat, nullptr, nullptr, nullptr, nullptr,
                 sc->d_prims.p, sc->d_shade.p);
  float3 rb[2];
  cudaMemcpyAsync(&rb[0], nmin.p, sizeof(float3), cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&rb[1], nmax.p, sizeof(float3), cudaMemcpyDeviceToHost, st);
  // keep the reference-format arrays for export
  sc->ref_left.swap(left);
  sc->ref_right.swap(right);
  sc->ref_start.swap(tstart);
  sc->ref_count.swap(tcount);
  sc->ref_min.swap(nmin);
  sc->ref_max.swap(nmax);
  sc->order.swap(order);
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  sc->root_min = rb[0];
  sc->root_max = rb[1];
  sc->n_nodes = n_nodes;
  sc->n_prims = n;
  sc->n_bvh_spheres = 0;
  sc->method = RX_BVH_REFERENCE;
  sc->exact_slab = 1;
  sc->leaf_size = leaf;
  return RX_OK;
}

// Upload of an externally built tree in the reference's node format.
int set_reference_nodes(Ctx* ctx, Scene* sc, int n_nodes, const float* node_min, const float* node_max,
                        const int* left, const int* right, const int* start, const int* count, const int* order) {
  cudaStream_t st = ctx->stream;
  int n = sc->n_tris;
  sc->clear_bvh();
  if (n <= 0 || n_nodes <= 0) return RX_OK;
  DevBuf<int> l(ctx, n_nodes), r(ctx, n_nodes), s(ctx, n_nodes), c(ctx, n_nodes), ord(ctx, n);
  DevBuf<float3> nmin(ctx, n_nodes), nmax(ctx, n_nodes);
  sc->d_nodes.alloc(ctx, (size_t)4 * n_nodes);
  sc->d_prims.alloc(ctx, (size_t)kPrimQuads * n);
  sc->d_shade.alloc(ctx, (size_t)3 * n);
  if (!all_ok(l, r, s, c, ord, nmin, nmax, sc->d_nodes, sc->d_prims, sc->d_shade)) {
    sc->clear_bvh();
    return set_error(ctx, "BVH upload: out of device memory"), RX_ERR_CAPACITY;
  }
  cudaMemcpyAsync(l.p, left, sizeof(int) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(r.p, right, sizeof(int) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(s.p, start, sizeof(int) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(c.p, count, sizeof(int) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(nmin.p, node_min, sizeof(float3) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(nmax.p, node_max, sizeof(float3) * n_nodes, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(ord.p, order, sizeof(int) * n, cudaMemcpyHostToDevice, st);
  k_ref_to_layout<<<grid_for(ctx, n_nodes), 256, 0, st>>>(n_nodes, l.p, r.p, s.p, c.p, nmin.p, nmax.p,
                                                           sc->d_nodes.p);
  launch_chained(st, true, dim3(grid_for(ctx, n)), 256, 0, k_gather_prims, n, ord.p, sc->n_tris, sc->d_v0, sc->d_v1,
                 sc->d_v2, sc->d_n0, sc->d_n1, sc->d_n2, sc->d_tri_mat, nullptr, nullptr, nullptr, nullptr,
                 sc->d_prims.p, sc->d_shade.p);
  sc->ref_left.swap(l);
  sc->ref_right.swap(r);
  sc->ref_start.swap(s);
  sc->ref_count.swap(c);
  sc->ref_min.swap(nmin);
  sc->ref_max.swap(nmax);
  sc->order.swap(ord);
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  sc->root_min = f3(node_min[0], node_min[1], node_min[2]);
  sc->root_max = f3(node_max[0], node_max[1], node_max[2]);
  sc->n_nodes = n_nodes;
  sc->n_prims = n;
  sc->n_bvh_spheres = 0;
  sc->method = RX_BVH_REFERENCE;
  sc->exact_slab = 1;
  sc->leaf_size = 0;
  return RX_OK;
}

// Mask, ranks and counts for n nodes.
struct MaskBuf {
  int blocks;
  DevBuf<uint32_t> mask;
  DevBuf<int> rank, counts;
  MaskBuf(Ctx* ctx, int n)
      : blocks((n + 32 * kRankWords - 1) / (32 * kRankWords)),
        mask(ctx, (size_t)blocks * kRankWords),
        rank(ctx, (size_t)blocks * kRankWords),
        counts(ctx, blocks) {}
  NodeMask view() const { return {mask.p, rank.p, counts.p}; }
};

// The 4-wide copy of the laid-out binary tree; at_lo: the first sorted
// position under each of its nodes.
static int build_wide(Ctx* ctx, Scene* sc, const int* at_lo) {
  cudaStream_t st = ctx->stream;
  const int nb = sc->n_nodes;
  sc->n_nodes4 = 0;
  if (nb <= 0) return RX_OK;
  if (!sc->d_nodes4.alloc(ctx, (size_t)8 * nb)) return set_error(ctx, "out of device memory for the 4-wide BVH"),
  RX_ERR_CAPACITY;
  MaskBuf m(ctx, nb);
  DevBuf<int4> kids(ctx, (size_t)2 * nb);
  DevBuf<int> total(ctx, 1);
  if (!all_ok(m.mask, m.rank, m.counts, kids, total)) return set_error(ctx, "out of device memory"), RX_ERR_CAPACITY;
  launch_chained(st, true, dim3((nb + 127) / 128), 128, 0, k_wide_kids, sc->d_nodes.p, nb, at_lo, kids.p, m.counts.p,
                 m.blocks, ctx->d_err);
  launch_chained(st, true, dim3((nb + 255) / 256), 256, 0, k_wide_roots, nb, kids.p, at_lo, m.view());
  launch_chained(st, true, dim3(m.blocks), kRankWords, 0, k_rank, m.view(), nb, total.p);
  launch_chained(st, true, dim3((nb + 127) / 128), 128, 0, k_wide_write, sc->d_nodes.p, nb, m.view(), sc->d_nodes4.p,
                 ctx->d_err);
  CUDA_TRY(ctx, cudaGetLastError());
  int n4 = 0;
  CUDA_TRY(ctx, cudaMemcpyAsync(&n4, total.p, sizeof(n4), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  sc->n_nodes4 = n4;
  return RX_OK;
}

int build_lbvh(Ctx* ctx, Scene* sc, int max_leaf, int spheres_in_bvh, float c_t, float c_i) {
  cudaStream_t st = ctx->stream;
  sc->clear_bvh();
  // bounded analytic objects (spheres, cubes) taken from the object slots
  // into the BVH; planes (unbounded) and slot triangles stay linear
  std::vector<float4> oa, ob;
  std::vector<int> obj_mat, obj_slot;
  sc->bvh_sphere_slots.clear();
  if (spheres_in_bvh) {
    for (int i = 0; i < (int)sc->objs.size(); ++i) {
      const ObjSlot& o = sc->objs[i];
      if (o.type == 0) {
        oa.push_back(make_float4(o.center.x, o.center.y, o.center.z, int_bits_as_float(PRIM_SPHERE)));
        ob.push_back(make_float4(o.radius, 0.0f, 0.0f, 0.0f));
      } else if (o.type == 2) {
        oa.push_back(make_float4(o.center.x, o.center.y, o.center.z, int_bits_as_float(PRIM_CUBE)));
        ob.push_back(make_float4(o.extra.x, o.extra.y, o.extra.z, 0.0f));
      } else {
        continue;
      }
      obj_mat.push_back(o.mat);
      obj_slot.push_back(i);
    }
  }
  sc->bvh_sphere_slots = obj_slot;
  sc->upload_linear_objects(ctx, spheres_in_bvh != 0);
  int n_obj = (int)oa.size();
  int n = sc->n_tris + n_obj;
  if (n <= 0) return RX_OK;
  DevBuf<float4> d_oa(ctx, std::max(n_obj, 1)), d_ob(ctx, std::max(n_obj, 1));
  DevBuf<int> d_obj_mat(ctx, std::max(n_obj, 1)), d_obj_slot(ctx, std::max(n_obj, 1));
  if (!all_ok(d_oa, d_ob, d_obj_mat, d_obj_slot)) return set_error(ctx, "LBVH: out of device memory"), RX_ERR_CAPACITY;
  if (n_obj) {
    cudaMemcpyAsync(d_oa.p, oa.data(), sizeof(float4) * n_obj, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_ob.p, ob.data(), sizeof(float4) * n_obj, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_obj_mat.p, obj_mat.data(), sizeof(int) * n_obj, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_obj_slot.p, obj_slot.data(), sizeof(int) * n_obj, cudaMemcpyHostToDevice, st);
  }
  DevBuf<float3> pmin(ctx, n), pmax(ctx, n);
  DevBuf<int> order(ctx, n);
  if (int rc = front_end(ctx, sc, n_obj, d_oa.p, d_ob.p, 1, pmin, pmax, order)) return rc;
  sc->d_prims.alloc(ctx, (size_t)kPrimQuads * n);
  sc->d_shade.alloc(ctx, (size_t)3 * n);
  if (!all_ok(sc->d_prims, sc->d_shade)) {
    sc->clear_bvh();
    return set_error(ctx, "LBVH: out of device memory"), RX_ERR_CAPACITY;
  }
  launch_chained(st, true, dim3(grid_for(ctx, n)), 256, 0, k_gather_prims, n, order.p, sc->n_tris, sc->d_v0, sc->d_v1,
                 sc->d_v2, sc->d_n0, sc->d_n1, sc->d_n2, sc->d_tri_mat, d_oa.p, d_ob.p, d_obj_mat.p, d_obj_slot.p,
                 sc->d_prims.p, sc->d_shade.p);
  float4 hb[2];  // the root's box: the union of all primitives'
  int n_int = n - 1;
  DevBuf<int> at_lo;  // first sorted position under each laid-out node
  if (n == 1) {
    if (!sc->d_nodes.alloc(ctx, 4) || !at_lo.alloc(ctx, 1)) {
      sc->clear_bvh();
      return set_error(ctx, "LBVH: out of device memory"), RX_ERR_CAPACITY;
    }
    k_single_leaf_root<<<1, 1, 0, st>>>(pmin.p, pmax.p, 1, sc->d_nodes.p);
    CUDA_TRY(ctx, cudaMemcpyAsync(&hb[0], pmin.p, sizeof(float3), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(ctx, cudaMemcpyAsync(&hb[1], pmax.p, sizeof(float3), cudaMemcpyDeviceToHost, st));
    sc->n_nodes = 1;
  } else {
    DevBuf<int4> range(ctx, n_int);
    DevBuf<int> par_int(ctx, n_int), par_leaf(ctx, n), flags(ctx, n_int);
    DevBuf<float4> rec(ctx, (size_t)2 * n_int);
    MaskBuf m(ctx, n_int);
    DevBuf<int> info(ctx, 2);  // nodes laid out, levels
    sc->d_nodes.alloc(ctx, (size_t)4 * n_int);
    at_lo.alloc(ctx, n_int);
    if (!all_ok(sc->d_nodes, at_lo, range, par_int, par_leaf, flags, rec, m.mask, m.rank, m.counts, info)) {
      sc->clear_bvh();
      return set_error(ctx, "LBVH: out of device memory"), RX_ERR_CAPACITY;
    }
    launch_chained(st, true, dim3(grid_for(ctx, n_int)), 256, 0, k_karras, n, sc->tmp_codes.p, range.p, par_int.p,
                   par_leaf.p, flags.p, m.counts.p, m.blocks);
    launch_chained(st, true, dim3((n + kUpLeaves - 1) / kUpLeaves), kUpLeaves, 0, k_lbvh_bottom_up, n, order.p, range.p,
                   par_int.p, par_leaf.p, pmin.p, pmax.p, rec.p, flags.p, max_leaf, c_t, c_i);
    launch_chained(st, true, dim3((n_int + 255) / 256), 256, 0, k_lbvh_keep, n_int, range.p, par_int.p, rec.p,
                     max_leaf, m.view(), info.p + 1);
    launch_chained(st, true, dim3(m.blocks), kRankWords, 0, k_rank, m.view(), n_int, info.p);
    launch_chained(st, true, dim3(grid_for(ctx, n_int)), 256, 0, k_lbvh_layout, n_int, range.p, order.p, pmin.p, pmax.p,
                   rec.p, m.view(), sc->d_nodes.p, at_lo.p);
    CUDA_TRY(ctx, cudaGetLastError());
    int h_info[2] = {0, 0};
    CUDA_TRY(ctx, cudaMemcpyAsync(hb, rec.p, sizeof(hb), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(ctx, cudaMemcpyAsync(h_info, info.p, sizeof(h_info), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(ctx, cudaStreamSynchronize(st));
    sc->n_nodes = h_info[0];
    sc->depth = h_info[1];
    if (sc->n_nodes == 0) {  // the whole tree is one leaf
      k_single_leaf_root<<<1, 1, 0, st>>>(reinterpret_cast<const float3*>(rec.p),
                                          reinterpret_cast<const float3*>(rec.p + 1), n, sc->d_nodes.p);
      sc->n_nodes = 1;
    }
  }
  sc->order.swap(order);
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  if (int rc = build_wide(ctx, sc, at_lo.p)) {
    sc->clear_bvh();
    return rc;
  }
  sc->root_min = f3(hb[0].x, hb[0].y, hb[0].z);
  sc->root_max = f3(hb[1].x, hb[1].y, hb[1].z);
  sc->n_prims = n;
  sc->n_bvh_spheres = n_obj;
  sc->method = RX_BVH_LBVH_SAH;
  sc->exact_slab = 0;
  sc->leaf_size = max_leaf;
  return RX_OK;
}

}  // namespace rx
