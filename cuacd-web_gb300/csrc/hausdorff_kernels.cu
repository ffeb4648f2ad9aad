// hausdorff_kernels.cu — bidirectional sampled Hausdorff distance of mesh
// pairs on sm_103a (the reference's src/gpu/hausdorff_shader.ts:13-153).
//
// Sampling rule (as the reference): res = max(1000, floor(2000 * area));
// each triangle gets floor(res / area * a_t) samples, or one on every
// step-th (or every even) triangle that gets none; barycentrics from a Wang
// hash of t * 65537 + k.
//
// The result of a pair is the largest, over the samples of both sides, of
// the smallest squared distance tri_sq(sample, triangle of the other side).
// Neither the order of the triangles nor that of the samples matters, and a
// sample or triangle that provably cannot decide it need not be looked at:
//   k_hd_prep   a block per mesh: areas, sample counts, the triangles in
//               Morton order of their centroids in clusters of 32 with
//               bounding boxes, and the samples' prefix in that order;
//   k_hd_tiles  the work list: 32 consecutive samples of a mesh each;
//   k_hd_near   a warp per 32 samples: the clusters whose box may hold a
//               nearest triangle, nearest box first, a centroid test per
//               triangle, tri_sq for the survivors; a sample whose distance
//               cannot exceed the pair's largest one so far is dropped. In a
//               target with slivers the samples that are left, and those
//               whose nearest triangle a sliver may rule out, go through its
//               triangles in order (hd_ordered).
// What bounds it: dependent loads and divergence in k_hd_near. Against a
// tensor-core bound of every sample-triangle pair, whose epilogue was bound by
// instruction issue: 24 cut halves of 1.5-30k triangles with their hulls
// 11.4 -> 1.48 ms, the 192 halves of 96 icosphere cuts 8.5 -> 0.83 ms, 192
// pairs of 160-6,000 triangles 5.8 + 0.71 -> 1.02 ms.
#include <cuda_bf16.h>

#include <algorithm>

#include "cuacd_dev.cuh"

namespace cuacd {

__device__ __forceinline__ uint32_t wang(uint32_t s) {
  s = (s ^ 61u) ^ (s >> 16);
  s = s * 9u;
  s = s ^ (s >> 4);
  s = s * 0x27d4eb2du;
  s = s ^ (s >> 15);
  return s;
}
__device__ __forceinline__ float tri_area(f3 a, f3 b, f3 c) {
  f3 n = cross(b - a, c - a);
  return 0.5f * sqrtf(dot(n, n));
}

// squared distance from p to triangle (a, b, c) (hausdorff_shader.ts:32-52)
__device__ __forceinline__ float seg_sq(f3 p, f3 a, f3 b) {
  const f3 ab = b - a, ap = p - a;
  const float ab2 = dot(ab, ab);
  float t = ab2 > 1e-20f ? dot(ap, ab) / ab2 : 0.0f;
  t = fminf(fmaxf(t, 0.0f), 1.0f);
  const f3 d = ap - t * ab;
  return dot(d, d);
}
__device__ __forceinline__ float tri_sq(f3 p, f3 a, f3 b, f3 c) {
  const f3 ab = b - a, ac = c - a, ap = p - a;
  const f3 n = cross(ab, ac);
  const float n2 = dot(n, n);
  if (n2 < 1e-20f) {
    const f3 bp = p - b, cp = p - c;
    return fminf(dot(ap, ap), fminf(dot(bp, bp), dot(cp, cp)));
  }
  const float d00 = dot(ab, ab), d01 = dot(ab, ac), d02 = dot(ab, ap);
  const float d11 = dot(ac, ac), d12 = dot(ac, ap);
  const float inv = 1.0f / (d00 * d11 - d01 * d01);
  const float u = (d11 * d02 - d01 * d12) * inv;
  const float v = (d00 * d12 - d01 * d02) * inv;
  if (u >= 0.0f && v >= 0.0f && u + v <= 1.0f) {
    const float dist = dot(n, ap);
    return (dist * dist) / n2;
  }
  return fminf(seg_sq(p, a, b), fminf(seg_sq(p, b, c), seg_sq(p, c, a)));
}

// the same as a call, for the few evaluations outside the search's loop:
// k_hd_near waits for instructions more than for anything else (5.8 of 12.1
// cycles an instruction in 83 KB of code, 2.7 of 9.4 in 72 KB), so the search
// has one copy of its visit and of tri_sq (55 KB)
__device__ __noinline__ float tri_sq_at(f3 p, const float4* g) { return tri_sq(p, xyz(g[0]), xyz(g[1]), xyz(g[2])); }

// ---------------------------------------------------------------------------
// prep

// threads of a prep block, and the triangles whose areas it computes between
// two barriers: warp 0 adds them while the other warps compute the next ones
#define HD_PREP 512u
#define HD_CHUNK ((HD_PREP - 32u) * 4u)
// Morton cells, 16 along the mesh's largest extent: a 60k-triangle surface
// occupies about 1,500 of them, so a cluster of 32 spans about one cell
#define HD_CELLS 4096u
static_assert(HD_CHUNK % 32 == 0 && 2 * HD_CHUNK <= HD_CELLS, "two area chunks share the cell counters' words");

__device__ __forceinline__ uint32_t spread4(uint32_t v) {
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}
__device__ __forceinline__ f3 centroid(f3 a, f3 b, f3 c) {
  return mk3((a.x + b.x + c.x) / 3.0f, (a.y + b.y + c.y) / 3.0f, (a.z + b.z + c.z) / 3.0f);
}
__device__ __forceinline__ void tri_load(const Dev& D, const PartDesc& pd, uint32_t t, f3& a, f3& b, f3& c) {
  const uint32_t* tr = D.T + pd.tOff + 3 * (size_t)t;
  const uint32_t i = tr[0], j = tr[1], k = tr[2];
  a = ldv(D.V, (size_t)pd.vOff + 3 * (size_t)i);
  b = ldv(D.V, (size_t)pd.vOff + 3 * (size_t)j);
  c = ldv(D.V, (size_t)pd.vOff + 3 * (size_t)k);
}
// inclusive scan over the block's HD_PREP threads; *total = the sum. The
// trailing barrier of the caller's loop separates two calls' use of ws.
__device__ __forceinline__ uint32_t prep_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t inc = warp_incl_u(v, lane);
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  const uint32_t x = lane < HD_PREP / 32 ? ws[lane] : 0u;
  const uint32_t xi = warp_incl_u(x, lane);
  *total = __shfl_sync(FULLMASK, xi, 31);
  const uint32_t before = __shfl_sync(FULLMASK, xi - x, w);
  __syncthreads();
  return before + inc;
}

// Areas of part descriptors [0, nMeshes) for the host, which turns them into
// sample capacities before a batch is sampled: per mesh the sum of the
// triangles' areas and a bound on how far that sum may be from the area in
// 64 bits. With u = 2^-24 an edge is off by u of its length, a cross product
// of edges ab, ac by 2u |ab||ac| through them and 2.9u |ab||ac| by its own
// rounding, its length by 3.5u more: at most 4.3u |ab||ac| per area, and 4e-23
// where squares underflow. The bound takes 3.2e-7 > 5u of |ab||ac| <= (|ab|^2 +
// |ac|^2) / 2. The host's serial sum of the same areas was 1.25 ms for the
// 370k triangles of 192 pairs and 1.88 ms for 192 halves of 96 icosphere
// cuts; this pass with its readback takes 0.04 ms, bound by its launch.
#define HD_AREA_TRIS 2048u
__global__ void __launch_bounds__(256) k_hd_area(const Dev D, double2* out) {
  const uint32_t m = blockIdx.x;
  const PartDesc pd = D.parts[m];
  double sum = 0.0, off = 0.0;
  for (uint32_t t0 = blockIdx.y * HD_AREA_TRIS; t0 < pd.nt; t0 += gridDim.y * HD_AREA_TRIS) {
    const uint32_t n = min(HD_AREA_TRIS, pd.nt - t0);
    for (uint32_t k = threadIdx.x; k < n; k += 256) {
      f3 a, b, c;
      tri_load(D, pd, t0 + k, a, b, c);
      sum += (double)tri_area(a, b, c);
      off += (double)(dot(b - a, b - a) + dot(c - a, c - a));
    }
  }
  sum = warp_sum_d(sum);
  off = warp_sum_d(off);
  if ((threadIdx.x & 31) == 0 && blockIdx.y * HD_AREA_TRIS < pd.nt) {
    atomicAdd(&out[m].x, sum);
    atomicAdd(&out[m].y, 1.6e-7 * off + 1e-22 * pd.nt);
  }
}

// One block per mesh. The total area is the double sum the sampling rule's
// counts were always made from: lane l of one warp adds the areas of
// triangles l, l + 32, ... in order and the lanes are folded in a tree, so
// the counts do not depend on the block's shape. That warp only adds, from
// shared memory; the gathers and square roots of the next chunk overlap it.
// 24 cut halves and their hulls, the largest about 40k triangles, take 0.40
// ms; one warp per mesh took 1.87 ms for the samples and a block of 256
// threads another 0.15 ms for the triangles' data.
__global__ void __launch_bounds__(HD_PREP) k_hd_prep(const HdArgs A, const Dev D) {
  __shared__ uint32_t cells[HD_CELLS];
  __shared__ uint32_t ws[32];
  __shared__ float box[6][HD_PREP / 32];
  __shared__ float sTotal;
  __shared__ uint32_t sBad;
  const uint32_t m = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const PartDesc pd = D.parts[A.partBase + m];
  const uint32_t nt = pd.nt, cap = A.capN[m];
  if (nt == 0) {
    if (tid == 0) A.ns[m] = 0;
    return;
  }
  uint32_t* cnt = A.cnt + A.triOff[m];
  uint32_t* soff = A.soff + A.triOff[m];
  uint32_t* perm = A.perm + A.triOff[m];
  // areas, their sum and the centroids' box
  {
    float* area = reinterpret_cast<float*>(cells);
    f3 lo = mk3(3.4e38f, 3.4e38f, 3.4e38f), hi = mk3(-3.4e38f, -3.4e38f, -3.4e38f);
    double sum = 0.0;
    uint32_t buf = 0;
    for (uint32_t c0 = 0; c0 < nt; c0 += HD_CHUNK, buf ^= HD_CHUNK) {
      if (warp > 0) {
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
          const uint32_t t = c0 + u * (HD_PREP - 32u) + tid - 32u;
          if (t < nt) {
            f3 a, b, c;
            tri_load(D, pd, t, a, b, c);
            const float ar = tri_area(a, b, c);
            area[buf + t - c0] = ar;
            cnt[t] = __float_as_uint(ar);
            const f3 g = centroid(a, b, c);
            lo = vmin3(lo, g);
            hi = vmax3(hi, g);
          }
        }
      }
      __syncthreads();
      if (warp == 0) {
        const uint32_t n = min(HD_CHUNK, nt - c0);
        for (uint32_t k = lane; k < n; k += 32) sum += (double)area[buf + k];
      }
    }
    if (warp == 0) {
      const float total = (float)warp_sum_d(sum);
      if (lane == 0) sTotal = total;
    }
    lo.x = warp_min_f(lo.x); lo.y = warp_min_f(lo.y); lo.z = warp_min_f(lo.z);
    hi.x = warp_max_f(hi.x); hi.y = warp_max_f(hi.y); hi.z = warp_max_f(hi.z);
    if (lane == 0) {
      box[0][warp] = lo.x; box[1][warp] = lo.y; box[2][warp] = lo.z;
      box[3][warp] = hi.x; box[4][warp] = hi.y; box[5][warp] = hi.z;
    }
    __syncthreads();
  }
  f3 lo = mk3(box[0][0], box[1][0], box[2][0]), hi = mk3(box[3][0], box[4][0], box[5][0]);
  for (uint32_t w = 1; w < HD_PREP / 32; w++) {
    lo = vmin3(lo, mk3(box[0][w], box[1][w], box[2][w]));
    hi = vmax3(hi, mk3(box[3][w], box[4][w], box[5][w]));
  }
  const float inv = 16.0f / fmaxf(fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z), 1e-30f);
  for (uint32_t k = tid; k < HD_CELLS; k += HD_PREP) cells[k] = 0;
  __syncthreads();
  // sample counts, cut off at the mesh's capacity in triangle order, and the
  // triangles' cells
  const float total = sTotal;
  float res = floorf(2000.0f * total);
  if (res < 1000.0f) res = 1000.0f;
  const uint32_t step = (float)nt > res ? nt / (uint32_t)res : 0;
  uint32_t run = 0;
  for (uint32_t c0 = 0; c0 < nt; c0 += 4 * HD_PREP) {
    uint32_t N[4], sum = 0;
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      const uint32_t t = c0 + 4 * tid + u;
      N[u] = 0;
      if (t < nt) {
        const float ta = __uint_as_float(cnt[t]);
        const uint32_t areaCount = total > 1e-20f ? (uint32_t)floorf((res / total) * ta) : 0u;
        if ((float)nt > res) N[u] = areaCount > 0 ? areaCount : ((t % max(step, 1u)) == 0 ? 1u : 0u);
        else N[u] = areaCount > 0 ? areaCount : ((t % 2u) == 0 ? 1u : 0u);
        f3 a, b, c;
        tri_load(D, pd, t, a, b, c);
        const f3 g = centroid(a, b, c);
        const uint32_t x = min((uint32_t)fmaxf((g.x - lo.x) * inv, 0.0f), 15u);
        const uint32_t y = min((uint32_t)fmaxf((g.y - lo.y) * inv, 0.0f), 15u);
        const uint32_t z = min((uint32_t)fmaxf((g.z - lo.z) * inv, 0.0f), 15u);
        const uint32_t code = spread4(x) | (spread4(y) << 1) | (spread4(z) << 2);
        soff[t] = code;
        atomicAdd(cells + code, 1u);
      }
      sum += N[u];
    }
    uint32_t tot;
    uint32_t at = run + prep_scan(sum, ws, &tot) - sum;
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      const uint32_t t = c0 + 4 * tid + u;
      if (t < nt) cnt[t] = at < cap ? min(N[u], cap - at) : 0u;
      at += N[u];
    }
    run += tot;
  }
  if (tid == 0) A.ns[m] = min(run, cap);
  __syncthreads();
  // counting sort by cell (the order within a cell does not matter)
  {
    constexpr uint32_t PER = HD_CELLS / HD_PREP;
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) sum += cells[PER * tid + k];
    uint32_t tot;
    uint32_t at = prep_scan(sum, ws, &tot) - sum;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) {
      const uint32_t v = cells[PER * tid + k];
      cells[PER * tid + k] = at;
      at += v;
    }
  }
  __syncthreads();
  for (uint32_t t = tid; t < nt; t += HD_PREP) perm[atomicAdd(cells + soff[t], 1u)] = t;
  __syncthreads();
  // the sorted triangles, the clusters' boxes and the samples' prefix
  const size_t base = A.triOff[m];
  run = 0;
  if (tid == 0) sBad = 0;
  __syncthreads();
  for (uint32_t c0 = 0; c0 < nt; c0 += 4 * HD_PREP) {
    const uint32_t i0 = c0 + 128 * warp + lane;
    uint32_t N[4], off[4], wsum = 0;
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      const uint32_t i = i0 + 32 * u;
      N[u] = 0;
      f3 blo = mk3(3.4e38f, 3.4e38f, 3.4e38f), bhi = mk3(-3.4e38f, -3.4e38f, -3.4e38f);
      bool sliver = false;
      if (i < nt) {
        const uint32_t t = perm[i];
        f3 a, b, c;
        tri_load(D, pd, t, a, b, c);
        N[u] = cnt[t];
        const f3 g = centroid(a, b, c);
        const float ra = sqrtf(dot(a - g, a - g)), rb = sqrtf(dot(b - g, b - g)), rc = sqrtf(dot(c - g, c - g));
        // radius rounded up past its float32 error
        float r = fmaxf(fmaxf(ra, rb), rc) * 1.00001f + 1e-30f;
        blo = vmin3(vmin3(a, b), c);
        bhi = vmax3(vmax3(a, b), c);
        // a triangle that is not finite is never culled (inf - inf and
        // NaN - NaN are NaN, which is not below 3.4e38)
        const float sumAbs = (l1(a) + l1(b)) + l1(c);
        if (!(sumAbs < 3.4e38f)) {
          r = INFINITY;
          blo = mk3(-INFINITY, -INFINITY, -INFINITY);
          bhi = mk3(INFINITY, INFINITY, INFINITY);
        }
        // a sliver (the angle at a below 0.57 degrees) or a degenerate
        // triangle: tri_sq may be far off its geometry (HdNear), so it is
        // marked by a negative radius
        const f3 ab = b - a, ac = c - a, nn = cross(ab, ac);
        const float n2 = dot(nn, nn);
        if (!(n2 > 1e-4f * dot(ab, ab) * dot(ac, ac)) || n2 < 1.1e-20f) {
          r = -r;
          sliver = true;
          A.bad[base + atomicAdd(&sBad, 1u)] = i;
        }
        cnt[t] = i;  // its samples have been read
        float4* G = A.triG + 3 * (base + i);
        G[0] = make_float4(a.x, a.y, a.z, 0.0f);
        G[1] = make_float4(b.x, b.y, b.z, 0.0f);
        G[2] = make_float4(c.x, c.y, c.z, 0.0f);
        A.triC[base + i] = make_float4(g.x, g.y, g.z, r);
      }
      if (i - lane < nt) {  // the warp's cluster holds a triangle
        const float4 l = make_float4(f_unord(__reduce_min_sync(FULLMASK, f_ord(blo.x))),
                                     f_unord(__reduce_min_sync(FULLMASK, f_ord(blo.y))),
                                     f_unord(__reduce_min_sync(FULLMASK, f_ord(blo.z))), 0.0f);
        const float4 h = make_float4(f_unord(__reduce_max_sync(FULLMASK, f_ord(bhi.x))),
                                     f_unord(__reduce_max_sync(FULLMASK, f_ord(bhi.y))),
                                     f_unord(__reduce_max_sync(FULLMASK, f_ord(bhi.z))), 0.0f);
        const bool has = __any_sync(FULLMASK, sliver);
        if (lane == 0) {
          float4* B = A.box + 2 * (size_t)((base + i) >> 5);
          B[0] = l;
          B[1] = make_float4(h.x, h.y, h.z, has ? 1.0f : 0.0f);
        }
      }
      const uint32_t inc = warp_incl_u(N[u], lane);
      off[u] = wsum + inc - N[u];
      wsum += __shfl_sync(FULLMASK, inc, 31);
    }
    uint32_t tot;
    // every lane holds its warp's total: scan the warps through lane 31's slot
    const uint32_t inc = prep_scan(lane == 31 ? wsum : 0u, ws, &tot);
    const uint32_t before = __shfl_sync(FULLMASK, inc, 31) - wsum;
#pragma unroll
    for (uint32_t u = 0; u < 4; u++)
      if (i0 + 32 * u < nt) soff[i0 + 32 * u] = run + before + off[u];
    run += tot;
  }
  if (tid == 0) A.slivers[m] = sBad;
  // a target with slivers: its triangles' centroids in their own order, with a
  // box and the largest radius per 32 (behind the last scan's barriers)
  if (sBad == 0 || nt < A.orderedMin) return;
  for (uint32_t t0 = 32 * warp; t0 < nt; t0 += HD_PREP) {
    const uint32_t t = t0 + lane;
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < nt) {
      c = A.triC[base + cnt[t]];
      A.triO[base + t] = c;
    }
    const int lo3 = f_ord(3.4e38f), hi3 = f_ord(-3.4e38f);
    const float4 l = make_float4(f_unord(__reduce_min_sync(FULLMASK, t < nt ? f_ord(c.x) : lo3)),
                                 f_unord(__reduce_min_sync(FULLMASK, t < nt ? f_ord(c.y) : lo3)),
                                 f_unord(__reduce_min_sync(FULLMASK, t < nt ? f_ord(c.z) : lo3)),
                                 __uint_as_float(__reduce_max_sync(FULLMASK, __float_as_uint(fabsf(c.w)))));
    const float4 h = make_float4(f_unord(__reduce_max_sync(FULLMASK, t < nt ? f_ord(c.x) : hi3)),
                                 f_unord(__reduce_max_sync(FULLMASK, t < nt ? f_ord(c.y) : hi3)),
                                 f_unord(__reduce_max_sync(FULLMASK, t < nt ? f_ord(c.z) : hi3)), 0.0f);
    if (lane == 0) {
      float4* B = A.boxO + 2 * (size_t)((base + t0) >> 5);
      B[0] = l;
      B[1] = h;
    }
  }
}

// tiles of 32 samples per mesh: their prefix over the meshes, and the work
// counter
__global__ void __launch_bounds__(1024) k_hd_tiles(const HdArgs A, const Dev D) {
  __shared__ uint32_t ws[32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t run = 0;
  for (uint32_t c0 = 0; c0 < A.nMeshes; c0 += 1024) {
    const uint32_t m = c0 + tid;
    uint32_t n = 0;
    if (m < A.nMeshes) {
      const uint32_t dst = m < A.nPairs ? m + A.nPairs : m - A.nPairs;
      const bool both = D.parts[A.partBase + m].nt != 0 && D.parts[A.partBase + dst].nt != 0;
      n = both ? (A.ns[m] + 31) / 32 : 0u;
    }
    const uint32_t inc = warp_incl_u(n, lane);
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    const uint32_t x = ws[lane];
    const uint32_t xi = warp_incl_u(x, lane);
    const uint32_t before = __shfl_sync(FULLMASK, xi - x, w);
    if (m < A.nMeshes) A.tilePre[m] = run + before + inc - n;
    run += __shfl_sync(FULLMASK, xi, 31);
    __syncthreads();
  }
  if (tid == 0) {
    A.tilePre[A.nMeshes] = run;
    *A.work = 0;
  }
}

// ---------------------------------------------------------------------------
// nearest triangles

#define HD_NEAR 128u
// slivers of a target that a sample asks one by one before it goes through the
// target in order: 32 steps of a warp, about what the pass takes. With it 192
// pairs take 1.02 ms, without 1.14; 24 cut halves 1.48 and 1.66; 192 icosphere
// halves 0.83 and 0.98. Parts cut 30 times have more slivers than that.
#define HD_FEW 1024u

// A sample's state in the culled search. best is the smallest tri_sq so far;
// ub bounds the tri_sq of some triangle from above by its centroid's distance
// (a centroid is a point of its triangle). The search keeps a triangle unless
// its bound |p - c| - r, or its cluster's box, is farther than reach(): the
// smaller of the two with a 1e-3 relative margin, and an absolute one of
// 3e-10 |p|^2 for distances that cancel far from the origin (coordinates
// round to 2^-24 of |p|, so squared distances below (1e-3 |p|)^2 may be off by
// 1e-3 of themselves).
//
// Both bounds hold for tri_sq as it is computed when the angle at a, which its
// barycentrics and its normal are formed from, has a sine s >= 0.01: the
// normal's direction is within about 2^-23 / s, so a plane distance is off
// by at most 1e-5 |p - a|, which ub's margin of 2 % and 1e-7 r^2 covers (|p -
// a| <= |p - c| + r); and the barycentrics are off by at most 2^-24 |p - a| /
// s^2 in length, so a point taken for one above the triangle lies within 6e-4
// |p - a| of it, 4e-7 of the squared distance. For a sliver the normal can
// be noise and the plane distance anything, and a triangle with |n|^2 < 1e-20
// counts by its corners alone: such triangles give no ub here. In a target
// below A.orderedMin triangles every one counts, as in an exhaustive search;
// in a larger one what counts is decided in the triangles' order (HdReach,
// hd_ordered). Parts that have been cut again and again are mostly slivers, and
// with every one counted the noise of far ones made the distances of 9 parts
// in 90 decompositions up to 32 % smaller than they are in 64 bits. Either way
// the distance does not depend on the order in which the tiles run.
struct HdNear {
  f3 p;
  float p2, best, ub;
  // the smallest |p - c|^2 of the slivers met, and the sorted numbers of that
  // sliver and of the triangles that gave best and ub
  float sliver;
  uint32_t atSliver, atBest, atUb;
  __device__ __forceinline__ float reach() const { return fminf(best, ub) * 1.001f + 3e-10f * p2 + 1e-30f; }
  // whether the sample can still raise the pair's largest distance
  __device__ __forceinline__ bool counts(float gmax) const { return best > gmax && !(ub + 3e-9f * p2 < gmax); }
  // for a sample that cannot: the triangle that shows it, and its lower bound
  __device__ __forceinline__ uint32_t shows(float gmax) const { return best > gmax ? atUb : atBest; }
  __device__ __forceinline__ float lower(float4 c) const {
    const f3 d = p - mk3(c.x, c.y, c.z);
    const float lo = sqrtf(dot(d, d)) - fabsf(c.w);
    return lo > 0.0f ? lo * lo : 0.0f;
  }
  __device__ __forceinline__ void meet(float d2, uint32_t i) {
    if (d2 < sliver) {
      sliver = d2;
      atSliver = i;
    }
  }
};

// What counts in a target with slivers, of at least A.orderedMin triangles: what
// a search of the triangles in order, 32 at a time, lets through by their
// centroids. With a margin e of 2^-13 (|p|^2 + |c|^2 + 2 |p|_1 |c|_1) on squared
// centroid distances, a triangle counts when its bound (sqrt(|p - c|^2 - e) -
// r)^2 is not above the smallest tri_sq of the 32s before and not above the
// smallest |p - c|^2 + e up to its own. Of ordinary triangles alone, one that
// is out of reach is not the nearest; but a sliver's tri_sq can lie on either
// side of its bounds, so it decides what comes after it, and the rule is one
// of values: |p - c|^2 is |p|^2 - 2 p.c + |c|^2 with p, -2c and |c|^2 taken to
// two bfloat16 terms each, as a bfloat16 contraction forms it (up to 6.5e-5
// |p|_1 |c|_1 from the plain one, which settled one of 70 halves of a mesh cut
// 30 times differently).
__device__ __forceinline__ float bf16_two(float x) {
  const float hi = __bfloat162float(__float2bfloat16_rn(x));
  return hi + __bfloat162float(__float2bfloat16_rn(x - hi));  // exact: within 24 bits
}
__device__ __forceinline__ f3 bf16_two(f3 v) { return mk3(bf16_two(v.x), bf16_two(v.y), bf16_two(v.z)); }
struct HdReach {
  float lb, ub, slack;
  // pt: the point to two terms
  __device__ __forceinline__ HdReach(f3 pt, float p2, float p1, float4 c4) {
    const f3 c = mk3(c4.x, c4.y, c4.z);
    const float c2 = dot(c, c), e = 1.220703125e-4f * (p2 + c2 + 2.0f * p1 * l1(c));
    const float q = p2 + (dot(pt, bf16_two(-2.0f * c)) + bf16_two(c2));
    const float lo = sqrtf(fmaxf(q - e, 0.0f)) - fabsf(c4.w);
    lb = lo > 0.0f ? lo * lo : 0.0f;
    ub = q + e;
    slack = 1e-10f * (p2 + c2) + 1e-30f;
  }
  __device__ __forceinline__ bool within(float bound) const { return lb <= bound * 1.001f + slack; }
};

__device__ __forceinline__ float warp_box_min(float v) { return f_unord(__reduce_min_sync(FULLMASK, f_ord(v))); }
__device__ __forceinline__ float warp_box_max(float v) { return f_unord(__reduce_max_sync(FULLMASK, f_ord(v))); }
// squared gap between two boxes (0 where they overlap)
__device__ __forceinline__ float box_gap(f3 alo, f3 ahi, float4 blo, float4 bhi) {
  const float dx = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x), 0.0f);
  const float dy = fmaxf(fmaxf(blo.y - ahi.y, alo.y - bhi.y), 0.0f);
  const float dz = fmaxf(fmaxf(blo.z - ahi.z, alo.z - bhi.z), 0.0f);
  return dx * dx + dy * dy + dz * dz;
}

// One warp: the smallest tri_sq of the triangles that count for the point p, or
// any value not above gmax once it is known not to be. 32 triangles are passed
// over when the box of their centroids and their largest radius put every lower
// bound above the smallest distance and upper bound so far: then none counts, and
// no upper bound is smaller. (e is at least 3.7 times what |p - c|^2 is off
// by, so 1.5 e and the margins below cover both.) What bounds it: dependent
// loads, 1,024 triangles a step where all are passed over. Every sliver
// against every sample in turn, 1,200 cycles a sliver, took 740 ms for 96
// unions of parts cut 30 times with their hulls (1.3 M triangles, two thirds
// slivers); this takes 12 ms, and the tensor-core bound took 43.
__device__ __noinline__ float hd_ordered(const float4* O, const float4* B, const float4* G, const uint32_t* at,
                                         uint32_t tnt, f3 p, float gmax, uint32_t& exact, uint32_t& met) {
  const uint32_t lane = threadIdx.x & 31;
  const float p2 = dot(p, p), p1 = l1(p);
  const f3 pt = bf16_two(p);
  const uint32_t nb = (tnt + 31) / 32;
  float best = 3.4e38f, up = 3.4e38f;
  uint32_t nExact = 0, nMet = 0;
  for (uint32_t g0 = 0; g0 < nb; g0 += 32) {
    const uint32_t g = g0 + lane;
    float lb = 0.0f, slack = 0.0f;
    if (g < nb) {
      const float4 l = B[2 * g], h = B[2 * g + 1];
      const f3 c = mk3(fmaxf(fabsf(l.x), fabsf(h.x)), fmaxf(fabsf(l.y), fabsf(h.y)), fmaxf(fabsf(l.z), fabsf(h.z)));
      const float c2 = dot(c, c), e = 1.83e-4f * (p2 + c2 + 2.0f * p1 * l1(c));
      const float lo = sqrtf(fmaxf(0.9999f * box_gap(p, p, l, h) - e, 0.0f)) - 1.0001f * l.w;
      lb = lo > 0.0f ? lo * lo : 0.0f;
      slack = 1.1e-10f * (p2 + c2) + 2e-30f;
    }
    auto near = [&]() { return g < nb && !(lb > fminf(best, up) * 1.0011f + slack); };
    unsigned todo = __ballot_sync(FULLMASK, near());
    while (todo) {
      const uint32_t j = __ffs(todo) - 1;
      const uint32_t t = 32 * (g0 + j) + lane;
      float lbT = 3.4e38f, ubT = 3.4e38f, slackT = 0.0f;
      uint32_t i = 0;
      if (t < tnt) {
        i = at[t];
        const HdReach R(pt, p2, p1, O[t]);
        lbT = R.lb;
        ubT = fminf(ubT, R.ub);
        slackT = R.slack;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(FULLMASK, ubT, o);
        if ((int)lane >= o) ubT = fminf(ubT, u);
      }
      ubT = fminf(ubT, up);  // the smallest upper bound up to the lane's triangle
      float v = 3.4e38f;
      if (t < tnt && lbT <= fminf(best, ubT) * 1.001f + slackT) {
        v = fminf(v, tri_sq_at(p, G + 3 * (size_t)i));
        nExact++;
      }
      nMet += 32;
      up = __shfl_sync(FULLMASK, ubT, 31);
      best = fminf(best, __uint_as_float(__reduce_min_sync(FULLMASK, __float_as_uint(v))));
      if (best <= gmax) break;
      todo = __ballot_sync(FULLMASK, near()) & ~((2u << j) - 1u);
    }
    if (best <= gmax) break;
  }
  exact = nExact;
  met = nMet;
  return best;
}

// Warps take tiles of 32 samples from the work list. Targets below
// A.screenMin triangles are searched exhaustively; for them the sort's boxes
// save nothing that the extra steps do not cost. Seven blocks an SM: 192 halves
// of 96 icosphere cuts 0.83 ms and 24 cut halves 1.48, with six 0.86 and 1.45.
__global__ void __launch_bounds__(HD_NEAR, 7) k_hd_near(const HdArgs A, const Dev D) {
  __shared__ float4 sCent[HD_NEAR / 32][32];
  const uint32_t lane = threadIdx.x & 31;
  float4* cent = sCent[threadIdx.x >> 5];
  const uint32_t nTiles = A.tilePre[A.nMeshes];
  unsigned long long nExact = 0, nScreen = 0;
  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(A.work, 1u);
    it = __shfl_sync(FULLMASK, it, 0);
    if (it >= nTiles) break;
    // the tile's mesh
    uint32_t m = 0, mEnd = A.nMeshes;
    while (mEnd - m > 1) {
      const uint32_t mid = (m + mEnd) >> 1;
      if (A.tilePre[mid] <= it) m = mid;
      else mEnd = mid;
    }
    const uint32_t pair = m < A.nPairs ? m : m - A.nPairs;
    const uint32_t dst = m < A.nPairs ? m + A.nPairs : pair;
    const uint32_t ns = A.ns[m], s0 = 32 * (it - A.tilePre[m]);
    const uint32_t tnt = D.parts[A.partBase + dst].nt;
    const size_t tb = A.triOff[dst];
    bool active = s0 + lane < ns;
    HdNear S;
    {
      // the lane's sample (past the end, the last one again: it takes part
      // in the tile's box only): its triangle is the last whose prefix
      // does not exceed it
      const uint32_t s = min(s0 + lane, ns - 1);
      const size_t sb = A.triOff[m];
      const uint32_t* soff = A.soff + sb;
      uint32_t i = 0, iEnd = D.parts[A.partBase + m].nt;
      while (iEnd - i > 1) {
        const uint32_t mid = (i + iEnd) >> 1;
        if (soff[mid] <= s) i = mid;
        else iEnd = mid;
      }
      const uint32_t t = A.perm[sb + i], k = s - soff[i];
      const float4 a4 = A.triG[3 * (sb + i)], b4 = A.triG[3 * (sb + i) + 1], c4 = A.triG[3 * (sb + i) + 2];
      const f3 pa = xyz(a4), pb = xyz(b4), pc = xyz(c4);
      const uint32_t ha = wang(t * 65537u + k);
      const uint32_t hb = wang(ha + 0x9e3779b9u);
      const float ra = (float)(ha & 0xFFFFFFu) / (float)0xFFFFFFu;
      const float rb = (float)(hb & 0xFFFFFFu) / (float)0xFFFFFFu;
      const float sqa = sqrtf(ra);
      S.p = ((1.0f - sqa) * pa + (sqa * (1.0f - rb)) * pb) + (sqa * rb) * pc;
    }
    uint32_t* gmaxAt = D.ctr + CTR_HD + pair;
    const float4* G = A.triG + 3 * tb;
    if (tnt < A.screenMin) {
      float best = 1e30f;
      for (uint32_t t = 0; t < tnt; t++) {
        const float4 a = G[3 * t], b = G[3 * t + 1], c = G[3 * t + 2];
        best = fminf(best, tri_sq(S.p, xyz(a), xyz(b), xyz(c)));
      }
      const uint32_t worst = __reduce_max_sync(FULLMASK, active ? __float_as_uint(best) : 0u);
      if (lane == 0) atomicMax(gmaxAt, worst);
      continue;
    }
    S.p2 = dot(S.p, S.p);
    // a small target's search starts where the exhaustive one does
    S.best = tnt < A.orderedMin ? 1e30f : 3.4e38f;
    S.ub = S.sliver = 3.4e38f;
    S.atSliver = S.atBest = S.atUb = 0;
    const uint32_t slivers = A.slivers[dst];
    const bool ordered = slivers != 0 && tnt >= A.orderedMin;
    uint32_t why = 0;  // of a sample dropped: the triangle that shows why
    auto settle = [&](float gmax) {
      if (active && !S.counts(gmax)) {
        active = false;
        why = S.shows(gmax);
      }
    };
    const float4* C = A.triC + tb;
    const float4* B = A.box + 2 * (tb >> 5);
    const uint32_t nc = (tnt + 31) / 32;
    // one cluster against the active samples
    auto visit = [&](uint32_t c) {
      const uint32_t cn = min(32u, tnt - 32 * c);
      __syncwarp();
      cent[lane] = lane < cn ? C[32 * c + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      __syncwarp();
      const float gmax = __uint_as_float(__ldcg(gmaxAt));
      // the nearest centroid, its triangle first
      float dmin = 3.4e38f;
      uint32_t jmin = 0;
      for (uint32_t j = 0; j < cn; j++) {
        const float4 g = cent[j];
        const f3 d = S.p - mk3(g.x, g.y, g.z);
        const float d2 = dot(d, d);
        if (d2 < dmin && g.w >= 0.0f) { dmin = d2; jmin = j; }
      }
      const float rmin = cent[jmin].w, ubMin = dmin * 1.02f + 1e-7f * rmin * rmin;
      if (dmin < 3.4e38f && ubMin < S.ub) {
        S.ub = ubMin;
        S.atUb = 32 * c + jmin;
      }
      settle(gmax);
      unsigned of = ordered ? __ballot_sync(FULLMASK, cent[lane].w < 0.0f) : 0u;
      while (of) {
        const uint32_t j = __ffs(of) - 1;
        of &= of - 1;
        const f3 d = S.p - xyz(cent[j]);
        S.meet(dot(d, d), 32 * c + j);
      }
      const unsigned any = __ballot_sync(FULLMASK, active);
      nScreen += (unsigned long long)__popc(any) * cn;  // the same on every lane
      if (any == 0) return;
      // pass 0: the nearest centroid's; pass 1: those within reach then
      uint32_t keep = active && dmin < 3.4e38f ? 1u << jmin : 0u;
      float rs = 3.4e38f;
#pragma unroll 1
      for (int pass = 0; pass < 2; pass++) {
        if (pass) {
          if (__ballot_sync(FULLMASK, active) == 0) return;
          rs = sqrtf(S.reach());
          keep = 0;
          for (uint32_t j = 0; j < cn; j++) {
            const float4 g = cent[j];
            const f3 d = S.p - mk3(g.x, g.y, g.z);
            const float q = rs + fabsf(g.w);
            if (!(dot(d, d) > q * q * 1.00001f) && !(ordered && g.w < 0.0f)) keep |= 1u << j;
          }
          if (dmin < 3.4e38f) keep &= ~(1u << jmin);
          if (!active) keep = 0;
        }
        while (keep) {
          const uint32_t j = __ffs(keep) - 1;
          keep &= keep - 1;
          const float4 m = cent[j];
          const f3 d = S.p - mk3(m.x, m.y, m.z);
          const float q = rs + fabsf(m.w);
          if (dot(d, d) > q * q * 1.00001f) continue;
          const float4* g = G + 3 * (size_t)(32 * c + j);
          const float4 a = g[0], b = g[1], cc = g[2];
          const float v = tri_sq(S.p, xyz(a), xyz(b), xyz(cc));
          if (v < S.best) {
            S.best = v;
            S.atBest = 32 * c + j;
          }
          nExact++;
          settle(gmax);
          if (!active) break;
          if (pass) rs = sqrtf(S.reach());
        }
      }
      __syncwarp();
    };
    // the tile's box and the cluster whose box is nearest to its centre
    f3 wlo = mk3(warp_box_min(S.p.x), warp_box_min(S.p.y), warp_box_min(S.p.z));
    f3 whi = mk3(warp_box_max(S.p.x), warp_box_max(S.p.y), warp_box_max(S.p.z));
    uint32_t first = 0;
    {
      const f3 ctr = 0.5f * (wlo + whi);
      uint32_t bk = 0xffffffffu, bc = 0;
      for (uint32_t c = lane; c < nc; c += 32) {
        const float4 l = B[2 * c], h = B[2 * c + 1];
        const float dx = 0.5f * (l.x + h.x) - ctr.x, dy = 0.5f * (l.y + h.y) - ctr.y, dz = 0.5f * (l.z + h.z) - ctr.z;
        const float v = box_gap(ctr, ctr, l, h) + 1e-2f * (dx * dx + dy * dy + dz * dz);
        const uint32_t k = v >= 0.0f ? __float_as_uint(v) : 0u;
        if (k < bk) { bk = k; bc = c; }
      }
      const uint32_t k = __reduce_min_sync(FULLMASK, bk);
      first = __reduce_min_sync(FULLMASK, bk == k ? bc : 0xffffffffu);
    }
    // the nearest cluster, then those that the samples left may need: the
    // nearest box of 32 boxes first
    float reach = 0.0f, gap = 0.0f;
    unsigned act = 0;
    bool need = false;
    for (uint32_t c = first, c0 = 0xffffffe0u; c != 0xffffffffu;) {
      visit(c);
      const unsigned left = __ballot_sync(FULLMASK, active);
      if (left != act) {  // the box of the samples left
        act = left;
        if (act == 0) break;
        const float inf = INFINITY;
        wlo = mk3(warp_box_min(active ? S.p.x : inf), warp_box_min(active ? S.p.y : inf), warp_box_min(active ? S.p.z : inf));
        whi = mk3(warp_box_max(active ? S.p.x : -inf), warp_box_max(active ? S.p.y : -inf), warp_box_max(active ? S.p.z : -inf));
      }
      reach = __uint_as_float(__reduce_max_sync(FULLMASK, active ? __float_as_uint(S.reach()) : 0u));
      need = need && !(gap > reach);
      for (c = 0xffffffffu; c == 0xffffffffu;) {
        if (__ballot_sync(FULLMASK, need) == 0) {
          c0 += 32;
          if (c0 >= nc) break;
          const uint32_t n = c0 + lane;
          if (n < nc && n != first) {
            gap = box_gap(wlo, whi, B[2 * n], B[2 * n + 1]);
            need = !(gap > reach);
          }
          continue;
        }
        const uint32_t key = need ? __float_as_uint(gap) : 0xffffffffu;
        const uint32_t k = __reduce_min_sync(FULLMASK, key);
        const uint32_t j = __ffs(__ballot_sync(FULLMASK, key == k && need)) - 1;
        if (lane == j) need = false;
        const float4 l = B[2 * (c0 + j)], h = B[2 * (c0 + j) + 1];
        if (__any_sync(FULLMASK, active && !(box_gap(S.p, S.p, l, h) > S.reach()))) c = c0 + j;
      }
    }
    if (ordered) {
      // A dropped sample stays dropped unless a sliver's upper bound may be
      // below the lower bound of the triangle u that dropped it, which then may
      // not count. The sliver whose centroid is nearest is the one to ask: no
      // upper bound of another sliver is below its lower bound, so either it
      // counts, or something nearer than u does. The clusters that the search
      // did not need are looked at for it.
      settle(__uint_as_float(__ldcg(gmaxAt)));
      const bool dropped = s0 + lane < ns && !active;
      const float shown = dropped ? S.lower(C[why]) : 0.0f;
      const float far = __uint_as_float(__reduce_max_sync(FULLMASK, dropped ? __float_as_uint(shown) : 0u));
      if (far > 0.0f) {
        const float inf = INFINITY;
        const bool d = dropped;
        wlo = mk3(warp_box_min(d ? S.p.x : inf), warp_box_min(d ? S.p.y : inf), warp_box_min(d ? S.p.z : inf));
        whi = mk3(warp_box_max(d ? S.p.x : -inf), warp_box_max(d ? S.p.y : -inf), warp_box_max(d ? S.p.z : -inf));
        for (uint32_t c0 = 0; c0 < nc; c0 += 32) {
          const uint32_t c = c0 + lane;
          bool need = false;
          if (c < nc) {
            const float4 l = B[2 * c], h = B[2 * c + 1];
            need = h.w != 0.0f && !(box_gap(wlo, whi, l, h) >= far);
          }
          unsigned todo = __ballot_sync(FULLMASK, need);
          while (todo) {
            const uint32_t k = c0 + __ffs(todo) - 1;
            todo &= todo - 1;
            const bool open = dropped && !(box_gap(S.p, S.p, B[2 * k], B[2 * k + 1]) >= fminf(shown, S.sliver));
            if (!__any_sync(FULLMASK, open)) continue;
            const float4 m = 32 * k + lane < tnt ? C[32 * k + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            unsigned of = __ballot_sync(FULLMASK, m.w < 0.0f);
            while (of) {
              const uint32_t j = __ffs(of) - 1;
              of &= of - 1;
              const f3 q = S.p - mk3(__shfl_sync(FULLMASK, m.x, j), __shfl_sync(FULLMASK, m.y, j),
                                     __shfl_sync(FULLMASK, m.z, j));
              S.meet(dot(q, q), 32 * k + j);
            }
          }
        }
      }
      bool open = dropped && shown > S.sliver;
      if (open) {
        open = !(tri_sq_at(S.p, G + 3 * (size_t)S.atSliver) <= __uint_as_float(__ldcg(gmaxAt)));
        nExact++;
      }
      // the others in the triangles' order, the one that is farthest first
      unsigned left = __ballot_sync(FULLMASK, active || open);
      while (left) {
        const uint32_t k = __reduce_max_sync(FULLMASK, ((left >> lane) & 1u) ? __float_as_uint(S.best) : 0u);
        const uint32_t l = __ffs(__ballot_sync(FULLMASK, ((left >> lane) & 1u) && __float_as_uint(S.best) == k)) - 1;
        left &= ~(1u << l);
        const float gmax = __uint_as_float(__ldcg(gmaxAt));
        if (__shfl_sync(FULLMASK, active && !S.counts(gmax) && !(S.lower(C[S.shows(gmax)]) > S.sliver), l)) continue;
        const f3 p = mk3(__shfl_sync(FULLMASK, S.p.x, l), __shfl_sync(FULLMASK, S.p.y, l), __shfl_sync(FULLMASK, S.p.z, l));
        // where no sliver is nearer than the nearest ordinary triangle, and none
        // rules that one out, it decides: nothing that counts is below it, so
        // neither a distance nor an ordinary triangle's upper bound puts it out
        // of reach. A few slivers are asked at once, a lane each
        float best = __shfl_sync(FULLMASK, S.best, l);
        bool plain = slivers <= HD_FEW &&
                     __shfl_sync(FULLMASK, active && !(S.lower(C[S.atBest]) > S.sliver), l);
        if (plain) {
          bool below = false;
          for (uint32_t k = lane; k < slivers; k += 32) {
            below = below || tri_sq_at(p, G + 3 * (size_t)A.bad[tb + k]) < best;
            nExact++;
          }
          plain = !__any_sync(FULLMASK, below);
        }
        uint32_t exact = 0, met = 0;
        if (!plain) best = hd_ordered(A.triO + tb, A.boxO + 2 * (tb >> 5), G, A.cnt + tb, tnt, p, gmax, exact, met);
        nExact += exact;
        nScreen += met;
        if (best > gmax && lane == 0) atomicMax(gmaxAt, __float_as_uint(best));
      }
      active = false;
    } else if (slivers != 0 && act) {
      // every sliver of a small target
      active = active && S.counts(__uint_as_float(__ldcg(gmaxAt)));
      for (uint32_t k = 0; k < slivers; k++) {
        if ((k & 31u) == 0 && __ballot_sync(FULLMASK, active) == 0) break;
        if (active) {
          S.best = fminf(S.best, tri_sq_at(S.p, G + 3 * (size_t)A.bad[tb + k]));
          nExact++;
        }
      }
    }
    const uint32_t worst = __reduce_max_sync(FULLMASK, active ? __float_as_uint(S.best) : 0u);
    if (lane == 0 && worst != 0) atomicMax(gmaxAt, worst);
  }
  for (int o = 16; o > 0; o >>= 1) nExact += __shfl_xor_sync(FULLMASK, nExact, o);
  if (lane == 0 && nScreen != 0) {
    add_bytes(D.ctr, CTR_HD_EXACT, nExact);
    add_bytes(D.ctr, CTR_HD_SCREENED, nScreen);
  }
}

void launch_hd_area(uint32_t nMeshes, uint32_t maxNt, const Dev& D, double2* out, cudaStream_t s) {
  if (nMeshes == 0 || maxNt == 0) return;
  k_hd_area<<<dim3(nMeshes, std::min(65535u, (maxNt - 1) / HD_AREA_TRIS + 1)), 256, 0, s>>>(D, out);
}

void launch_hd(const HdArgs& A, const Dev& D, int nSM, cudaStream_t s) {
  if (A.nPairs == 0) return;
  k_hd_prep<<<A.nMeshes, HD_PREP, 0, s>>>(A, D);
  k_hd_tiles<<<1, 1024, 0, s>>>(A, D);
  k_hd_near<<<nSM * 8, HD_NEAR, 0, s>>>(A, D);
}

}  // namespace cuacd
