// concave_kernels.cu — candidate cutting planes from concave mesh edges
// (src/cpu/concave.ts:25-92) on the GPU, for a batch of meshes.
//
// The planes are the host restatement's (csrc/host_mesh.cpp) bit for bit:
//   degree     one thread per directed edge: out-degree of every vertex; a
//              scan gives each vertex's edge list (the directed-edge CSR of
//              mesh.ts:79-98, each list in arbitrary order);
//   normals    one thread per face;
//   edges      one thread per directed edge v0 -> v1 with v1 > v0 that is the
//              lowest of its kind: the lowest face holding v1 -> v0, the
//              dihedral angle, the concave test, a count per v0; a scan of the
//              counts, and each concave edge's rank among v0's by v1 gives the
//              (v0, v1) order. A vertex of valence d costs d threads d steps
//              each; one thread per vertex took d^2 steps on the hub of a fan
//              (2.3 ms a launch in a decomposition of an 8k-triangle mesh);
//   reservoir  one warp per mesh: the reference's seeded LCG reservoir
//              (concave.ts:37-74) over the ordered concave edges, 32 draws at a
//              time up to the first that is taken, then two face-offset planes
//              and, unless the normals are nearly opposite, two bisector
//              planes per kept edge.
// Everything is double arithmetic on float32 inputs compiled with
// --fmad=false (the host restatement compiles without contraction); the
// dihedral angle uses CUDA's acos where the host uses the C library's: both
// are within an ulp, so only an edge whose dihedral lies within an ulp of
// the threshold could be classified differently.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/cuacd.h"
#include "concave_engine.h"
#include "dev_ptr.h"
#include "dev_scan.cuh"

#define CONC_NONE 0xffffffffu

namespace cuacd {
int set_error(int code, const char* msg);

namespace conc {

struct MeshDesc {
  uint32_t vOff, nv, tOff, nt;  // the mesh in the input pools
  uint32_t vBase, eBase;        // its ranges in the per-vertex and per-directed-edge scratch
  uint32_t seed, pad;
};

struct EdgeRec {
  uint32_t v0, v1, f0, f1;
};

__device__ __forceinline__ uint32_t find_seg(const uint32_t* __restrict__ pre, uint32_t n, uint32_t g) {
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void k_degree(const MeshDesc* __restrict__ M, const uint32_t* __restrict__ ePre, uint32_t nm, uint32_t total,
                         const uint32_t* __restrict__ T, uint32_t* __restrict__ deg) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const MeshDesc& m = M[find_seg(ePre, nm, g)];
  const uint32_t e = g - m.eBase;
  atomicAdd(deg + m.vBase + T[3 * (size_t)m.tOff + e], 1u);
}

// list entry: (destination vertex, directed edge 3 face + k); the lowest edge
// is on the lowest face
__global__ void k_fill(const MeshDesc* __restrict__ M, const uint32_t* __restrict__ ePre, uint32_t nm, uint32_t total,
                       const uint32_t* __restrict__ T, const uint32_t* __restrict__ off, uint32_t* __restrict__ fill,
                       uint2* __restrict__ list) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const MeshDesc& m = M[find_seg(ePre, nm, g)];
  const uint32_t e = g - m.eBase, t = e / 3, k = e % 3;
  const uint32_t* tri = T + 3 * ((size_t)m.tOff + t);
  const uint32_t a = tri[k], b = tri[(k + 1) % 3];
  const uint32_t at = atomicAdd(fill + m.vBase + a, 1u);
  list[off[m.vBase + a] + at] = make_uint2(b, e);
}

// unit normal of every face; zero when it has none
__global__ void k_normals(const MeshDesc* __restrict__ M, const uint32_t* __restrict__ ePre, uint32_t nm,
                          uint32_t total, const float* __restrict__ Vpool, const uint32_t* __restrict__ Tpool,
                          double* __restrict__ nrm) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;  // a face of the batch
  if (g >= total) return;
  const MeshDesc& m = M[find_seg(ePre, nm, 3 * g)];
  const float* V = Vpool + 3 * (size_t)m.vOff;
  const uint32_t* tri = Tpool + 3 * (size_t)g;
  const float* A = V + 3 * (size_t)tri[0];
  const float* B = V + 3 * (size_t)tri[1];
  const float* C = V + 3 * (size_t)tri[2];
  const double e1x = (double)B[0] - A[0], e1y = (double)B[1] - A[1], e1z = (double)B[2] - A[2];
  const double e2x = (double)C[0] - A[0], e2y = (double)C[1] - A[1], e2z = (double)C[2] - A[2];
  const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
  const double l = sqrt(nx * nx + ny * ny + nz * nz);
  const bool ok = !(l < 1e-12);
  nrm[3 * (size_t)g] = ok ? nx / l : 0.0;
  nrm[3 * (size_t)g + 1] = ok ? ny / l : 0.0;
  nrm[3 * (size_t)g + 2] = ok ? nz / l : 0.0;
}
__device__ __forceinline__ bool face_normal(const double* nrm, uint32_t f, double n[3]) {
  n[0] = nrm[3 * (size_t)f];
  n[1] = nrm[3 * (size_t)f + 1];
  n[2] = nrm[3 * (size_t)f + 2];
  return n[0] != 0.0 || n[1] != 0.0 || n[2] != 0.0;
}

// cosLo, cosHi: cosines of the dihedral angle's part beyond pi, thr - pi, with
// 1e-9 on either side (cosHi < cosLo when thr - pi is not in (0, pi)): outside
// them the concave test needs no acos, whose rounding and the sums' are
// below 1e-14
__global__ void k_edges(const MeshDesc* __restrict__ M, const uint32_t* __restrict__ ePre, uint32_t nm, uint32_t total,
                        const float* __restrict__ Vpool, const uint32_t* __restrict__ Tpool,
                        const uint32_t* __restrict__ off, const uint2* __restrict__ list,
                        const double* __restrict__ nrm, double thr, double cosLo, double cosHi,
                        EdgeRec* __restrict__ slots, uint32_t* __restrict__ cnt) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;  // a list entry
  if (g >= total) return;
  const MeshDesc& m = M[find_seg(ePre, nm, g)];
  const uint32_t* T = Tpool + 3 * (size_t)m.tOff;
  const uint2 en = list[g];
  const uint32_t v0 = T[en.y], v1 = en.x;
  EdgeRec r;
  r.v0 = CONC_NONE;
  r.v1 = r.f0 = r.f1 = 0;
  slots[g].v0 = CONC_NONE;
  if (v1 <= v0) return;
  // the lowest edge v0 -> v1, and the lowest v1 -> v0
  const uint32_t s0 = off[m.vBase + v0], s1 = off[m.vBase + v0 + 1];
  for (uint32_t k = s0; k < s1; k++) {
    const uint2 o = list[k];
    if (o.x == v1 && o.y < en.y) return;
  }
  uint32_t back = CONC_NONE;
  for (uint32_t k = off[m.vBase + v1]; k < off[m.vBase + v1 + 1]; k++) {
    const uint2 o = list[k];
    if (o.x == v0) back = min(back, o.y);
  }
  if (back == CONC_NONE) return;
  const uint32_t fa = en.y / 3, fb = back / 3;
  r.f0 = min(fa, fb);
  r.f1 = max(fa, fb);
  double n0[3], n1[3];
  const double* N = nrm + 3 * (size_t)m.tOff;
  if (!face_normal(N, r.f0, n0) || !face_normal(N, r.f1, n1)) return;
  uint32_t vOther = CONC_NONE;
  for (int i = 0; i < 3; i++) {
    const uint32_t vv = T[3 * (size_t)r.f0 + i];
    if (vv != v0 && vv != v1) {
      vOther = vv;
      break;
    }
  }
  if (vOther == CONC_NONE) return;
  const float* V = Vpool + 3 * (size_t)m.vOff;
  const double dx = (double)V[3 * (size_t)vOther] - V[3 * (size_t)v0];
  const double dy = (double)V[3 * (size_t)vOther + 1] - V[3 * (size_t)v0 + 1];
  const double dz = (double)V[3 * (size_t)vOther + 2] - V[3 * (size_t)v0 + 2];
  const double d = dx * n1[0] + dy * n1[1] + dz * n1[2];
  double cosA = n0[0] * n1[0] + n0[1] * n1[1] + n0[2] * n1[2];
  cosA = fmax(-1.0, fmin(1.0, cosA));
  bool concave;
  if (cosLo <= cosHi && (!(d > 0) || cosA < cosLo || cosA > cosHi)) {
    concave = d > 0 && cosA < cosLo;  // pi - alpha <= pi < thr
  } else {
    const double alpha = acos(cosA);
    const double dihedral = d > 0 ? M_PI + alpha : M_PI - alpha;
    concave = dihedral > thr;
  }
  if (!concave) return;
  r.v0 = v0;
  r.v1 = v1;
  slots[g] = r;
  atomicAdd(cnt + m.vBase + v0, 1u);
}

// every concave edge to its place: v0's first, plus its rank by v1
__global__ void k_place(const MeshDesc* __restrict__ M, const uint32_t* __restrict__ ePre, uint32_t nm, uint32_t total,
                        const uint32_t* __restrict__ off, const EdgeRec* __restrict__ slots,
                        const uint32_t* __restrict__ cpre, EdgeRec* __restrict__ ordered) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const EdgeRec r = slots[g];
  if (r.v0 == CONC_NONE) return;
  const MeshDesc& m = M[find_seg(ePre, nm, g)];
  const uint32_t v = m.vBase + r.v0;
  const uint32_t c0 = cpre[v], n = cpre[v + 1] - c0;
  uint32_t rank = 0;
  if (n > 1)
    for (uint32_t k = off[v]; k < off[v + 1]; k++) {
      const uint2 o = *reinterpret_cast<const uint2*>(slots + k);  // v0, v1
      rank += (o.x != CONC_NONE && o.y < r.v1) ? 1u : 0u;
    }
  ordered[c0 + rank] = r;
}

// One warp per mesh. The reference draws one LCG value per edge past the
// first nEdges, and a second one for an edge that it takes; between two taken
// edges the values are those of plain LCG steps, so the lanes form the next 32
// from the state by jumps and the first taken lane ends the batch. Taken
// edges are few (nEdges ln(n / nEdges)): a thread per mesh stepped through
// every edge, 0.51 ms for 16 meshes of up to 56k triangles; this takes 0.02.
__global__ void __launch_bounds__(32) k_reservoir(const MeshDesc* __restrict__ M, uint32_t nm,
                                                  const float* __restrict__ Vpool, const double* __restrict__ nrm,
                                                  const uint32_t* __restrict__ cpre,
                                                  const EdgeRec* __restrict__ ordered, int nEdges, double eps,
                                                  uint32_t* __restrict__ res, float* __restrict__ out,
                                                  int32_t* __restrict__ counts) {
  const uint32_t mi = blockIdx.x, lane = threadIdx.x;
  const MeshDesc& m = M[mi];
  uint32_t* rs = res + (size_t)mi * nEdges;  // the kept edges, by number
  float* o = out + (size_t)mi * 16 * nEdges;
  if (m.nt == 0 || nEdges <= 0) {
    if (lane == 0) counts[mi] = 0;
    return;
  }
  const uint32_t e0 = cpre[m.vBase], n = cpre[m.vBase + m.nv] - e0;
  const uint32_t nRes = min(n, (uint32_t)nEdges);
  for (uint32_t k = lane; k < nRes; k += 32) rs[k] = k;
  __syncwarp();
  // lane j: the state after j + 1 steps is mul * state + add
  uint32_t mul = 1664525u, add = 1013904223u;
  for (uint32_t j = 0; j < lane; j++) {
    add = add * 1664525u + 1013904223u;
    mul *= 1664525u;
  }
  uint32_t rng = m.seed;
  const float share = (float)nEdges * 4294967296.0f;
  for (uint32_t k0 = nRes; k0 < n;) {
    const uint32_t k = k0 + lane, x = rng * mul + add;
    bool take = false;
    if (k < n) {
      // the threshold within 1e-6 of itself in float32; the double
      // expression only beside it
      const float t = share / (float)(k + 1), f = (float)x;
      if (f < t * 1.00001f + 2.0f) {
        if (f < t * 0.99999f - 2.0f) take = true;
        else take = (double)x < floor((double)nEdges / (double)(k + 1) * 4294967295.0);
      }
    }
    const unsigned any = __ballot_sync(0xffffffffu, take);
    if (any) {
      const uint32_t j = __ffs(any) - 1;
      rng = __shfl_sync(0xffffffffu, x, j) * 1664525u + 1013904223u;
      if (lane == 0) rs[rng % (uint32_t)nEdges] = k0 + j;
      k0 += j + 1;
    } else {
      rng = __shfl_sync(0xffffffffu, x, 31);
      k0 += 32;
    }
  }
  __syncwarp();
  const float* V = Vpool + 3 * (size_t)m.vOff;
  const double* N = nrm + 3 * (size_t)m.tOff;
  uint32_t np = 0;
  for (uint32_t k0 = 0; k0 < nRes; k0 += 32) {
    const uint32_t k = k0 + lane;
    EdgeRec r;
    r.v0 = r.v1 = r.f0 = r.f1 = 0;
    double n0[3], n1[3], bx = 0, by = 0, bz = 0;
    uint32_t c = 0;
    if (k < nRes) {
      r = ordered[e0 + rs[k]];
      if (face_normal(N, r.f0, n0) && face_normal(N, r.f1, n1)) {
        bx = n0[0] + n1[0];
        by = n0[1] + n1[1];
        bz = n0[2] + n1[2];
        const double bl = sqrt(bx * bx + by * by + bz * bz);
        c = 2;
        if (bl >= 1e-4) {
          bx /= bl;
          by /= bl;
          bz /= bl;
          c = 4;
        }
      }
    }
    uint32_t inc = c;
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
      if ((int)lane >= d) inc += u;
    }
    if (c) {
      const double mx = ((double)V[3 * (size_t)r.v0] + V[3 * (size_t)r.v1]) / 2;
      const double my = ((double)V[3 * (size_t)r.v0 + 1] + V[3 * (size_t)r.v1 + 1]) / 2;
      const double mz = ((double)V[3 * (size_t)r.v0 + 2] + V[3 * (size_t)r.v1 + 2]) / 2;
      uint32_t at = np + inc - c;
      auto push = [&](double a, double b, double cc, double d) {
        o[4 * at] = (float)a;
        o[4 * at + 1] = (float)b;
        o[4 * at + 2] = (float)cc;
        o[4 * at + 3] = (float)d;
        at++;
      };
      push(n1[0], n1[1], n1[2], -(n1[0] * mx + n1[1] * my + n1[2] * mz + eps));
      push(n0[0], n0[1], n0[2], -(n0[0] * mx + n0[1] * my + n0[2] * mz + eps));
      if (c == 4) {
        push(bx, by, bz, -(bx * mx + by * my + bz * mz + eps));
        push(bx, by, bz, -(bx * mx + by * my + bz * mz - eps));
      }
    }
    np += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) counts[mi] = (int32_t)np;
}

// ---------------------------------------------------------------------------
// host side

struct Buf {
  void* p = nullptr;
  size_t bytes = 0;
  int ensure(size_t need) {
    if (need <= bytes) return 0;
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
    need = std::max<size_t>(need, 256);
    if (cudaMalloc(&p, need) != cudaSuccess) return set_error(CUACD_E_CUDA, "concave: device allocation failed");
    bytes = need;
    return 0;
  }
  template <typename T>
  T* as() const {
    return static_cast<T*>(p);
  }
  ~Buf() {
    if (p) cudaFree(p);
  }
};

struct Engine {
  Buf inV, inT, desc, ePre, deg, off, fill, list, nrm, slots, cnt, cpre, ordered, res, out, counts, tiles;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

Engine* engine_create() {
  Engine* e = new Engine();
  if (cudaEventCreate(&e->ev0) != cudaSuccess || cudaEventCreate(&e->ev1) != cudaSuccess) {
    delete e;
    return nullptr;
  }
  return e;
}

void engine_destroy(Engine* e) {
  if (!e) return;
  if (e->ev0) cudaEventDestroy(e->ev0);
  if (e->ev1) cudaEventDestroy(e->ev1);
  delete e;
}

size_t engine_device_bytes(const Engine* e) {
  if (!e) return 0;
  size_t n = 0;
  for (const Buf* b : {&e->inV, &e->inT, &e->desc, &e->ePre, &e->deg, &e->off, &e->fill, &e->list, &e->nrm, &e->slots,
                       &e->cnt, &e->cpre, &e->ordered, &e->res, &e->out, &e->counts, &e->tiles})
    n += b->bytes;
  return n;
}

#define CONCK(x)                                                                                 \
  do {                                                                                           \
    cudaError_t err_ = (x);                                                                      \
    if (err_ != cudaSuccess)                                                                     \
      return set_error(CUACD_E_CUDA, (std::string("concave: ") + #x + ": " + cudaGetErrorString(err_)).c_str()); \
  } while (0)

static inline uint32_t blocks(uint64_t n, uint32_t t) { return (uint32_t)std::max<uint64_t>(1, (n + t - 1) / t); }

int engine_run(Engine* e, cudaStream_t s, const cuacd_mesh* meshes, int nMeshes, int nConcaveEdges, double eps,
               double thr, const uint32_t* seeds, float* out, int32_t* counts, float* gpuMs) {
  if (!e || nMeshes < 0 || (nMeshes > 0 && (!meshes || !seeds || !out || !counts)))
    return set_error(CUACD_E_INVALID, "concave: invalid argument");
  if (gpuMs) *gpuMs = 0;
  if (nMeshes == 0) return CUACD_OK;
  const int nE = std::max(nConcaveEdges, 0);
  const uint32_t nm = (uint32_t)nMeshes;
  std::vector<MeshDesc> desc(nm);
  std::vector<uint32_t> ePre(nm + 1, 0);
  uint64_t totV = 0, totT = 0;
  for (uint32_t i = 0; i < nm; i++) {
    const cuacd_mesh& m = meshes[i];
    if ((m.nv && !m.verts) || (m.nt && !m.tris)) return set_error(CUACD_E_INVALID, "concave: null mesh buffer");
    // a device mesh is copied on the device and its indices are the
    // caller's to vouch for; a host mesh is checked
    const bool dv = is_device_ptr(m.verts), dt = is_device_ptr(m.tris);
    if ((m.nv && m.nt && dv != dt) || (!m.nv && dt) || (!m.nt && dv))
      return set_error(CUACD_E_INVALID, "concave: a mesh's buffers must both be host or both be device memory");
    if (!dt && !indices_below(m.tris, 3ull * m.nt, m.nv))
      return set_error(CUACD_E_INVALID, "concave: triangle index out of range");
    MeshDesc& d = desc[i];
    d.vOff = (uint32_t)totV;
    d.nv = m.nv;
    d.tOff = (uint32_t)totT;
    d.nt = nE > 0 ? m.nt : 0;  // no edges are looked at when no plane is asked for
    d.vBase = (uint32_t)totV;
    d.eBase = 3 * (uint32_t)totT;
    d.seed = seeds[i];
    d.pad = 0;
    totV += m.nv;
    totT += d.nt;
    ePre[i + 1] = 3 * (uint32_t)totT;
  }
  if (totV >= (1ull << 31) || 3 * totT >= (1ull << 31)) return set_error(CUACD_E_CAPACITY, "concave: batch too large");
  const uint64_t totE = 3 * totT;
  int rc;
  if ((rc = e->inV.ensure(12 * totV)) || (rc = e->inT.ensure(12 * totT)) || (rc = e->desc.ensure(sizeof(MeshDesc) * nm)) ||
      (rc = e->nrm.ensure(24 * totT)) || (rc = e->ePre.ensure(4 * (nm + 1))) || (rc = e->deg.ensure(4 * totV)) ||
      (rc = e->off.ensure(4 * (totV + 1))) || (rc = e->fill.ensure(4 * totV)) || (rc = e->list.ensure(8 * totE)) ||
      (rc = e->slots.ensure(sizeof(EdgeRec) * totE)) || (rc = e->cnt.ensure(4 * totV)) ||
      (rc = e->cpre.ensure(4 * (totV + 1))) || (rc = e->ordered.ensure(sizeof(EdgeRec) * totE)) ||
      (rc = e->res.ensure(4 * (size_t)nm * std::max(nE, 1))) ||
      (rc = e->out.ensure(64 * (size_t)nm * std::max(nE, 1))) || (rc = e->counts.ensure(4 * nm)) ||
      (rc = e->tiles.ensure(4 * (scan::tiles_for((uint32_t)totV) + 1))))
    return rc;
  CONCK(cudaEventRecord(e->ev0, s));
  for (uint32_t i = 0; i < nm; i++) {
    const cuacd_mesh& m = meshes[i];
    if (m.nv) CONCK(cudaMemcpyAsync(e->inV.as<float>() + 3 * (size_t)desc[i].vOff, m.verts, 12ull * m.nv, cudaMemcpyDefault, s));
    if (desc[i].nt)
      CONCK(cudaMemcpyAsync(e->inT.as<uint32_t>() + 3 * (size_t)desc[i].tOff, m.tris, 12ull * m.nt, cudaMemcpyDefault, s));
  }
  CONCK(cudaMemcpyAsync(e->desc.p, desc.data(), sizeof(MeshDesc) * nm, cudaMemcpyHostToDevice, s));
  CONCK(cudaMemcpyAsync(e->ePre.p, ePre.data(), 4 * (nm + 1), cudaMemcpyHostToDevice, s));
  if (totV) {
    CONCK(cudaMemsetAsync(e->deg.p, 0, 4 * totV, s));
    CONCK(cudaMemsetAsync(e->fill.p, 0, 4 * totV, s));
    CONCK(cudaMemsetAsync(e->cnt.p, 0, 4 * totV, s));
  }
  const MeshDesc* dM = e->desc.as<MeshDesc>();
  if (totE) k_degree<<<blocks(totE, 256), 256, 0, s>>>(dM, e->ePre.as<uint32_t>(), nm, (uint32_t)totE, e->inT.as<uint32_t>(),
                                                        e->deg.as<uint32_t>());
  scan::exclusive<uint32_t>(e->deg.as<uint32_t>(), (uint32_t)totV, e->off.as<uint32_t>(), e->tiles.as<uint32_t>(), s);
  if (totE) k_fill<<<blocks(totE, 256), 256, 0, s>>>(dM, e->ePre.as<uint32_t>(), nm, (uint32_t)totE, e->inT.as<uint32_t>(),
                                                      e->off.as<uint32_t>(), e->fill.as<uint32_t>(), e->list.as<uint2>());
  const double beyond = thr - M_PI;
  const bool cosines = beyond > 0 && beyond < M_PI;
  if (totE) {
    k_normals<<<blocks(totT, 256), 256, 0, s>>>(dM, e->ePre.as<uint32_t>(), nm, (uint32_t)totT, e->inV.as<float>(),
                                                e->inT.as<uint32_t>(), e->nrm.as<double>());
    k_edges<<<blocks(totE, 128), 128, 0, s>>>(dM, e->ePre.as<uint32_t>(), nm, (uint32_t)totE, e->inV.as<float>(),
                                              e->inT.as<uint32_t>(), e->off.as<uint32_t>(), e->list.as<uint2>(),
                                              e->nrm.as<double>(), thr, cosines ? std::cos(beyond) - 1e-9 : 1.0,
                                              cosines ? std::cos(beyond) + 1e-9 : -1.0, e->slots.as<EdgeRec>(),
                                              e->cnt.as<uint32_t>());
  }
  scan::exclusive<uint32_t>(e->cnt.as<uint32_t>(), (uint32_t)totV, e->cpre.as<uint32_t>(), e->tiles.as<uint32_t>(), s);
  if (totE) k_place<<<blocks(totE, 256), 256, 0, s>>>(dM, e->ePre.as<uint32_t>(), nm, (uint32_t)totE,
                                                       e->off.as<uint32_t>(), e->slots.as<EdgeRec>(),
                                                       e->cpre.as<uint32_t>(), e->ordered.as<EdgeRec>());
  k_reservoir<<<nm, 32, 0, s>>>(dM, nm, e->inV.as<float>(), e->nrm.as<double>(), e->cpre.as<uint32_t>(),
                                e->ordered.as<EdgeRec>(), nE, eps, e->res.as<uint32_t>(), e->out.as<float>(),
                                e->counts.as<int32_t>());
  CONCK(cudaGetLastError());
  CONCK(cudaMemcpyAsync(counts, e->counts.p, 4 * nm, cudaMemcpyDeviceToHost, s));
  if (nE > 0) CONCK(cudaMemcpyAsync(out, e->out.p, 64 * (size_t)nm * nE, cudaMemcpyDeviceToHost, s));
  CONCK(cudaEventRecord(e->ev1, s));
  CONCK(cudaStreamSynchronize(s));
  if (gpuMs) cudaEventElapsedTime(gpuMs, e->ev0, e->ev1);
  return CUACD_OK;
}

}  // namespace conc
}  // namespace cuacd
