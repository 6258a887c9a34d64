// fcdem_meshmap.cu -- the distance map of a closed triangle mesh: at every
// lattice vertex the distance to the closest point of the mesh, negative
// inside (the generalized winding number, the summed solid angles over 4 pi,
// above 1/2), and that closest point as the contact point -- what
// DistanceMapMesh::ComputeDistance (distancegridcgal.hpp:36-69) stores.
//
// Beyond a few triangles (kMeshFew) neither part looks at every pair of a lattice
// vertex and a triangle:
//
//   * closest point: the triangles are put in Morton order of their centroids
//     and cut into clusters of 32 with a bounding box each.  A warp takes a
//     4 x 4 x 2 brick of lattice vertices, starts from the distance to the
//     nearest cluster's first vertex, and evaluates the triangles of the
//     clusters whose box is not farther than what it has.  Of triangles at
//     the same distance the one that comes first in the caller's list counts,
//     as in a scan of that list;
//   * sign: the winding number of a mesh without boundary only changes across
//     its surface, and two neighbouring lattice vertices with no surface point
//     between them (one of them farther from the mesh than the lattice step)
//     have the same one.  Each vertex points to such a neighbour with a lower
//     index; the solid angles are summed at the vertices without one (the
//     roots, a thin shell around the surface) and the others take their
//     root's sign.  In a mesh with a boundary every vertex is a root, and where
//     the roots' list and the distances beside it (13 bytes per vertex) cannot be
//     had: a map needs no more device memory than its vertices and triangles.
//
// Both kernels are bound by instruction issue.  The 128-cell map of a torus
// mesh of 32,768 triangles, host work and the vertices' copy to the host
// included: 6.9 ms against 128 ms with every pair evaluated (closest points
// 3.3 ms, solid angles 2.8 ms, signs 0.35 ms); the same bits.  Replacing the
// solid angles of far clusters by those of their area vectors, with a rigorous
// bound of the error, gained nothing: the clusters are too wide for the bound.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fcdem_map.cuh"

namespace fcdem {
namespace {

// Closest point of triangle (a, b, c) to p: the region-based method of
// Ericson, Real-Time Collision Detection, section 5.1.5 (vertex, edge or face
// region from the barycentric signs).
__device__ __forceinline__ float3 closestOnTriangle(float3 p, float3 a, float3 b, float3 c) {
  const float3 ab = make_float3(b.x - a.x, b.y - a.y, b.z - a.z);
  const float3 ac = make_float3(c.x - a.x, c.y - a.y, c.z - a.z);
  const float3 ap = make_float3(p.x - a.x, p.y - a.y, p.z - a.z);
  auto dot = [](float3 u, float3 v) { return u.x * v.x + u.y * v.y + u.z * v.z; };
  auto lerp = [](float3 o, float3 d, float t) {
    return make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
  };
  const float d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0.0f && d2 <= 0.0f) return a;
  const float3 bp = make_float3(p.x - b.x, p.y - b.y, p.z - b.z);
  const float d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0.0f && d4 <= d3) return b;
  const float vc = d1 * d4 - d3 * d2;
  if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) return lerp(a, ab, d1 / (d1 - d3));
  const float3 cp = make_float3(p.x - c.x, p.y - c.y, p.z - c.z);
  const float d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0.0f && d5 <= d6) return c;
  const float vb = d5 * d2 - d1 * d6;
  if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) return lerp(a, ac, d2 / (d2 - d6));
  const float va = d3 * d6 - d5 * d4;
  if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
    const float3 bc = make_float3(c.x - b.x, c.y - b.y, c.z - b.z);
    return lerp(b, bc, (d4 - d3) / ((d4 - d3) + (d5 - d6)));
  }
  const float den = 1.0f / (va + vb + vc);
  const float v = vb * den, w = vc * den;
  return make_float3(a.x + ab.x * v + ac.x * w, a.y + ab.y * v + ac.y * w,
                     a.z + ab.z * v + ac.z * w);
}

// Solid angle of triangle (a, b, c) seen from p, signed by the triangle's
// orientation (Van Oosterom and Strackee, IEEE Trans. Biomed. Eng. 30, 1983).
__device__ __forceinline__ float solidAngle(float3 p, float3 a, float3 b, float3 c) {
  const float3 A = make_float3(a.x - p.x, a.y - p.y, a.z - p.z);
  const float3 B = make_float3(b.x - p.x, b.y - p.y, b.z - p.z);
  const float3 C = make_float3(c.x - p.x, c.y - p.y, c.z - p.z);
  const float la = sqrtf(A.x * A.x + A.y * A.y + A.z * A.z);
  const float lb = sqrtf(B.x * B.x + B.y * B.y + B.z * B.z);
  const float lc = sqrtf(C.x * C.x + C.y * C.y + C.z * C.z);
  const float det = A.x * (B.y * C.z - B.z * C.y) - A.y * (B.x * C.z - B.z * C.x) +
                    A.z * (B.x * C.y - B.y * C.x);
  const float den = la * lb * lc + (A.x * B.x + A.y * B.y + A.z * B.z) * lc +
                    (A.x * C.x + A.y * C.y + A.z * C.z) * lb +
                    (B.x * C.x + B.y * C.y + B.z * C.z) * la;
  return 2.0f * atan2f(det, den);
}


constexpr unsigned kCluster = 32;  // triangles per cluster

// A lattice of vx x vy x vz vertices at vmin + i * cs.
struct Lattice {
  int vx, vy, vz;
  float3 vmin;
  float cs;
};

__device__ __forceinline__ float3 latticePoint(const Lattice &L, int i, int j, int k) {
  return make_float3(vcoord(L.vmin.x, i, L.cs), vcoord(L.vmin.y, j, L.cs),
                     vcoord(L.vmin.z, k, L.cs));
}

// Morton code (10 bits an axis) of each triangle's centroid in the mesh box.
__global__ void __launch_bounds__(256)
kMeshKeys(const float4 *__restrict__ tri, unsigned nt, float3 lo, float3 scale,
          unsigned *__restrict__ key, unsigned *__restrict__ val) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const float4 a = __ldg(tri + 3 * t), b = __ldg(tri + 3 * t + 1), c = __ldg(tri + 3 * t + 2);
  auto axis = [](float x, float y, float z, float l, float s) {
    return (unsigned)fminf(fmaxf(((x + y + z) * (1.0f / 3.0f) - l) * s, 0.0f), 1023.0f);
  };
  key[t] = mortonSpread(axis(a.x, b.x, c.x, lo.x, scale.x)) |
           (mortonSpread(axis(a.y, b.y, c.y, lo.y, scale.y)) << 1) |
           (mortonSpread(axis(a.z, b.z, c.z, lo.z, scale.z)) << 2);
  val[t] = t;
}

// The triangles in sorted order, the caller's index in the first vertex's w,
// and each cluster's box (lower corner, upper corner).  One warp per cluster.
__global__ void __launch_bounds__(256)
kMeshClusters(const float4 *__restrict__ tri, const unsigned *__restrict__ order, unsigned nt,
              float4 *__restrict__ sorted, float4 *__restrict__ box) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
  if (t - lane >= nt) return;
  const float inf = __int_as_float(0x7f800000);
  float3 lo = make_float3(inf, inf, inf), hi = make_float3(-inf, -inf, -inf);
  if (t < nt) {
    const unsigned o = min(__ldg(order + t), nt - 1u);
    float4 v[3];
    bool finite = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v[c] = __ldg(tri + 3 * o + c);
      finite = finite && !inertPos(v[c]);
      lo = make_float3(fminf(lo.x, v[c].x), fminf(lo.y, v[c].y), fminf(lo.z, v[c].z));
      hi = make_float3(fmaxf(hi.x, v[c].x), fmaxf(hi.y, v[c].y), fmaxf(hi.z, v[c].z));
    }
    if (!finite) {  // never culled
      lo = make_float3(-inf, -inf, -inf);
      hi = make_float3(inf, inf, inf);
    }
    v[0].w = __uint_as_float(o);
    for (int c = 0; c < 3; ++c) sorted[3 * t + c] = v[c];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
  if (lane == 0) {
    box[2 * (t / kCluster)] = make_float4(lo.x, lo.y, lo.z, 0.0f);
    box[2 * (t / kCluster) + 1] = make_float4(hi.x, hi.y, hi.z, 0.0f);
  }
}

// Distance between two intervals (0 when they meet).
__device__ __forceinline__ float gap(float lo, float hi, float a, float b) {
  return fmaxf(fmaxf(lo - b, a - hi), 0.0f);
}

// Unsigned distance and closest point of every lattice vertex, one warp per
// 4 x 4 x 2 brick.  A cluster is left out only where its box is farther than
// a distance already reached plus `slack`, which covers the rounding of
// closestOnTriangle and of the box distances.
constexpr int kNearWarps = 4;
__global__ void __launch_bounds__(32 * kNearWarps)
kMeshNearest(float4 *__restrict__ vert, float *__restrict__ dist, Lattice L,
             const float4 *__restrict__ tri, unsigned nt, const float4 *__restrict__ box,
             float slack) {
  __shared__ float4 sTri[kNearWarps][3 * kCluster];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const int bx = (L.vx + 3) / 4, by = (L.vy + 3) / 4, bz = (L.vz + 1) / 2;
  const long long brick = (long long)blockIdx.x * kNearWarps + warp;
  if (brick >= (long long)bx * by * bz) return;  // whole warps leave
  const int i0 = 4 * (int)(brick % bx), j0 = 4 * (int)((brick / bx) % by),
            k0 = 2 * (int)(brick / ((long long)bx * by));
  const int i = i0 + (int)(lane & 3u), j = j0 + (int)((lane >> 2) & 3u), k = k0 + (int)(lane >> 4);
  const bool valid = i < L.vx && j < L.vy && k < L.vz;
  const float3 p = latticePoint(L, min(i, L.vx - 1), min(j, L.vy - 1), min(k, L.vz - 1));
  const float3 lo = latticePoint(L, i0, j0, k0);
  const float3 hi = latticePoint(L, min(i0 + 3, L.vx - 1), min(j0 + 3, L.vy - 1),
                                 min(k0 + 1, L.vz - 1));
  const float3 mid = make_float3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y),
                                 0.5f * (lo.z + hi.z));
  const unsigned clusters = (nt + kCluster - 1) / kCluster;
  // the first bound: the nearest of the clusters' first vertices, seen from
  // the brick's middle
  float near2 = 3.4e38f;
  unsigned nearest = 0u;
  for (unsigned c = lane; c < clusters; c += 32) {
    const float4 a = __ldg(tri + 3 * (size_t)c * kCluster);
    if (isinf(__ldg(&box[2 * c].x))) continue;  // a triangle that is not finite
    const float dx = a.x - mid.x, dy = a.y - mid.y, dz = a.z - mid.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 < near2) {
      near2 = d2;
      nearest = c;
    }
  }
  {
    const float own = near2;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      near2 = fminf(near2, __shfl_xor_sync(0xffffffffu, near2, o));
    const unsigned who = __ballot_sync(0xffffffffu, own == near2);
    nearest = __shfl_sync(0xffffffffu, nearest, who ? __ffs((int)who) - 1 : 0);
  }
  float bound;  // the closest point is no farther than this (plus slack)
  {
    const float dx = p.x - mid.x, dy = p.y - mid.y, dz = p.z - mid.z;
    bound = sqrtf(near2) + sqrtf(dx * dx + dy * dy + dz * dz);
  }
  float best = 3.4e38f;
  unsigned bestTri = 0xffffffffu;
  float3 bestCp = p;
  float4 *s = sTri[warp];
  // the closest points of one cluster's triangles
  auto evaluate = [&](unsigned c) {
    const unsigned t0 = c * kCluster, cnt = min(kCluster, nt - t0);
    __syncwarp();
    for (unsigned e = lane; e < 3 * cnt; e += 32) s[e] = __ldg(tri + 3 * (size_t)t0 + e);
    __syncwarp();
    for (unsigned q = 0; q < cnt; ++q) {
      const float4 a4 = s[3 * q], b4 = s[3 * q + 1], c4 = s[3 * q + 2];
      const float3 cp = closestOnTriangle(p, make_float3(a4.x, a4.y, a4.z),
                                          make_float3(b4.x, b4.y, b4.z),
                                          make_float3(c4.x, c4.y, c4.z));
      const float dx = p.x - cp.x, dy = p.y - cp.y, dz = p.z - cp.z;
      const float d2 = dx * dx + dy * dy + dz * dz;
      const unsigned id = __float_as_uint(a4.w);
      if (d2 < best || (d2 == best && id < bestTri)) {
        best = d2;
        bestTri = id;
        bestCp = cp;
      }
    }
    bound = fminf(bound, sqrtf(best));
  };
  evaluate(nearest);  // most of the bound's slack goes here
  for (unsigned c0 = 0; c0 < clusters; c0 += 32) {
    // 32 clusters against the brick, one a lane
    float far = bound;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
    bool take = false;
    if (c0 + lane < clusters) {
      const float4 a = __ldg(box + 2 * (c0 + lane)), b = __ldg(box + 2 * (c0 + lane) + 1);
      const float gx = gap(lo.x, hi.x, a.x, b.x), gy = gap(lo.y, hi.y, a.y, b.y),
                  gz = gap(lo.z, hi.z, a.z, b.z);
      take = c0 + lane != nearest && !(sqrtf(gx * gx + gy * gy + gz * gz) > far + slack);
    }
    unsigned todo = __ballot_sync(0xffffffffu, take);
    while (todo) {
      const unsigned c = c0 + (unsigned)__ffs((int)todo) - 1u;
      todo &= todo - 1u;
      const float4 a = __ldg(box + 2 * c), b = __ldg(box + 2 * c + 1);
      const float gx = gap(p.x, p.x, a.x, b.x), gy = gap(p.y, p.y, a.y, b.y),
                  gz = gap(p.z, p.z, a.z, b.z);
      const bool need = !(sqrtf(gx * gx + gy * gy + gz * gz) > bound + slack);
      if (__any_sync(0xffffffffu, need)) evaluate(c);
    }
  }
  if (valid) {
    const long long v = ((long long)k * L.vy + j) * L.vx + i;
    const float d = sqrtf(best);
    vert[v] = make_float4(d, bestCp.x, bestCp.y, bestCp.z);
    if (dist) dist[v] = d;
  }
}

// Few triangles: one thread per lattice vertex evaluates all of them, from shared
// memory.  There the sort, the clusters and the sign's passes cost more than they
// save.  One map, few / clusters: 18 triangles on 8 and 128 cells 72 / 142 and 331 /
// 826 us, 128 on 128 cells 873 / 924, 256 on 32 and 128 cells 164 / 210 and 1,464 /
// 973, 480 on 32 cells 259 / 267, 1,024 on 8 cells 403 / 397.  So it takes up to 128
// triangles, and up to 512 on lattices of at most 65,536 vertices.
constexpr unsigned kFewTriangles = 512;
__host__ inline bool fewTriangles(unsigned nt, long long vertices) {
  return nt <= 128u || (nt <= kFewTriangles && vertices <= 65536);
}
__global__ void __launch_bounds__(128)
kMeshFew(float4 *__restrict__ vert, Lattice L, const float4 *__restrict__ tri, unsigned nt) {
  __shared__ float4 sTri[3 * kFewTriangles];
  for (unsigned e = threadIdx.x; e < 3 * nt; e += blockDim.x) sTri[e] = __ldg(tri + e);
  __syncthreads();
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (long long)L.vx * L.vy * L.vz) return;
  const float3 p = latticePoint(L, (int)(v % L.vx), (int)(v / L.vx % L.vy),
                                (int)(v / ((long long)L.vx * L.vy)));
  float best = 3.4e38f, omega = 0.0f;
  float3 bestCp = p;
  for (unsigned q = 0; q < nt; ++q) {
    const float4 a4 = sTri[3 * q], b4 = sTri[3 * q + 1], c4 = sTri[3 * q + 2];
    const float3 a = make_float3(a4.x, a4.y, a4.z), b = make_float3(b4.x, b4.y, b4.z),
                 c = make_float3(c4.x, c4.y, c4.z);
    const float3 cp = closestOnTriangle(p, a, b, c);
    const float dx = p.x - cp.x, dy = p.y - cp.y, dz = p.z - cp.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    if (d2 < best) {  // (of equal distances the first triangle's)
      best = d2;
      bestCp = cp;
    }
    omega += solidAngle(p, a, b, c);
  }
  const float d = sqrtf(best);
  const bool inside = omega > 2.0f * 3.14159265358979f;  // winding number > 1/2
  vert[v] = make_float4(inside ? -d : d, bestCp.x, bestCp.y, bestCp.z);
}

// The lower neighbour whose sign vertex v shares, or -1 (v is a root): the
// segment between the two is shorter than one end's distance to the mesh.
__device__ __forceinline__ long long signParent(const float *__restrict__ dist, const Lattice &L,
                                                long long v) {
  const float step = L.cs * 1.001f;
  const long long sy = L.vx, sz = (long long)L.vx * L.vy;
  const float d = __ldg(dist + v);
  const bool x = v % sy != 0, y = (v / sy) % L.vy != 0, z = v >= sz;
  if (x && (d > step || __ldg(dist + v - 1) > step)) return v - 1;
  if (y && (d > step || __ldg(dist + v - sy) > step)) return v - sy;
  if (z && (d > step || __ldg(dist + v - sz) > step)) return v - sz;
  return -1;
}

// Lists the roots.
__global__ void __launch_bounds__(256)
kMeshRoots(const float *__restrict__ dist, Lattice L, long long *__restrict__ list,
           unsigned long long *__restrict__ count) {
  const long long total = (long long)L.vx * L.vy * L.vz;
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool root = v < total && signParent(dist, L, v) < 0;
  const unsigned lane = threadIdx.x & 31u, m = __ballot_sync(0xffffffffu, root);
  unsigned long long at = 0;
  if (lane == 0 && m) at = atomicAdd(count, (unsigned long long)__popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (root) list[at + __popc(m & ((1u << lane) - 1u))] = v;
}

// inside[v] of the listed roots: 32 roots per CTA at a time, one a lane, the
// triangles shared out over the warps.  kAll: the sign of every vertex instead.
constexpr int kWindWarps = 8;
template <bool kAll>
__global__ void __launch_bounds__(32 * kWindWarps)
kMeshWinding(Lattice L, const float4 *__restrict__ tri, unsigned nt,
             const long long *__restrict__ list, const unsigned long long *__restrict__ count,
             unsigned char *__restrict__ inside, float4 *__restrict__ vert) {
  __shared__ float4 sTri[kWindWarps][3 * kCluster];
  __shared__ float sOmega[kWindWarps][32];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const unsigned long long n = kAll ? (unsigned long long)L.vx * L.vy * L.vz : *count;
  const unsigned clusters = (nt + kCluster - 1) / kCluster;
  float4 *s = sTri[warp];
  for (unsigned long long base = blockIdx.x * 32u; base < n; base += gridDim.x * 32u) {
    const unsigned long long at = min(base + lane, n - 1ull);
    const long long v = kAll ? (long long)at : __ldg(list + at);
    const float3 p = latticePoint(L, (int)(v % L.vx), (int)(v / L.vx % L.vy),
                                  (int)(v / ((long long)L.vx * L.vy)));
    float omega = 0.0f;
    for (unsigned c = warp; c < clusters; c += kWindWarps) {
      const unsigned t0 = c * kCluster, cnt = min(kCluster, nt - t0);
      __syncwarp();
      for (unsigned e = lane; e < 3 * cnt; e += 32) s[e] = __ldg(tri + 3 * (size_t)t0 + e);
      __syncwarp();
      for (unsigned q = 0; q < cnt; ++q) {
        const float4 a = s[3 * q], b = s[3 * q + 1], c4 = s[3 * q + 2];
        omega += solidAngle(p, make_float3(a.x, a.y, a.z), make_float3(b.x, b.y, b.z),
                            make_float3(c4.x, c4.y, c4.z));
      }
    }
    sOmega[warp][lane] = omega;
    __syncthreads();
    if (warp == 0 && base + lane < n) {
      for (int w = 1; w < kWindWarps; ++w) omega += sOmega[w][lane];
      const bool in = omega > 2.0f * 3.14159265358979f;  // winding number > 1/2
      if (!kAll)
        inside[v] = in;
      else if (in)
        vert[v].x = -vert[v].x;
    }
    __syncthreads();
  }
}

// The sign of every vertex, from its root (parents are found from the
// unsigned distances).
__global__ void __launch_bounds__(256)
kMeshSign(float4 *__restrict__ vert, const float *__restrict__ dist, Lattice L,
          const unsigned char *__restrict__ inside) {
  const long long total = (long long)L.vx * L.vy * L.vz;
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= total) return;
  long long r = v;
  for (long long q = v; q >= 0; q = signParent(dist, L, r)) r = q;
  if (inside[r]) vert[v].x = -__ldg(dist + v);
}

// Whether every edge of the mesh is passed equally often in both directions
// (vertices told apart by their coordinates): the winding number is then
// constant off the surface.  Each directed edge adds a 64-bit hash of its
// ends with its direction's sign; a mesh with a boundary sums to zero with a
// probability of 2^-64.
bool meshClosed(const float *v3, uint nv, const uint *t3, uint nt) {
  auto mix = [](unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
  };
  std::vector<unsigned long long> hash(nv);
  for (uint v = 0; v < nv; ++v) {
    unsigned long long h = 0x9e3779b97f4a7c15ull;
    for (int a = 0; a < 3; ++a) {
      const float x = v3[3 * (size_t)v + a] + 0.0f;  // -0 and 0 are one place
      unsigned b;
      std::memcpy(&b, &x, 4);
      h = mix(h + b + 0x9e3779b97f4a7c15ull);
    }
    hash[v] = h;
  }
  unsigned long long sum = 0;
  for (size_t t = 0; t < nt; ++t)
    for (int c = 0; c < 3; ++c) {
      const unsigned long long a = hash[t3[3 * t + c]], b = hash[t3[3 * t + (c + 1) % 3]];
      if (a < b) sum += mix(a + 3 * mix(b));
      if (b < a) sum -= mix(b + 3 * mix(a));
    }
  return sum == 0;
}

// The map's vertices from the triangles (device, three float4 each).
bool meshMap(fcdemDistanceMap *m, const float4 *tri, unsigned nt, const float *vertices3,
             unsigned nv, const uint *triangles3, const float lo[3], const float hi[3]) {
  const Lattice L{m->cells[0] + 1, m->cells[1] + 1, m->cells[2] + 1,
                  make_float3(m->vmin[0], m->vmin[1], m->vmin[2]), m->cellSize};
  const long long total = (long long)L.vx * L.vy * L.vz;
  cudaStream_t st = curStream();
  if (fewTriangles(nt, total)) {
    kMeshFew<<<(unsigned)((total + 127) / 128), 128, 0, st>>>(m->vert, L, tri, nt);
    return launchOk() && cudaOk(cudaStreamSynchronize(st));
  }
  const unsigned clusters = (nt + kCluster - 1) / kCluster;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t sortedAt = al((size_t)nt * 8), boxAt = sortedAt + al((size_t)nt * 48),
               listAt = boxAt + al((size_t)clusters * 32), distAt = listAt + al((size_t)total * 8),
               insideAt = distAt + al((size_t)total * 4), countAt = insideAt + al((size_t)total);
  char *buf = nullptr;
  // without the per-vertex part every vertex is a root
  bool roots = cudaMalloc(&buf, countAt + 256) == cudaSuccess;
  if (!roots) {
    cudaGetLastError();
    if (cudaMalloc(&buf, listAt) != cudaSuccess) {
      cudaGetLastError();
      setError(FCDEM_ERR_ALLOC);
      return false;
    }
  }
  unsigned *key = (unsigned *)buf, *order = key + nt;
  float4 *sorted = (float4 *)(buf + sortedAt), *box = (float4 *)(buf + boxAt);
  long long *list = roots ? (long long *)(buf + listAt) : nullptr;
  float *dist = roots ? (float *)(buf + distAt) : nullptr;
  unsigned char *inside = roots ? (unsigned char *)(buf + insideAt) : nullptr;
  unsigned long long *count = roots ? (unsigned long long *)(buf + countAt) : nullptr;
  float3 scale;
  auto per = [&](int a) { return hi[a] > lo[a] ? 1024.0f / (hi[a] - lo[a]) : 0.0f; };
  scale = make_float3(per(0), per(1), per(2));
  float extent = 0.0f;
  for (int a = 0; a < 3; ++a)
    extent = std::fmax(extent, std::fmax(std::fabs(m->vmin[a]), std::fabs(m->vmax[a])));
  const unsigned vBlocks = (unsigned)((total + 255) / 256);
  const long long bricks = (long long)((L.vx + 3) / 4) * ((L.vy + 3) / 4) * ((L.vz + 1) / 2);
  bool ok = !roots || cudaOk(cudaMemsetAsync(count, 0, 8, st));
  kMeshKeys<<<(nt + 255) / 256, 256, 0, st>>>(tri, nt, make_float3(lo[0], lo[1], lo[2]), scale, key,
                                             order);
  ok = ok && launchOk();
  // (in the caller's order the clusters are wide, and as right)
  if (ok && scratch(ctx(), radixScratchBytes(nt), true)) radixSortPairs(ctx(), key, order, nt, 30);
  kMeshClusters<<<(clusters * 32 + 255) / 256, 256, 0, st>>>(tri, order, nt, sorted, box);
  ok = ok && launchOk();
  kMeshNearest<<<(unsigned)((bricks + kNearWarps - 1) / kNearWarps), 32 * kNearWarps, 0, st>>>(
      m->vert, dist, L, sorted, nt, box, 1e-5f * extent);
  ok = ok && launchOk();
  roots = meshClosed(vertices3, nv, triangles3, nt) && roots;  // meanwhile
  if (roots) {
    kMeshRoots<<<vBlocks, 256, 0, st>>>(dist, L, list, count);
    ok = ok && launchOk();
    kMeshWinding<false><<<numSms() * 4, 32 * kWindWarps, 0, st>>>(L, sorted, nt, list, count,
                                                                  inside, nullptr);
    ok = ok && launchOk();
    kMeshSign<<<vBlocks, 256, 0, st>>>(m->vert, dist, L, inside);
  } else {
    kMeshWinding<true><<<numSms() * 4, 32 * kWindWarps, 0, st>>>(L, sorted, nt, nullptr, nullptr,
                                                                 nullptr, m->vert);
  }
  ok = ok && launchOk() && cudaOk(cudaStreamSynchronize(st));
  cudaFree(buf);
  return ok;
}

}  // namespace
}  // namespace fcdem

using namespace fcdem;

extern "C" fcdemDistanceMap *fcdemDistMapFromMesh(const float *vertices3, uint numVertices,
                                       const uint *triangles3, uint numTriangles,
                                       int cellsPerAxis, float margin) {
  if (!vertices3 || !triangles3 || numVertices < 3 || numTriangles < 1 || cellsPerAxis < 1 ||
      !(margin >= 0.0f)) {
    setError(FCDEM_ERR_INVALID_VALUE);
    return nullptr;
  }
  float lo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, hi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
  for (uint v = 0; v < numVertices; ++v)
    for (int a = 0; a < 3; ++a) {
      lo[a] = std::fmin(lo[a], vertices3[3 * v + a]);
      hi[a] = std::fmax(hi[a], vertices3[3 * v + a]);
    }
  std::vector<float4> tri((size_t)numTriangles * 3);
  for (uint t = 0; t < numTriangles; ++t)
    for (int c = 0; c < 3; ++c) {
      const uint v = triangles3[3 * (size_t)t + c];
      if (v >= numVertices) { setError(FCDEM_ERR_INVALID_VALUE); return nullptr; }
      const float *x = vertices3 + 3 * (size_t)v;
      tri[3 * (size_t)t + c] = make_float4(x[0], x[1], x[2], 0.0f);
    }
  // cubic cells over the mesh box plus the margin, centred on the box: the
  // largest axis cut into cellsPerAxis cells, the others into whole cells
  float centre[3], ex[3], big = 0.0f;
  for (int a = 0; a < 3; ++a) {
    centre[a] = 0.5f * (lo[a] + hi[a]);
    ex[a] = 0.5f * (hi[a] - lo[a]) + margin;
    big = std::fmax(big, ex[a]);
  }
  if (!(big > 0.0f)) { setError(FCDEM_ERR_INVALID_VALUE); return nullptr; }
  const float cs = 2.0f * big / (float)cellsPerAxis;
  int cells[3];
  float vmin[3], vmax[3];
  for (int a = 0; a < 3; ++a) {
    cells[a] = std::max(1, (int)std::ceil(2.0f * ex[a] / cs));
    vmin[a] = centre[a] - 0.5f * cells[a] * cs;
    vmax[a] = vmin[a] + cells[a] * cs;
  }
  fcdemDistanceMap *m = fcdemDistMapCreate(nullptr, nullptr, vmin, vmax, cs, cells);
  if (!m) return nullptr;
  float4 *dTri = nullptr;
  if (cudaMalloc(&dTri, tri.size() * sizeof(float4)) != cudaSuccess) {
    cudaGetLastError();
    fcdemDistMapDestroy(m);
    setError(FCDEM_ERR_ALLOC);
    return nullptr;
  }
  const bool ok =
      uploadNow(dTri, tri.data(), tri.size() * sizeof(float4)) &&
      meshMap(m, dTri, numTriangles, vertices3, numVertices, triangles3, lo, hi);
  cudaFree(dTri);
  if (!ok) {
    fcdemDistMapDestroy(m);
    return nullptr;
  }
  return m;
}
