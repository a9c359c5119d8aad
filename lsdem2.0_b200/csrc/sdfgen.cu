// Level-set grid of a closed triangle mesh, computed on the device.
//
// Per grid node this is the work of LevelSetObject::Base::buildGrid
// (FunDEM/kernel/helper/LevelSetObjectGenerator.h:122-224) over
// TriangleMeshParticle::evaluateImplicitFunctionValueAndGradient (:888-914):
//   * the closest point of the mesh: per triangle, the Voronoi-region tests of
//     C. Ericson, "Real-Time Collision Detection" (2005), section 5.1.5 — the
//     reference's closestPointOnTriangle (:454-500); the nearest over all
//     triangles (the reference's BVH prunes only boxes farther than the best
//     so far, so it finds the same distance);
//   * inside or outside: the sum of the signed solid angles of all triangles
//     seen from the node, A. Van Oosterom and J. Strackee, IEEE Trans. Biomed.
//     Eng. 30 (1983) 125-126 (the reference's solidAngleFromPointToTriangle and
//     isPointInsideClosedTriangleMesh, :758-802), summed in triangle order;
//   * value = -+d, gradient -+(p - cp)/d, optionally negated (level set positive
//     inside), then buildGrid's value / |gradient|, or -+h/2 where |gradient|
//     <= 1e-12.
//
// Nearest triangle (k_nearest): the triangles in clusters of 32 with a bounding sphere. A node evaluates the cluster of its smallest upper bound, then every
// cluster whose sphere can come as near as what it has found; the smallest (distance, index)
// pair is the brute force's first smallest distance, bit for bit.
//
// Inside or outside: on a closed mesh (the edges' signed sum is zero) the sum is 4 pi times
// an integer that only changes across the surface, so nodes joined by a grid step no
// longer than the sum of their distances to the mesh share it. The nodes are joined by a
// union-find (k_join) and the sum is taken once per component, by a block, in FP32 (its
// error, 1e-6 per triangle, is far from the half that decides; a sum that is no
// integer within 0.05 is taken again in FP64). A component's node within 1e-6 spacings of the surface,
// where rounding decides, sums in FP64 in triangle order as the reference does.
// A mesh that is not closed takes k_mesh_grid: one thread per grid node, the mesh streamed through
// shared memory in tiles of kTile triangles, every node every triangle.
// 20,480-triangle mesh on a 49 x 39 x 31 grid: 23.9 ms by brute force (FP64 bound, 1.2e9
// node-triangle pairs with an atan2 each), 1.6 ms this way, 0.55 of them on the device.
//
// The file is compiled with --fmad=false so that products and sums round as the
// reference's host arithmetic does; distances are then bit-identical to the
// host computation and only the solid-angle sum can differ in its last bits
// (atan2), which moves the inside decision only for nodes on the surface.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "../../include/lsdem_b200.h"
#include "common.cuh"

namespace lsdem {
namespace {

constexpr int kTile = 128;
constexpr int kTriD = 10;     // doubles of one gathered triangle (9, and one for 16-byte loads)
constexpr int kThreads = 128;

LD double3 closest_on_triangle(double3 p, double3 a, double3 b, double3 c) {
  const double3 ab = b - a;
  const double3 ac = c - a;
  const double3 ap = p - a;
  const double d1 = dot(ab, ap);
  const double d2 = dot(ac, ap);
  if (d1 <= 0.0 && d2 <= 0.0) return a;
  const double3 bp = p - b;
  const double d3v = dot(ab, bp);
  const double d4 = dot(ac, bp);
  if (d3v >= 0.0 && d4 <= d3v) return b;
  const double vc = d1 * d4 - d3v * d2;
  if (vc <= 0.0 && d1 >= 0.0 && d3v <= 0.0) return a + (d1 / (d1 - d3v)) * ab;
  const double3 cp = p - c;
  const double d5 = dot(ab, cp);
  const double d6 = dot(ac, cp);
  if (d6 >= 0.0 && d5 <= d6) return c;
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) return a + (d2 / (d2 - d6)) * ac;
  const double va = d3v * d6 - d5 * d4;
  if (va <= 0.0 && (d4 - d3v) >= 0.0 && (d5 - d6) >= 0.0) {
    const double3 bc = c - b;
    return b + ((d4 - d3v) / ((d4 - d3v) + (d5 - d6))) * bc;
  }
  const double denom = 1.0 / (va + vb + vc);
  const double v = vb * denom;
  const double w = vc * denom;
  return a + ab * v + ac * w;
}

LD double solid_angle(double3 p, double3 a, double3 b, double3 c) {
  const double3 r0 = a - p;
  const double3 r1 = b - p;
  const double3 r2 = c - p;
  const double l0 = len(r0);
  const double l1 = len(r1);
  const double l2 = len(r2);
  if (l0 < 1e-30 || l1 < 1e-30 || l2 < 1e-30) return 0.0;
  const double num = dot(r0, cross(r1, r2));
  const double den = l0 * l1 * l2 + dot(r0, r1) * l2 + dot(r1, r2) * l0 + dot(r2, r0) * l1;
  return 2.0 * atan2(num, den);
}

// tri: kTriD doubles per triangle (vertex a, b, c).
__global__ void __launch_bounds__(kThreads) k_mesh_grid(const double* __restrict__ tri, int nt, double3 origin,
                                                        int nx, int ny, int nz, double h, int positive_inside,
                                                        double* __restrict__ out) {
  __shared__ double s_tri[kTile * 9];
  const long long n = (long long)nx * ny * nz;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  const long long ii = active ? i : 0;
  const int ix = (int)(ii % nx);
  const int iy = (int)((ii / nx) % ny);
  const int iz = (int)(ii / ((long long)nx * ny));
  const double3 p = d3(origin.x + double(ix) * h, origin.y + double(iy) * h, origin.z + double(iz) * h);
  double best = 1.7976931348623157e308;
  double3 cp = d3(0., 0., 0.);
  double sum = 0.0;
  for (int t0 = 0; t0 < nt; t0 += kTile) {
    const int m = min(kTile, nt - t0);
    __syncthreads();
    for (int k = threadIdx.x; k < m * 9; k += blockDim.x) s_tri[k] = tri[(long long)(t0 + k / 9) * kTriD + k % 9];
    __syncthreads();
    for (int k = 0; k < m; ++k) {
      const double* q = s_tri + 9 * k;
      const double3 a = d3(q[0], q[1], q[2]);
      const double3 b = d3(q[3], q[4], q[5]);
      const double3 c = d3(q[6], q[7], q[8]);
      const double3 x = closest_on_triangle(p, a, b, c);
      const double d2 = len2(p - x);
      if (d2 < best) {
        best = d2;
        cp = x;
      }
      sum += solid_angle(p, a, b, c);
    }
  }
  if (!active) return;
  const double d = len(p - cp);
  const bool inside = fabs(sum / (4.0 * 3.14159265358979323846)) > 0.5;
  double value = inside ? -d : d;
  double3 g = d3(0., 0., 0.);
  if (d > 1e-30) {
    const double3 u = (p - cp) / d;
    g = inside ? -u : u;
  }
  if (positive_inside) {
    value = -value;
    g = -g;
  }
  const double gn = len(g);
  out[i] = gn > 1e-12 ? value / gn : (value <= 0.0 ? -1.0 : 1.0) * 0.5 * h;
}

// The value of buildGrid from the distance d and the gradient norm gn of its direction.
LD double grid_value(double d, double gn, bool inside, int positive_inside, double h) {
  double v = inside ? -d : d;
  if (positive_inside) v = -v;
  return gn > 1e-12 ? v / gn : (v <= 0.0 ? -1.0 : 1.0) * 0.5 * h;
}

constexpr int kCluster = 32;  // triangles of one bounding sphere

struct GridArgs {
  double3 origin;
  double h;
  int nx, ny, nz;
  LD double3 node(int x, int y, int z) const {
    return d3(origin.x + double(x) * h, origin.y + double(y) * h, origin.z + double(z) * h);
  }
};

// Gathers the triangles and bounds each cluster by a sphere, one warp per cluster.
__global__ void k_clusters(const double* __restrict__ verts, const int* __restrict__ tris, int nt,
                           double* __restrict__ tri, float4* __restrict__ trif, double scale,
                           float4* __restrict__ sphere) {
  const int lane = threadIdx.x & 31, c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c * kCluster >= nt) return;
  const int t = min(c * kCluster + lane, nt - 1);
  double3 p[3], lo = d3(1e300, 1e300, 1e300), hi = d3(-1e300, -1e300, -1e300);
  for (int k = 0; k < 3; ++k) {
    const double* q = verts + 3 * (size_t)tris[3 * (size_t)t + k];
    p[k] = d3(q[0], q[1], q[2]);
    lo = d3(fmin(lo.x, q[0]), fmin(lo.y, q[1]), fmin(lo.z, q[2]));
    hi = d3(fmax(hi.x, q[0]), fmax(hi.y, q[1]), fmax(hi.z, q[2]));
  }
  if (c * kCluster + lane < nt) {
    double* o = tri + (size_t)kTriD * t;
    for (int k = 0; k < 3; ++k) { o[3 * k] = p[k].x; o[3 * k + 1] = p[k].y; o[3 * k + 2] = p[k].z; }
    o[9] = 0.0;
    // FP32 copy scaled to the mesh's size, for the components' sums
    float4* f = trif + 3 * (size_t)t;
    for (int k = 0; k < 3; ++k)
      f[k] = make_float4((float)(p[k].x * scale), (float)(p[k].y * scale), (float)(p[k].z * scale), 0.f);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = d3(fmin(lo.x, __shfl_xor_sync(~0u, lo.x, o)), fmin(lo.y, __shfl_xor_sync(~0u, lo.y, o)),
            fmin(lo.z, __shfl_xor_sync(~0u, lo.z, o)));
    hi = d3(fmax(hi.x, __shfl_xor_sync(~0u, hi.x, o)), fmax(hi.y, __shfl_xor_sync(~0u, hi.y, o)),
            fmax(hi.z, __shfl_xor_sync(~0u, hi.z, o)));
  }
  const float4 m = make_float4((float)(0.5 * (lo.x + hi.x)), (float)(0.5 * (lo.y + hi.y)), (float)(0.5 * (lo.z + hi.z)), 0.f);
  double r = 0.0;  // about the rounded centre; a NaN corner makes the radius NaN, which excludes nothing
  for (int k = 0; k < 3; ++k) {
    const double l = len(p[k] - d3(m.x, m.y, m.z));
    r = l <= r ? r : l;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double l = __shfl_xor_sync(~0u, r, o);
    r = l <= r ? r : l;
  }
  if (lane == 0) sphere[c] = make_float4(m.x, m.y, m.z, __double2float_ru(r * (1.0 + 1e-9)));
}

// Distance to the nearest triangle and norm of its direction, one warp per node: its lanes share
// the clusters' bounds and then the triangles of each cluster that can hold the nearest. (One
// thread per node evaluated, with its warp, every cluster that any of 32 nodes needed, near the
// middle of a body most of them: 3.0 ms of the case above against 0.37.)
__global__ void __launch_bounds__(128) k_nearest(const double* __restrict__ tri, int nt,
                                                 const float4* __restrict__ sphere, int nc, GridArgs g, int n,
                                                 double* __restrict__ dist, double* __restrict__ norm) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // thread numbers pass 32 bits at 2^27 nodes
  if (i >= n) return;
  const double3 p = g.node(i % g.nx, i / g.nx % g.ny, i / (g.nx * g.ny));
  const float px = (float)p.x, py = (float)p.y, pz = (float)p.z;
  // distance from the node to a sphere's centre, and the bound of its error (roundings of p, of
  // the difference and of the root: below 4 ulps of the coordinates and of the distance)
  auto centre = [&](const float4& q) {
    const float dx = px - q.x, dy = py - q.y, dz = pz - q.z;
    return sqrtf(dx * dx + dy * dy + dz * dz);
  };
  const float slack = 1e-6f * (fabsf(px) + fabsf(py) + fabsf(pz));
  double bd = 1.7976931348623157e308;  // this lane's best: smallest (d2, triangle)
  int bt = 0x7fffffff;
  double3 cp = d3(0., 0., 0.);
  double thr = bd;  // at least the warp's smallest d2
  auto cluster = [&](int c) {
    const int t = c * kCluster + lane;
    if (t < nt) {
      const double2* q = reinterpret_cast<const double2*>(tri + (size_t)kTriD * t);
      const double2 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2), q3 = __ldg(q + 3), q4 = __ldg(q + 4);
      const double3 x = closest_on_triangle(p, d3(q0.x, q0.y, q1.x), d3(q1.y, q2.x, q2.y), d3(q3.x, q3.y, q4.x));
      const double d2 = len2(p - x);
      if (d2 < bd || (d2 == bd && t < bt)) {
        bd = d2;
        bt = t;
        cp = x;
      }
    }
    // d2 >= 0, whose high words order as integers: the smallest, rounded up
    const unsigned hi = __reduce_min_sync(~0u, (unsigned)__double2hiint(bd));
    thr = hi < 0x7fefffffu ? __hiloint2double((int)(hi + 1), 0) * (1.0 + 1e-9) : 1.7976931348623157e308;
  };
  // the cluster of the smallest upper bound first
  float ub = 3e38f;
  int cu = 0;
  for (int c = lane; c < nc; c += 32) {
    const float4 s = __ldg(sphere + c);
    const float u = centre(s) + s.w;
    if (u < ub) {
      ub = u;
      cu = c;
    }
  }
  const unsigned least = __reduce_min_sync(~0u, __float_as_uint(ub));
  cu = __shfl_sync(~0u, cu, __ffs(__ballot_sync(~0u, __float_as_uint(ub) == least)) - 1);
  cluster(cu);
  for (int c0 = 0; c0 < nc; c0 += 32) {
    const int c = c0 + lane;
    double l2 = -1.0;  // NaN bounds never exclude a cluster
    bool left = c < nc && c != cu;
    if (left) {
      const float4 s = __ldg(sphere + c);
      const float l = centre(s) * (1.0f - 1e-5f) - s.w * (1.0f + 1e-5f) - slack;
      l2 = l > 0.f ? (double)l * (double)l : -1.0;
    }
    for (unsigned m; (m = __ballot_sync(~0u, left && !(l2 > thr))) != 0;) {
      const int b = __ffs(m) - 1;
      if (lane == b) left = false;
      cluster(c0 + b);
    }
  }
  // the smallest (d2, triangle) of the warp
  const unsigned hi = __double2hiint(bd), lo = __double2loint(bd);
  const unsigned mh = __reduce_min_sync(~0u, hi);
  const unsigned ml = __reduce_min_sync(~0u, hi == mh ? lo : 0xffffffffu);
  const bool tie = hi == mh && lo == ml;
  const int mt = (int)__reduce_min_sync(~0u, tie ? (unsigned)bt : 0xffffffffu);
  if (!(tie && bt == mt) || (bt == 0x7fffffff && lane > 0)) return;
  const double d = len(p - cp);
  double3 u = d3(0., 0., 0.);
  if (d > 1e-30) u = (p - cp) / d;
  dist[i] = d;
  norm[i] = len(u);
}

// Signed sums of the undirected edges in an open-addressing table (key 0: empty; keys are
// offset by one): closed when all are zero. Slots are at least twice the edges, so a probe ends.
__global__ void k_edges(const int* __restrict__ tris, int nt, unsigned long long* keys, int* sums, unsigned mask) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * nt) return;
  const int t = e / 3, k = e % 3;
  const unsigned u = tris[3 * (size_t)t + k], v = tris[3 * (size_t)t + (k + 1) % 3];
  const unsigned a = min(u, v), b = max(u, v);
  const unsigned long long key = (((unsigned long long)a << 32) | b) + 1ull;
  unsigned slot = (a * 0x9E3779B1u ^ b * 0x85EBCA77u);
  slot ^= slot >> 15;
  for (unsigned n = 0; n <= mask; ++n, ++slot) {
    const unsigned long long was = atomicCAS(&keys[slot & mask], 0ull, key);
    if (was == 0ull || was == key) {
      atomicAdd(&sums[slot & mask], u < v ? 1 : -1);
      return;
    }
  }
}
__global__ void k_closed(const int* __restrict__ sums, unsigned slots, int* open) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < slots && sums[i] != 0) *open = 1;
}

// Union-find over the nodes: parent[i] <= i, roots are their own parents.
LD int find_root(int* parent, int i) {
  int p = __ldcg(parent + i);
  while (p != i) {
    const int g = __ldcg(parent + p);
    if (g != p) parent[i] = g;  // halves the path; any ancestor is a valid parent
    i = p;
    p = g;
  }
  return i;
}
// True when no point of the mesh can lie on the step of squared length l2 (in spacings) between
// nodes at distances da and db from it.
LD bool joined(double da, double db, int l2, const GridArgs& g) {
  const double L = g.h * sqrt((double)l2) * (1.0 + 1e-9) + 1e-12 * (fabs(g.origin.x) + fabs(g.origin.y) + fabs(g.origin.z));
  return da + db > L;
}
// Nodes joined along x under the first of their run (or 64 nodes back in it).
__global__ void k_runs(const double* __restrict__ dist, GridArgs g, int* parent) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nx * g.ny * g.nz) return;
  const int x = i % g.nx;
  int k = 0;
  for (double d = dist[i]; k < min(x, 64); ++k) {
    const double e = dist[i - k - 1];
    if (!joined(d, e, 1, g)) break;
    d = e;
  }
  parent[i] = i - k;
}
// The runs joined across rows. A step whose two ends and the step before it along x are all
// joined adds nothing, which leaves a few steps per pair of runs.
__global__ void k_join(const double* __restrict__ dist, GridArgs g, int* parent) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nx * g.ny * g.nz) return;
  const int x = i % g.nx, y = i / g.nx % g.ny, z = i / (g.nx * g.ny);
  const double d = dist[i], dp = x > 0 ? dist[i - 1] : 0.0;
  const bool back = x > 0 && joined(d, dp, 1, g);
  for (int k = 0; k < 12; ++k) {  // the 26 neighbours of smaller index, but the one along x
    const int dx = k % 3 - 1, dy = k < 9 ? k / 3 - 1 : -1, dz = k < 9 ? -1 : 0;
    const int X = x + dx, Y = y + dy, Z = z + dz;
    if (X < 0 || X >= g.nx || Y < 0 || Y >= g.ny || Z < 0) continue;
    const int j = X + g.nx * (Y + g.ny * Z), l2 = dx * dx + dy * dy + dz * dz;
    const double e = dist[j];
    if (!joined(d, e, l2, g)) continue;
    if (back && X > 0) {
      const double ep = dist[j - 1];
      if (joined(e, ep, 1, g) && joined(dp, ep, l2, g)) continue;
    }
    int a = find_root(parent, i), b = find_root(parent, j);
    while (a != b) {  // the larger root goes under the smaller; each retry has a smaller root
      if (a < b) { const int t = a; a = b; b = t; }
      const int was = atomicCAS(parent + a, a, b);
      if (was == a) break;
      a = find_root(parent, was);
      b = find_root(parent, b);
    }
  }
}
__global__ void k_roots(int* parent, int n, int* __restrict__ list, int* count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && find_root(parent, i) == i) list[atomicAdd(count, 1)] = i;
}

// Solid angle in FP32; false where that is not sure of it: next to the triangle, where the
// determinant's sign turns the angle by 4 pi (its FP32 error is about 1e-6 of the lengths' product).
LD bool solid_angle_f(float3 p, float4 a, float4 b, float4 c, float& angle) {
  const float x0 = a.x - p.x, y0 = a.y - p.y, z0 = a.z - p.z, x1 = b.x - p.x, y1 = b.y - p.y, z1 = b.z - p.z,
              x2 = c.x - p.x, y2 = c.y - p.y, z2 = c.z - p.z;
  const float l0 = sqrtf(x0 * x0 + y0 * y0 + z0 * z0), l1 = sqrtf(x1 * x1 + y1 * y1 + z1 * z1),
              l2 = sqrtf(x2 * x2 + y2 * y2 + z2 * z2);
  const float num = x0 * (y1 * z2 - z1 * y2) + y0 * (z1 * x2 - x1 * z2) + z0 * (x1 * y2 - y1 * x2);
  const float lll = l0 * l1 * l2;
  const float den = lll + (x0 * x1 + y0 * y1 + z0 * z1) * l2 + (x1 * x2 + y1 * y2 + z1 * z2) * l0 +
                    (x2 * x0 + y2 * y0 + z2 * z0) * l1;
  if (!(den > 1e-3f * lll || fabsf(num) > 1e-3f * lll)) return false;
  angle = 2.0f * atan2f(num, den);
  return true;
}

// Solid-angle sum of each component's root: inside[root], one block per root at a time (four at
// a time read the triangles together, but leave the chip two blocks an SM for the thousand-odd
// components of a body: 278 us against 131). In FP32
// the mesh and the node are rounded to 1e-7 of the mesh's size, each vertex alike in all its
// triangles, so the mesh stays closed, and nodes farther than 1e-5 of that size from it stay on
// their side. Nodes nearer than that sum in FP64, and those on the surface as far as rounding goes
// in the triangles' order, which is the reference's: a block's threads take the angles and one of
// them adds (43,200 triangles of a box, 11,600 of 91,000 nodes on its faces: 300 ms for the call with
// one thread taking the angles, too, 5.4 ms with the block).
__global__ void __launch_bounds__(128) k_component_sign(const double* __restrict__ tri, const float4* __restrict__ trif,
                                                        int nt, GridArgs g, double scale,
                                                        const double* __restrict__ dist, const int* __restrict__ list,
                                                        const int* __restrict__ count, unsigned char* inside) {
  __shared__ double s_sum[128];
  const int n = *count, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto angle = [&](double3 q, int t) {
    const double* r = tri + (size_t)kTriD * t;
    return solid_angle(q, d3(r[0], r[1], r[2]), d3(r[3], r[4], r[5]), d3(r[6], r[7], r[8]));
  };
  auto block_sum = [&](double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
    __syncthreads();  // the last sum has been read
    if (lane == 0) s_sum[warp] = v;
    __syncthreads();
    return s_sum[0] + s_sum[1] + s_sum[2] + s_sum[3];
  };
  const double pi4 = 4.0 * 3.14159265358979323846;
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    const int i = list[k];
    const double3 p = g.node(i % g.nx, i / g.nx % g.ny, i / (g.nx * g.ny));
    const double d = dist[i];
    double w = 0.0;
    bool sure = d == 0.0;  // the value there does not depend on the side
    if (d * scale > 1e-5) {
      const float3 q = make_float3((float)(p.x * scale), (float)(p.y * scale), (float)(p.z * scale));
      double sum = 0.0;
      for (int t = tid; t < nt; t += 128) {
        const float4 a = __ldg(trif + 3 * (size_t)t), b = __ldg(trif + 3 * (size_t)t + 1), c = __ldg(trif + 3 * (size_t)t + 2);
        float f;
        sum += solid_angle_f(q, a, b, c, f) ? (double)f : angle(p, t);
      }
      w = block_sum(sum) / pi4;
      sure = fabs(w - rint(w)) < 0.05;
    }
    if (!sure && d < 1e-6 * g.h) {
      double sum = 0.0;
      for (int t0 = 0; t0 < nt; t0 += 128) {
        __syncthreads();  // the last angles have been added
        if (t0 + tid < nt) s_sum[tid] = angle(p, t0 + tid);
        __syncthreads();
        if (tid == 0)
          for (int t = 0; t < min(128, nt - t0); ++t) sum += s_sum[t];
      }
      w = sum / pi4;  // the first thread's
    } else if (!sure) {
      double sum = 0.0;
      for (int t = tid; t < nt; t += 128) sum += angle(p, t);
      w = block_sum(sum) / pi4;
    }
    if (tid == 0) inside[i] = fabs(w) > 0.5;
  }
}

__global__ void k_grid_values(const double* __restrict__ dist, const double* __restrict__ norm, int* parent, int n,
                              const unsigned char* __restrict__ inside, int positive_inside, double h,
                              double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = grid_value(dist[i], norm[i], inside[find_root(parent, i)] != 0, positive_inside, h);
}

bool mesh_valid(int nv, const int* tris, int nt) {
  if (nv <= 0 || nt <= 0) return false;
  for (int t = 0; t < nt; ++t) {
    const int a = tris[3 * t], b = tris[3 * t + 1], c = tris[3 * t + 2];
    if (a < 0 || b < 0 || c < 0 || a >= nv || b >= nv || c >= nv) return false;
    if (a == b || b == c || c == a) return false;
  }
  return true;
}

}  // namespace
}  // namespace lsdem

extern "C" int lsdem_mesh_grid_box(const double* verts, int n_verts, double spacing, int pad, double* origin3,
                                   int* size3) {
  if (!verts || n_verts <= 0 || !(spacing > 0.0) || !origin3 || !size3) return LSDEM_ERR_ARG;
  double mn[3] = {verts[0], verts[1], verts[2]}, mx[3] = {verts[0], verts[1], verts[2]};
  for (int v = 1; v < n_verts; ++v)
    for (int a = 0; a < 3; ++a) {
      mn[a] = std::min(mn[a], verts[3 * v + a]);
      mx[a] = std::max(mx[a], verts[3 * v + a]);
    }
  const double padding = double(std::max(1, pad)) * spacing;
  for (int a = 0; a < 3; ++a) {
    const double lo = spacing * std::floor((mn[a] - padding) / spacing);
    const double hi = spacing * std::ceil((mx[a] + padding) / spacing);
    const int n = int(std::floor((hi - lo) / spacing + 0.5)) + 1;
    if (n <= 0) return LSDEM_ERR_ARG;
    origin3[a] = lo;
    size3[a] = n;
  }
  return LSDEM_OK;
}

extern "C" int lsdem_mesh_grid(const double* verts, int n_verts, const int* tris, int n_tris, const double* origin3,
                               const int* size3, double spacing, int positive_inside, double* sdf_out, int device) {
  using namespace lsdem;
  if (!verts || !tris || !origin3 || !size3 || !sdf_out || !(spacing > 0.0)) return LSDEM_ERR_ARG;
  if (size3[0] <= 0 || size3[1] <= 0 || size3[2] <= 0) return LSDEM_ERR_ARG;
  if (!mesh_valid(n_verts, tris, n_tris)) return LSDEM_ERR_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return LSDEM_ERR_NODEVICE;
  if (device < 0 || device >= ndev) return LSDEM_ERR_ARG;
  int prev = 0;
  cudaGetDevice(&prev);
  if (cudaSetDevice(device) != cudaSuccess) return LSDEM_ERR_CUDA;
  const long long n = (long long)size3[0] * size3[1] * size3[2];
  // node and triangle indices are 32-bit on the way below the brute force
  bool small = n < (1ll << 30) && n_tris < (1 << 28);
  const int nc = (n_tris + kCluster - 1) / kCluster;
  unsigned slots = 64;
  while (small && slots < 6u * (unsigned)n_tris) slots *= 2;
  // one allocation for the call
  size_t bytes, o_vert, o_tris, o_tri, o_sph, o_trif, o_out, o_dist, o_norm, o_par, o_list, o_in, o_zero, o_keys, o_sums, o_flag;
  auto layout = [&] {
    bytes = 0;
    auto part = [&](size_t b) {
      const size_t at = bytes;
      bytes += (b + 255) & ~(size_t)255;
      return at;
    };
    o_vert = part(24 * (size_t)n_verts), o_tris = part(12 * (size_t)n_tris);
    o_tri = part(8 * (size_t)kTriD * n_tris), o_sph = part(16 * (size_t)nc), o_trif = part(48 * (size_t)n_tris);
    o_out = part(8 * (size_t)n);
    const size_t m = small ? (size_t)n : 0;
    o_dist = part(8 * m), o_norm = part(8 * m), o_par = part(4 * m), o_list = part(4 * m), o_in = part(m);
    o_zero = bytes, o_keys = part(small ? 8 * (size_t)slots : 0), o_sums = part(small ? 4 * (size_t)slots : 0);
    o_flag = part(8);  // {open, components}
  };
  layout();
  char* d = nullptr;
  int rc = LSDEM_OK;
  cudaStream_t st = nullptr;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) rc = LSDEM_ERR_CUDA;
  if (rc == LSDEM_OK && cudaMalloc(&d, bytes) != cudaSuccess) {
    d = nullptr;
    if (small) {  // 33 bytes a node do not fit: the brute force takes 8
      small = false;
      layout();
      if (cudaMalloc(&d, bytes) != cudaSuccess) d = nullptr;
    }
    cudaGetLastError();
    if (!d) rc = LSDEM_ERR_NOMEM;
  }
  if (rc == LSDEM_OK) {
    auto at = [&](size_t o) { return d + o; };
    double* d_tri = (double*)at(o_tri);
    double* d_out = (double*)at(o_out);
    int* flag = (int*)at(o_flag);
    const GridArgs g{d3(origin3[0], origin3[1], origin3[2]), spacing, size3[0], size3[1], size3[2]};
    double ext = 0.0;  // largest coordinate of the mesh or of the grid's box
    for (int v = 0; v < 3 * n_verts; ++v) ext = std::max(ext, std::fabs(verts[v]));
    for (int k = 0; k < 3; ++k)
      ext = std::max({ext, std::fabs(origin3[k]), std::fabs(origin3[k] + spacing * size3[k])});
    const double scale = ext > 0.0 ? 1.0 / ext : 1.0;
    cudaMemcpyAsync(at(o_vert), verts, 24 * (size_t)n_verts, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(at(o_tris), tris, 12 * (size_t)n_tris, cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(at(o_zero), 0, bytes - o_zero, st);
    k_clusters<<<(unsigned)((32ll * nc + 127) / 128), 128, 0, st>>>((const double*)at(o_vert), (const int*)at(o_tris), n_tris,
                                                                   d_tri, (float4*)at(o_trif), scale, (float4*)at(o_sph));
    int open = 1;
    if (small) {
      const unsigned blocks = (unsigned)((n + 255) / 256);
      k_edges<<<(unsigned)((3ll * n_tris + 255) / 256), 256, 0, st>>>((const int*)at(o_tris), n_tris,
                                                                     (unsigned long long*)at(o_keys), (int*)at(o_sums), slots - 1);
      k_closed<<<(slots + 255) / 256, 256, 0, st>>>((const int*)at(o_sums), slots, flag);
      cudaMemcpyAsync(&open, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
      if (cudaStreamSynchronize(st) != cudaSuccess) open = 1;
      if (!open) {
        double* dist = (double*)at(o_dist);
        double* norm = (double*)at(o_norm);
        int* parent = (int*)at(o_par);
        k_nearest<<<(unsigned)((n + 3) / 4), 128, 0, st>>>(d_tri, n_tris, (const float4*)at(o_sph), nc, g, (int)n, dist, norm);
        k_runs<<<blocks, 256, 0, st>>>(dist, g, parent);
        k_join<<<blocks, 256, 0, st>>>(dist, g, parent);
        k_roots<<<blocks, 256, 0, st>>>(parent, (int)n, (int*)at(o_list), flag + 1);
        k_component_sign<<<148 * 8, 128, 0, st>>>(d_tri, (const float4*)at(o_trif), n_tris, g, scale, dist, (const int*)at(o_list),
                                                  flag + 1, (unsigned char*)at(o_in));
        k_grid_values<<<blocks, 256, 0, st>>>(dist, norm, parent, (int)n, (const unsigned char*)at(o_in), positive_inside,
                                              spacing, d_out);
      }
    }
    if (open) {
      const long long blocks = (n + kThreads - 1) / kThreads;
      k_mesh_grid<<<(unsigned)blocks, kThreads, 0, st>>>(d_tri, n_tris, g.origin, g.nx, g.ny, g.nz, spacing,
                                                         positive_inside, d_out);
    }
    cudaMemcpyAsync(sdf_out, d_out, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = LSDEM_ERR_CUDA;
  }
  if (d) cudaFree(d);
  if (st) cudaStreamDestroy(st);
  cudaSetDevice(prev);
  return rc;
}
