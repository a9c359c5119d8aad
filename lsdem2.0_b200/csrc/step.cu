// Level-set DEM step kernels for sm_100a.
//
// Kernel map against the reference hot path (paths relative to the reference root):
//   k_integrate_first  half kick + drift + cell key (+ wall drift/key); replaces
//                      particleVelocityAngularVelocityIntegrationKernel + particlePositionOrientationIntegrationKernel
//                      (FunDEM/kernel/CUDAKernelFunction/particleIntegrationKernel.cu:3-40) and
//                      calculateHashKernel (myUtility/mySpatialGrid.cu:4-26)
//   k_candidates       particle-level candidate partners from the cell grid (new: replaces the
//                      per-node 27-cell scan of LSParticleContactDetectionKernel.cu:44-61)
//   k_screen_f         node-vs-SDF rejections (LSParticleContactDetectionKernel.cu:4-590), FP32
//   k_contacts_f       node-vs-SDF tests of the rest, history carry-over (…cu:280-289) and the
//                      linear contact force (contactKernel.cuh:4-77, contactKernel.cu:46-271)
//   k_kick             second half kick (particleIntegrationKernel.cu:3-24)
//   k_periodic         wrap + ghost images + ghost keys (mySpatialGrid.cu:28-56, 87-152, 214-240)
//   k_bonds            V-bond forces (contactKernel.cuh:138-199, contactKernel.cu:273-351)
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.h"
#include "images.cuh"
#include "separation.cuh"

namespace lsdem {

static constexpr unsigned FULL = 0xffffffffu;
static constexpr int NP_WARPS = 4;     // warps per narrowphase block
static constexpr int MAXCL = 256;      // clusters of 32 nodes per shape (8192 nodes)

LD unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename T>
LD T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
LD double3 warp_sum3(double3 v) { return d3(warp_sum(v.x), warp_sum(v.y), warp_sum(v.z)); }
LD void atomic_add3(double3* arr, int i, double3 v) {
  atomicAdd(&arr[i].x, v.x);
  atomicAdd(&arr[i].y, v.y);
  atomicAdd(&arr[i].z, v.z);
}

// Absolute slack for conservative culling: covers FP64 rounding of coordinates.
LD double coord_slack(double3 a, double3 b) {
  return 1e-14 * (fabs(a.x) + fabs(a.y) + fabs(a.z) + fabs(b.x) + fabs(b.y) + fabs(b.z)) + 1e-300;
}

static int g_num_sms = 0;
static int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

// ---------------------------------------------------------------------------
// Integration, first half of the step (reference step order, LSSolver.h:1000-1011). Bound by
// memory: 0.4 KB a particle. Inside a batch it also does the second half kick of the step
// before, with a.kick, from the force and orientation it reads anyway (as a launch of its own
// the kick took 68 us of a step of 2M particles and 5 us of one of 2,000).
LD double3 kicked(double3 v, double3 acc, double h) { return d3(fma(acc.x, h, v.x), fma(acc.y, h, v.y), fma(acc.z, h, v.z)); }
__global__ void k_integrate_first(StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    // contacts of the previous step: largest demand of the batch, then reset
    if (a.C_old.count) atomicMax(&a.status->need_contact, *a.C_old.count);
    *a.C.count = 0;
    if (a.reuse_next) *a.reuse_next = 0;
    if (a.G.count) *a.G.count = 0;
    if (a.mb.ctr) a.mb.ctr[0] = a.mb.ctr[1] = a.mb.ctr[2] = 0;
    if (a.pl.ctr) a.pl.ctr[0] = a.pl.ctr[1] = a.pl.ctr[2] = 0;
    for (int l = 0; l < 2; ++l)
      if (a.net[l].ctr) {
        a.net[l].ctr[0] = a.net[l].ctr[1] = 0;
        for (int k = 0; k < a.nshapes; ++k) a.net[l].cnt[k] = 0;
      }
  }
  if (i < a.P.n) {
    const BodyView& P = a.P;
    const double h = 0.5 * a.dt;
    double3 v = P.vel[i], w = P.angvel[i];
    Quat q = P.quat[i];
    const double im = P.invmass[i];
    if (!is_zero(im)) {
      const double3 acc = P.force[i] * im + a.gravity, ang = mul(rotate_inv_inertia(q, P.invI[i]), P.torque[i]);
      if (a.kick) {  // the last step's second half kick, from the same force and orientation
        v = kicked(v, acc, h);
        w = kicked(w, ang, h);
      }
      v = kicked(v, acc, h);
      w = kicked(w, ang, h);
      P.vel[i] = v;
      P.angvel[i] = w;
    }
    double3 x = P.pos[i];
    x += a.dt * v;
    q = quat_integrate(q, w, a.dt);
    P.pos[i] = x;
    P.quat[i] = q;
    P.force[i] = d3(0., 0., 0.);
    P.torque[i] = d3(0., 0., 0.);
    const int key = hash_key(x, a.pg);
    if (a.reuse) {
      // a move or turn beyond the neighbour-list margin (a periodic wrap included) needs a
      // new sort and new lists; so does a body entering or leaving the domain, since the
      // lists hold only bodies that were in a cell at the build
      const double3 m = x - a.xb[i];
      const float4 b = a.qb[i];
      const double dq = (q.q0 - b.x) * (q.q0 - b.x) + (q.q1 - b.y) * (q.q1 - b.y) + (q.q2 - b.z) * (q.q2 - b.z) +
                        (q.q3 - b.w) * (q.q3 - b.w);
      // a point of the body at distance p from its centre has moved by at most |m| + 2 |dq| p
      // (|dq| is 2 sin(angle / 4), its chord 2 sin(angle / 2) p); FP32 roundings, that of qb
      // among them, are within the 1e-6
      const float r = a.turn[i];
      const float move = sqrtf((float)dot(m, m)) + (2.0f * sqrtf((float)dq) + 1e-6f) * r;
      // so does a body beyond a periodic face, whose wrap k_wrap does
      const GridP& g = a.pg;
      const bool beyond = ((a.wrap_axes & 1) && (x.x < g.mn.x || x.x >= g.mx.x)) ||
                          ((a.wrap_axes & 2) && (x.y < g.mn.y || x.y >= g.mx.y)) ||
                          ((a.wrap_axes & 4) && (x.z < g.mn.z || x.z >= g.mx.z));
      if (!(move * (1.0f + 1e-6f) <= a.move) || (key >= 0) != (a.kin[i] != 0) || beyond) atomicOr(a.reuse, 2);
    }
    P.key[i] = key;
    if (a.reuse) {  // the candidate search's records
      a.rec[2 * i] = make_float4((float)x.x, (float)x.y, (float)x.z, __int_as_float(key));
      a.rec[2 * i + 1] = make_float4((float)q.q0, (float)q.q1, (float)q.q2, (float)q.q3);
    }
    if (a.pgh.cnt) a.pgh.cnt[i] = 0;
  } else if (i < a.P.n + a.W.n) {
    const int k = i - a.P.n;
    const BodyView& W = a.W;
    double3 x = W.pos[k];
    x += a.dt * W.vel[k];
    W.pos[k] = x;
    W.quat[k] = quat_integrate(W.quat[k], W.angvel[k], a.dt);
    W.key[k] = hash_key(x, a.wg);
  }
}

void launch_integrate_first(const StepArgs& a, cudaStream_t s) {
  int n = a.P.n + a.W.n;
  if (n < 1) n = 1;
  k_integrate_first<<<(n + 255) / 256, 256, 0, s>>>(a);
}

// Radius within which a body's points count for the lists. A node of another body counts against a
// body only within its bounding radius, but against its images wherever their grid's solid reaches.
__global__ void k_turn_radius(int n, const float4* __restrict__ rec_s, const float* __restrict__ sup_t,
                              float* __restrict__ turn) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 s = rec_s[i];
  turn[i] = sup_t ? fmaxf(s.x, s.y * sup_t[__float_as_int(s.z)]) : s.x;
}
void launch_turn_radius(int n, const float4* rec_s, const float* sup_t, float* turn, cudaStream_t s) {
  if (n > 0) k_turn_radius<<<(n + 255) / 256, 256, 0, s>>>(n, rec_s, sup_t, turn);
}

__global__ void k_kick(StepArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.P.n) return;
  const BodyView& P = a.P;
  const double im = P.invmass[i];
  if (is_zero(im)) return;
  const double h = 0.5 * a.dt;
  P.vel[i] = kicked(P.vel[i], P.force[i] * im + a.gravity, h);
  P.angvel[i] = kicked(P.angvel[i], mul(rotate_inv_inertia(P.quat[i], P.invI[i]), P.torque[i]), h);
}

void launch_kick(const StepArgs& a, cudaStream_t s) {
  if (a.P.n > 0) k_kick<<<(a.P.n + 255) / 256, 256, 0, s>>>(a);
}

// The batch's state and history aside in one launch: plain arrays, and of the candidate slots
// only the filled ones (the slots of 2M particles are 0.8 GB, 0.1 of them per particle filled;
// as one copy per array the backup was 23 launches, 60 us of a batch of a small system).
__global__ void k_backup(BackupArgs b) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, T = (long long)gridDim.x * blockDim.x;
  for (int s = 0; s < b.nseg; ++s) {
    const CopySeg& g = b.seg[s];  // words of 4 bytes, 16-byte aligned
    const long long v = g.words >> 2;
    for (long long i = tid; i < v; i += T) reinterpret_cast<uint4*>(g.dst)[i] = reinterpret_cast<const uint4*>(g.src)[i];
    for (long long i = 4 * v + tid; i < g.words; i += T) g.dst[i] = g.src[i];
  }
  for (int k = 0; k < 3; ++k) {
    const SlotView &f = b.from[k], &t = b.to[k];
    if (!f.cnt) continue;
    for (long long A = tid; A < b.n; A += T) {
      const int c = f.cnt[A];
      t.cnt[A] = c;
      for (size_t j = A * f.cap; j < (size_t)A * f.cap + min(c, f.cap); ++j) {
        t.id[j] = f.id[j];
        t.seg_start[j] = f.seg_start[j];
        t.seg_cnt[j] = f.seg_cnt[j];
      }
    }
  }
}
void launch_backup(const BackupArgs& b, cudaStream_t s) {
  long long m = b.n;
  for (int k = 0; k < b.nseg; ++k) m = std::max(m, b.seg[k].words / 4);
  if (m > 0) k_backup<<<(unsigned)std::min<long long>((m + 255) / 256, num_sms() * 8), 256, 0, s>>>(b);
}

// ---------------------------------------------------------------------------
// Box distance helpers for conservative culling (body frame).
LD double box_dist(double3 l, double3 lo, double3 hi) {
  double dx = fmax(fmax(lo.x - l.x, l.x - hi.x), 0.0);
  double dy = fmax(fmax(lo.y - l.y, l.y - hi.y), 0.0);
  double dz = fmax(fmax(lo.z - l.z, l.z - hi.z), 0.0);
  return sqrt(dx * dx + dy * dy + dz * dz);
}
LD void grid_box(const double3 o, double invh, int3 gs, double3& lo, double3& hi) {
  lo = o;
  hi = d3(o.x + (gs.x - 1) / invh, o.y + (gs.y - 1) / invh, o.z + (gs.z - 1) / invh);
}

// True when no point within `reach` of l (wall frame) that lies in wall w's grid
// box can have phi <= 0, so that no node of a particle of that bounding radius can
// pass the wall's SDF test (sdf_eval rejects nodes outside the box, and inside it
// the interpolated phi is positive). q is l's grid position projected onto the
// box; for a node position p in the box |p - q| <= |p - l| (projection onto a
// convex set does not expand distances), the segment p-q stays in the box, and
// along it phi changes by at most the template's cell gradient-norm bound per
// grid unit (lip[3 sh + 1] spacings per spacing). phi(q) is the FP64 trilinear
// value of the grid, as the node test computes it, with a rounding margin.
LD bool wall_far(const StepArgs& a, int w, double3 l, double reach) {
  const int sh = a.W.shape[w];
  const int3 gs = a.S.gsize[sh];
  const double invh = a.W.invh[w];
  const double3 o = a.W.origin[w];
  const double qx = fmin(fmax((l.x - o.x) * invh, 0.0), (double)(gs.x - 1));
  const double qy = fmin(fmax((l.y - o.y) * invh, 0.0), (double)(gs.y - 1));
  const double qz = fmin(fmax((l.z - o.z) * invh, 0.0), (double)(gs.z - 1));
  const int i0 = min((int)qx, gs.x - 2), j0 = min((int)qy, gs.y - 2), k0 = min((int)qz, gs.z - 2);
  const double fx = qx - i0, fy = qy - j0, fz = qz - k0;
  const int sy = gs.x, sz = gs.x * gs.y;
  const double* b = a.S.sdf + a.S.sdf_off[sh] + ((size_t)k0 * sz + (size_t)j0 * sy + i0);
  const double sc = a.W.scale[w];
  double cmax = 0.0, acc = 0.0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {  // the four x-edges of the cell
    const int dy = e & 1, dz = e >> 1;
    const double* be = b + dz * sz + dy * sy;
    const double v0 = __ldg(be), v1 = __ldg(be + 1);
    cmax = fmax(cmax, fmax(fabs(v0), fabs(v1)));
    acc += (v0 * (1.0 - fx) + v1 * fx) * (dy ? fy : 1.0 - fy) * (dz ? fz : 1.0 - fz);
  }
  const double phi = sc * acc;
  const double bound = (double)a.S.lip[3 * sh + 1] * reach * (1.0 + 1e-9) + 1e-12 * sc * cmax + 1e-300;
  return phi > bound;
}

// Entry of a flat pair list: A * cap + slot in 32 bits, unsigned (alloc_slots bounds it).
LD int pair_code(int A, int cap, int slot) { return (int)((unsigned)A * cap + slot); }

// Appends this lane's entries (A, j), j < cnt, to a flat pair list, with
// one atomic per warp (all lanes of the warp call it).
LD void append_pairs(int* list, int* ctr, int A, int cap, int cnt) {
  const int lane = threadIdx.x & 31;
  int incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += v;
  }
  const int tot = __shfl_sync(FULL, incl, 31);
  int base = 0;
  if (lane == 31 && tot > 0) base = atomicAdd(ctr, tot);
  base = __shfl_sync(FULL, base, 31) + incl - cnt;
  for (int j = 0; j < cnt; ++j) list[base + j] = pair_code(A, cap, j);
}

// Centres and bounding radii in a sorted order (idx), FP32, for the candidate
// walks (the particle grid's, then the image search's).
__global__ void k_pack_cells(StepArgs a, const int* __restrict__ idx) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < a.P.n) pack_cell(a, k, idx[k]);
}

// ---------------------------------------------------------------------------
// Support tables and the separation test of a candidate pair.
// The support of a point set P, h(w) = max over p in P of w . p, is convex and
// positively homogeneous in w. A direction u falls on one face of a cube map (the axis
// of its largest |component|, m = that |component|), where w = u / m = (+-1, p, q) in
// the face's coordinates (gnomonic square [-1, 1]^2, SUP_M x SUP_M cells). Restricted
// to the face's plane, h is convex in (p, q), so on each half of a cell (the triangles
// below and above its (p + 1, q) - (p, q + 1) diagonal) it lies below the linear
// interpolation of its values at the triangle's corners. The tables hold, per shape,
// those values at the cube map's vertices (rounded up), packed four per cell; the
// support along the unit direction u / |u| is h(w) m / |u|. Sets: the template's
// surface nodes (sup_n) and the solid, every point where B's trilinear phi is <= 0 (sup_s).

// Face coordinates of vertex (i, j) of face f as an unnormalised direction.
LD double3 sup_vertex(int f, int i, int j) {
  const double sg = (f & 1) ? -1.0 : 1.0;
  const double p = -1.0 + 2.0 * i / SUP_M, q = -1.0 + 2.0 * j / SUP_M;
  return f < 2 ? d3(sg, p, q) : (f < 4 ? d3(q, sg, p) : d3(p, q, sg));
}

// One warp per (shape, table, vertex): the largest projection, rounded up.
//
// Solid: pts holds the corners c of every grid cell with a point of phi = 0 (or of phi <= 0
// on the grid's boundary), and phi_c. A point x of such a cell with phi(x) <= 0 has
// w . x <= w . x - l phi(x) for every l >= 0, and the right side is trilinear on the cell, so
// its maximum is at a corner: the support of the solid along w is at most
// max over c of (w . c - l phi_c). l = 0 is the projection of the cells themselves, up to a
// spacing beyond the surface. For the signed distance of a convex body and l = |w| every term
// is at most the body's own support (its distance outside is at least w . c / |w| - h, and
// inside the ball of radius -phi_c about c is in it), so the bound has no dilation at all; other
// fields take the best of the few l tried. (Corners of a grid refined by two, l = 0, stood
// half a spacing off: settling configuration of 2M particles, 225k pairs kept per step
// against 25k.)
__constant__ double SUP_L[8] = {0.0, 0.5, 0.7, 0.85, 1.0, 1.2, 1.5, 2.5};
__global__ void k_support_vertices(int nshapes, const double3* __restrict__ node_pos, const int* __restrict__ node_off,
                                   const int* __restrict__ node_cnt, const double4* __restrict__ pts,
                                   const long long* __restrict__ pts_off, float* __restrict__ vtx,
                                   float* __restrict__ sup_r, int* __restrict__ sup_t) {
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= 2LL * nshapes * SUP_VERTS) return;
  const int sh = (int)(w / (2 * SUP_VERTS)), tab = (int)((w / SUP_VERTS) & 1), v = (int)(w % SUP_VERTS);
  const int f = v / ((SUP_M + 1) * (SUP_M + 1)), j = (v / (SUP_M + 1)) % (SUP_M + 1), i = v % (SUP_M + 1);
  const double3 c = sup_vertex(f, i, j);
  double mx = -1e300, slack = 0.;
  if (tab == 0) {
    for (int k = lane; k < node_cnt[sh]; k += 32) mx = fmax(mx, dot(c, node_pos[node_off[sh] + k]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
  } else {
    const double lw = len(c);
    double m[8], mag[2] = {0., 0.};  // largest |w| |c| and |w| |phi_c|
    for (int q = 0; q < 8; ++q) m[q] = -1e300;
    for (long long k = pts_off[sh] + lane; k < pts_off[sh + 1]; k += 32) {
      const double4 p = pts[k];
      const double wc = c.x * p.x + c.y * p.y + c.z * p.z;
#pragma unroll
      for (int q = 0; q < 8; ++q) m[q] = fmax(m[q], wc - SUP_L[q] * lw * p.w);
      mag[0] = fmax(mag[0], sqrt(p.x * p.x + p.y * p.y + p.z * p.z));
      mag[1] = fmax(mag[1], fabs(p.w));
    }
    for (int o = 16; o > 0; o >>= 1) {
      for (int q = 0; q < 8; ++q) m[q] = fmax(m[q], __shfl_xor_sync(FULL, m[q], o));
      for (int q = 0; q < 2; ++q) mag[q] = fmax(mag[q], __shfl_xor_sync(FULL, mag[q], o));
    }
    mx = 1e300;
    for (int q = 0; q < 8; ++q) {
      // covers the rounding of these sums and of the node test's interpolated phi
      const double e = 1e-11 * lw * (mag[0] + SUP_L[q] * mag[1]);
      if (m[q] + e < mx + slack) { mx = m[q]; slack = e; }
    }
    // the largest |p| of the solid: at a corner of its cells
    if (v == 0 && lane == 0) sup_r[sh] = __double2float_ru(mag[0] * (1.0 + 1e-9));
    // The largest |p| of the solid itself. For p along u = sum l_i v_i (l_i >= 0, v_i the vertices of
    // u's triangle) |p| = u . p <= sum l_i h(v_i) <= max(h(v) / |v|) sum l_i |v_i|, and the last sum is at
    // most 1 / cos(0.1179) = 1.0070, a cell of the cube map being 1 / 12 wide at distance 1 or more.
    if (lane == 0 && mx > 0.) atomicMax(&sup_t[sh], __float_as_int(__double2float_ru((mx + slack) / lw * 1.0071)));
  }
  // relative 1e-9 covers the rounding of the dot products and of the vertex coordinates
  if (lane == 0) vtx[w] = mx > -1e299 ? __double2float_ru(mx + slack + 1e-9 * fabs(mx) + 1e-30) : -1e30f;
}

// One thread per (shape, table, cell): its four corner values in one float4.
__global__ void k_support_pack(int nshapes, const float* __restrict__ vtx, float4* __restrict__ sup_n,
                               float4* __restrict__ sup_s) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2LL * nshapes * SUP_CELLS) return;
  const int sh = (int)(t / (2 * SUP_CELLS)), tab = (int)((t / SUP_CELLS) & 1), cell = (int)(t % SUP_CELLS);
  const int f = cell / (SUP_M * SUP_M), j = (cell / SUP_M) % SUP_M, i = cell % SUP_M;
  const float* V = vtx + ((size_t)sh * 2 + tab) * SUP_VERTS + (size_t)f * (SUP_M + 1) * (SUP_M + 1);
  const float4 c = make_float4(V[j * (SUP_M + 1) + i], V[j * (SUP_M + 1) + i + 1], V[(j + 1) * (SUP_M + 1) + i],
                               V[(j + 1) * (SUP_M + 1) + i + 1]);
  (tab == 0 ? sup_n : sup_s)[(size_t)sh * SUP_CELLS + cell] = c;
}

void launch_support_tables(int nshapes, const double3* node_pos, const int* node_off, const int* node_cnt,
                           const double4* pts, const long long* pts_off, float* vtx, float4* sup_n, float4* sup_s,
                           float* sup_r, float* sup_t, cudaStream_t s) {
  const long long warps = 2LL * nshapes * SUP_VERTS;
  if (warps <= 0) return;
  k_support_vertices<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(nshapes, node_pos, node_off, node_cnt, pts,
                                                                         pts_off, vtx, sup_r, reinterpret_cast<int*>(sup_t));
  const long long cells = 2LL * nshapes * SUP_CELLS;
  k_support_pack<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(nshapes, vtx, sup_n, sup_s);
}

// Candidate partners of each particle A.
// Particle partners: B > A, visible (in a cell), bounding spheres within
// reach (|xA - xB| <= rA + rB is necessary for any node of A to pass the
// reference's |node - xB| <= rB test, which in turn implies B lies in the
// node's 27-cell window since cells are at least 2 max radius wide). The test
// runs on the FP32 copies (reach_f), so the candidates are a superset of the
// exact ones; the narrowphase decides every node exactly. A pair that some direction
// separates (pair_separated) has no node of A inside B and is dropped.
// Wall partners: visible walls whose SDF grid box the bounding sphere reaches and
// whose interpolated phi is not provably positive over it (wall_far).

// FP32 copy of a wall's grid box for a first cull: axes (rows of the inverse rotation), centre
// and half extents in the world and wall frames, and the error bound that goes with them. Every
// particle is tested against every wall, nearly always far off; in FP64 that test was a third
// of the search of 2M settling particles.
struct WallBox {
  float m[9];
  float c[3], h[3];
  float e;
};
static constexpr int WALLS_SH = 16;  // walls with a copy in shared memory
LD void load_wall_box(const StepArgs& a, int w, WallBox& b) {
  double3 lo, hi;
  grid_box(a.W.origin[w], a.W.invh[w], a.S.gsize[a.W.shape[w]], lo, hi);
  const Quat q = a.W.quat[w];
  const double3 u[3] = {rotate(q, d3(1., 0., 0.)), rotate(q, d3(0., 1., 0.)), rotate(q, d3(0., 0., 1.))};
  const double3 mid = 0.5 * (lo + hi), half = 0.5 * (hi - lo), c = a.W.pos[w] + rotate(q, mid);
  for (int k = 0; k < 3; ++k) {
    b.m[3 * k] = (float)u[k].x; b.m[3 * k + 1] = (float)u[k].y; b.m[3 * k + 2] = (float)u[k].z;
  }
  b.c[0] = (float)c.x; b.c[1] = (float)c.y; b.c[2] = (float)c.z;
  b.h[0] = (float)half.x; b.h[1] = (float)half.y; b.h[2] = (float)half.z;
  // roundings of c and h (2^-24 each) and of the rotation, taken tenfold; the box's own size
  // covers a quaternion that is off unit length by less than 1e-6
  b.e = 4e-6f * (fabsf(b.c[0]) + fabsf(b.c[1]) + fabsf(b.c[2]) + b.h[0] + b.h[1] + b.h[2]);
}
// True when the ball (x, r) cannot reach the box.
LD bool wall_box_far(const WallBox& b, float3 x, float r) {
  const float dx = x.x - b.c[0], dy = x.y - b.c[1], dz = x.z - b.c[2];
  const float n1 = fabsf(x.x) + fabsf(x.y) + fabsf(x.z);
  float d2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float l = fabsf(fmaf(b.m[3 * k], dx, fmaf(b.m[3 * k + 1], dy, b.m[3 * k + 2] * dz)));
    const float o = fmaxf(l - b.h[k], 0.f);
    d2 = fmaf(o, o, d2);
  }
  const float R = r * (1.0f + 1e-5f) + b.e + 4e-6f * n1;
  return d2 > R * R * (1.0f + 1e-5f);
}

// Wall partners of particle A (few), in wall order; returns how many there are.
LD int wall_candidates(const StepArgs& a, const WallBox* box, int A, double3 xA, double rA) {
  const int capw = a.pw.cap;
  int nw = 0;
  for (int w = 0; w < a.W.n; ++w) {
    if (w < WALLS_SH && wall_box_far(box[w], make_float3((float)xA.x, (float)xA.y, (float)xA.z), (float)rA)) continue;
    if (a.W.key[w] < 0) continue;
    const double3 l = rotate_inv(xA - a.W.pos[w], a.W.quat[w]);
    double3 lo, hi;
    grid_box(a.W.origin[w], a.W.invh[w], a.S.gsize[a.W.shape[w]], lo, hi);
    const double reach = rA * (1.0 + 1e-9) + coord_slack(xA, a.W.pos[w]) + 1e-12 * len(hi - lo);
    if (box_dist(l, lo, hi) > reach) continue;
    if (wall_far(a, w, l, reach)) continue;
    if (nw < capw) a.pw.id[(size_t)A * capw + nw] = w;
    ++nw;
  }
  if (capw > 0) a.pw.cnt[A] = nw < capw ? nw : capw;
  if (nw > capw) atomicOr(&a.status->flags, OVF_WALL);
  return nw;
}

// End of a candidate kernel (all lanes of the warp): the flat pair lists, the largest demands,
// one atomic per warp.
LD void candidates_done(const StepArgs& a, int A, bool on, int n, int nw) {
  append_pairs(a.pl.list[0], &a.pl.ctr[0], A, a.pp.cap, on ? min(n, a.pp.cap) : 0);
  if (a.pw.cap > 0) append_pairs(a.pl.list[1], &a.pl.ctr[1], A, a.pw.cap, on ? min(nw, a.pw.cap) : 0);
  n = __reduce_max_sync(FULL, n);
  nw = __reduce_max_sync(FULL, nw);
  if ((threadIdx.x & 31) == 0) {
    if (n > 0) atomicMax(&a.status->need_pp, n);
    if (nw > 0) atomicMax(&a.status->need_wall, nw);
  }
}

// Slots of A in ascending (cell key, index) order, the walk's.
LD void order_slots(const StepArgs& a, int* out, int n) {
  for (int u = 1; u < n; ++u) {
    const int B = out[u], kb = a.P.key[B];
    int v = u - 1;
    for (; v >= 0; --v) {
      const int C = out[v], kc = a.P.key[C];
      if (kc < kb || (kc == kb && C < B)) break;
      out[v + 1] = C;
    }
    out[v + 1] = B;
  }
}

// Candidates from the neighbour lists (k_rebuild, neighbours.cu): per particle A the bodies
// B > A that the step's tests may find, in (cell key, index) order at the build. A pair of a
// step is a listed one whose cell is in the window of A's cell, whose spheres reach and that no
// direction separates; the slots are in the order of the present (key, index), the walk's.
//
// The warp's list entries are tested one lane per entry, whoever owns it: a particle has 0 to 4
// of them, so a lane testing its own would leave most lanes idle. Everything is in particle
// order, so that only the partners' records are gathered. A warp takes PER particles: as many
// as leave half the resident warps busy, since with lists this short (0.3 entries a particle
// in the settling configuration) a round of the warp's lanes is filled by a hundred of them
// (2M settling particles: 221 us with 32, 135 us with 128).
//
// Walls: with 8 particles a warp, a lane per particle would leave three of four lanes without
// a wall to test, after the pairs' chain of loads; the walls take blocks of their own there,
// all lanes busy, beside the pairs' (2000 bodies over a floor: 39.8 -> 39.0 us a step; 12k
// bonded ones 61.5 -> 60.0). With 32 and more, every lane has a particle and the pairs' blocks
// fill the chip, so that they test the walls themselves.
template <int PER>
__global__ void __launch_bounds__(128) k_candidates(StepArgs a) {
  constexpr int Q = PER < 32 ? 1 : PER / 32;  // particles per lane: t0 + lane + 32 q
  __shared__ int s_pre[4][PER + 1];           // exclusive counts of the warp's entries
  __shared__ int s_cnt[4][PER];               // candidates found
  __shared__ WallBox s_wall[WALLS_SH];
  const int lane = threadIdx.x & 31;
  int* pre = s_pre[threadIdx.x >> 5];
  int* cnt = s_cnt[threadIdx.x >> 5];
  const int t0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * PER;
  if (PER < 32 && t0 >= a.P.n) {
    // a small system's walls, in blocks of their own beside the pairs': one lane per particle
    const int A = (blockIdx.x - (a.P.n + 4 * PER - 1) / (4 * PER)) * blockDim.x + threadIdx.x;
    if (blockIdx.x * 4 * PER < (unsigned)a.P.n) return;  // the last pair block's idle warps
    if ((int)threadIdx.x < min(a.W.n, WALLS_SH)) load_wall_box(a, threadIdx.x, s_wall[threadIdx.x]);
    __syncthreads();
    const bool on = A < a.P.n;
    const int nw = on ? wall_candidates(a, s_wall, A, a.P.pos[A], a.P.radius[A]) : 0;
    candidates_done(a, A, on, 0, nw);
    return;
  }
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  const int cap = a.pp.cap;
  int total = 0;
  {
    int listed[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int A = t0 + lane + 32 * q;
      listed[q] = lane < PER && A < a.P.n ? min(max(a.nbr_cnt[A], 0), a.nbr_cap) : 0;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      int incl = listed[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane < PER) {
        pre[lane + 32 * q] = total + incl - listed[q];
        cnt[lane + 32 * q] = 0;
      }
      total += __shfl_sync(FULL, incl, 31);
    }
    if (lane == 0) pre[PER] = total;
  }
  unsigned moved[Q];  // this lane's owners one of whose partners changed its place in the order
#pragma unroll
  for (int q = 0; q < Q; ++q) moved[q] = 0;
  __syncwarp();
  for (int i0 = 0; i0 < total; i0 += 32) {
    const int i = i0 + lane;
    int ow = 0;  // the owner of entry i: the last whose exclusive count does not exceed it
#pragma unroll
    for (int o = PER / 2; o > 0; o >>= 1)
      if (pre[ow + o] <= i) ow += o;
    const int first = pre[ow], j = i - first, oA = t0 + ow;
    bool keep = false, after = true;
    int B = -1, kA = -1, kB = -1;
    CandRec ra, rb;
    if (i < total) {
      B = __ldg(a.nbr + (size_t)j * a.P.n + oA);
      ra = cand_rec(a, oA, kA);
      rb = cand_rec(a, B, kB);
    }
    const int pB = __shfl_up_sync(FULL, B, 1), pk = __shfl_up_sync(FULL, kB, 1);
    if (i < total) {
      if (j > 0) {
        const int C = lane > 0 ? pB : __ldg(a.nbr + (size_t)(j - 1) * a.P.n + oA);
        const int kC = lane > 0 ? pk : a.P.key[C];
        after = kC < kB || (kC == kB && C < B);
      }
      const float n1a = n1_f(ra.p), R = reach_f(ra.p, n1a, rb.p);
      if (kB >= 0 && kB < a.pg.ncells && !(dist2_f(ra.p, rb.p) > __fmul_rn(R, R))) {
        const int sx = a.pg.size.x, sy = a.pg.size.y;
        const int3 c = kA >= 0 && kA < a.pg.ncells ? make_int3(kA % sx, (kA / sx) % sy, kA / (sx * sy))
                                                   : clamp_cell(cell_of(a.P.pos[oA], a.pg), a.pg.size);
        const int bx = kB % sx, by = (kB / sx) % sy, bz = kB / (sx * sy);
        keep = abs(bx - c.x) <= 1 && abs(by - c.y) <= 1 && abs(bz - c.z) <= 1 &&
               !pair_separated(sup, ra.p, n1a, ra.q, ra.sc, ra.sh, rb.p, rb.q, rb.sc, rb.sh);
      }
    }
    const unsigned m = __ballot_sync(FULL, keep);
    const int at = cnt[ow] + __popc(m & lanemask_lt() & (~0u << max(min(first - i0, 31), 0)));
    if (keep && at < cap) a.pp.id[(size_t)oA * cap + at] = B;
    const int nx = __shfl_down_sync(FULL, ow, 1);
    __syncwarp();
    if (i < total && (lane == 31 || nx != ow || i + 1 == total)) cnt[ow] = at + keep;
    if (__any_sync(FULL, !after)) {
#pragma unroll
      for (int q = 0; q < Q; ++q) moved[q] |= __reduce_or_sync(FULL, !after && (ow >> 5) == q ? 1u << (ow & 31) : 0u);
    }
    __syncwarp();
  }
  const bool walls = PER >= 32 && a.W.n > 0;
  if (walls) {
    if ((int)threadIdx.x < min(a.W.n, WALLS_SH)) load_wall_box(a, threadIdx.x, s_wall[threadIdx.x]);
    __syncthreads();
  }
#pragma unroll 1
  for (int q = 0; q < Q; ++q) {
    const int A = t0 + lane + 32 * q;
    const bool on = lane < PER && A < a.P.n;
    int n = 0, nw = 0;
    if (on) {
      n = cnt[lane + 32 * q];
      if (((moved[q] >> lane) & 1u) && n <= cap) order_slots(a, a.pp.id + (size_t)A * cap, n);
      a.pp.cnt[A] = n < cap ? n : cap;
      if (n > cap) atomicOr(&a.status->flags, OVF_PP);
      if (walls) nw = wall_candidates(a, s_wall, A, a.P.pos[A], a.P.radius[A]);
    }
    candidates_done(a, A, on, n, nw);
  }
}

// Candidates without neighbour lists: every step sorts the cells and walks the 27 of each
// particle. One thread per particle, threads in cell-sorted order: the lanes of a warp
// mostly share a cell, so they walk the same cells (z, y, x order) in step and their occupant
// loads are broadcasts. The walk visits the cells of the window in ascending key order and
// the occupants of a cell in ascending index (stable sort), so its partners come in ascending
// (cell key, index) order.
// The bounding-sphere test fills the slots with sorted positions (the first SLOT_SH of a
// particle in shared memory, the rest in their place in global memory); the separation test
// then runs over the warp's filled slots with one lane per pair, whoever owns it (a particle
// has 0 to 4 of them, so a lane testing its own would leave most lanes idle), and each lane
// compacts what is left of its own slots, in order.
static constexpr int SLOT_SH = 8;
LD bool pair_separated_at(const SupTabs& sup, const float4* pk, const int4* meta, const float4* q, int t, int k) {
  const float4 pa = pk[t], pb = pk[k];
  const int4 ma = meta[t], mb = meta[k];
  return pair_separated(sup, pa, __fadd_rn(__fadd_rn(fabsf(pa.x), fabsf(pa.y)), fabsf(pa.z)), q[t],
                        __int_as_float(ma.w), ma.z, pb, q[k], __int_as_float(mb.w), mb.z);
}
// Out of line, for the rare particle whose slots are full.
__device__ __noinline__ bool pair_separated_call(SupTabs sup, const float4* pk, const int4* meta, const float4* q, int t,
                                                 int k) {
  return pair_separated_at(sup, pk, meta, q, t, k);
}

__global__ void __launch_bounds__(128) k_candidates_walk(StepArgs a) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, t0 = t - lane;
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  const int cap = a.pp.cap;
  __shared__ int s_slot[4][32][SLOT_SH + 1];
  __shared__ WallBox s_wall[WALLS_SH];
  if ((int)threadIdx.x < min(a.W.n, WALLS_SH)) load_wall_box(a, threadIdx.x, s_wall[threadIdx.x]);
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  auto slot = [&](int owner, int A, int j) -> int& {
    return j < SLOT_SH ? s_slot[warp][owner][j] : a.pp.id[(size_t)A * cap + j];
  };
  int n = 0, nw = 0, A = 0;
  int fixed = 0;  // leading slots whose pairs have been tested already
  int extra = 0;  // pairs that found no slot
  double3 xA = d3(0., 0., 0.);
  double rA = 0.;
  int* out = a.pp.id;
  if (t < a.P.n) {
    A = a.cell_idx[t];
    xA = a.P.pos[A];
    rA = a.P.radius[A];
    out = a.pp.id + (size_t)A * cap;
    const float4 pa = a.cell_pk[t];
    const float n1a = __fadd_rn(__fadd_rn(fabsf(pa.x), fabsf(pa.y)), fabsf(pa.z));
    // when the slots are full the pairs in them are tested at once to make room
    auto push = [&](int k) {
      if (n < cap) {
        slot(lane, A, n++) = k;
        return;
      }
      int w = fixed;
#pragma unroll 1
      for (int j = fixed; j <= n; ++j) {
        const int kj = j < n ? slot(lane, A, j) : k;
        if (pair_separated_call(sup, a.cell_pk, a.pk_meta, a.pk_q, t, kj)) continue;
        if (w < cap) slot(lane, A, w++) = kj;
        else ++extra;
      }
      n = fixed = w;
    };
    const int3 c = clamp_cell(cell_of(xA, a.pg), a.pg.size);
    // the (up to) 3 cells of a row along x are contiguous in the sorted order
    const int x0 = max(c.x - 1, 0), x1 = min(c.x + 1, a.pg.size.x - 1);
    for (int z = max(c.z - 1, 0); z <= min(c.z + 1, a.pg.size.z - 1); ++z) {
      for (int y = max(c.y - 1, 0); y <= min(c.y + 1, a.pg.size.y - 1); ++y) {
        const int h0 = lin3(make_int3(x0, y, z), a.pg.size);
        const int st = __ldg(a.cell_off + h0 + 1), en = __ldg(a.cell_off + h0 + (x1 - x0) + 2);
#pragma unroll 2
        for (int k = st; k < en; ++k) {
          const float4 pb = __ldg(a.cell_pk + k);  // read-only: loads may run ahead of the slot stores
          const float R = reach_f(pa, n1a, pb);
          if (dist2_f(pa, pb) > __fmul_rn(R, R)) continue;
          if (a.pk_meta[k].y <= A) continue;
          push(k);
        }
      }
    }
  }
  // separation test, one lane per filled slot of the warp
  int incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  __syncwarp();
  for (int i0 = 0; i0 < total; i0 += 32) {
    const int i = i0 + lane;
    const int ow = lane_of(incl, i);
    const int j = i - (__shfl_sync(FULL, incl, ow) - __shfl_sync(FULL, n, ow));
    const int oA = __shfl_sync(FULL, A, ow), ofix = __shfl_sync(FULL, fixed, ow);
    if (i < total) {
      int& o = slot(ow, oA, j);
      const int k = o;
      int B = a.pk_meta[k].y;
      if (j >= ofix && pair_separated_at(sup, a.cell_pk, a.pk_meta, a.pk_q, t0 + ow, k)) B = -1;
      o = B;
    }
  }
  __syncwarp();
  if (t < a.P.n) {
    int w = 0;
    for (int j = 0; j < n; ++j) {
      const int B = slot(lane, A, j);
      if (B >= 0) out[w++] = B;
    }
    n = w + extra;
    a.pp.cnt[A] = n < cap ? n : cap;
    if (n > cap) atomicOr(&a.status->flags, OVF_PP);
    nw = wall_candidates(a, s_wall, A, xA, rA);
  }
  candidates_done(a, A, t < a.P.n, n, nw);
}

void launch_candidates(const StepArgs& a, cudaStream_t s) {
  if (a.P.n <= 0) return;
  if (a.nbr) {
    const int half = num_sms() * 10;  // warps
    if (a.P.n >= half * 128) k_candidates<128><<<(a.P.n + 511) / 512, 128, 0, s>>>(a);
    else if (a.P.n >= half * 32) k_candidates<32><<<(a.P.n + 127) / 128, 128, 0, s>>>(a);
    else k_candidates<8><<<(a.P.n + 31) / 32 + (a.W.n > 0 ? (a.P.n + 127) / 128 : 0), 128, 0, s>>>(a);
    return;
  }
  k_pack_cells<<<(a.P.n + 255) / 256, 256, 0, s>>>(a, a.cell_idx);
  k_candidates_walk<<<(a.P.n + 127) / 128, 128, 0, s>>>(a);
}

// ---------------------------------------------------------------------------
// Narrowphase.
enum { KIND_PP = 0, KIND_WALL = 1, KIND_GHOST = 2 };

// Position of the owner of a pair: image pairs take the wrapped one where the step's wrap has
// yet to be done.
template <int KIND>
LD double3 owner_pos(const StepArgs& a, int A) {
  const double3 x = a.P.pos[A];
  return KIND == KIND_GHOST && a.wrap_axes ? wrap_pos(x, a.pg, a.wrap_axes) : x;
}

// The owner particle A of the warp.
struct SelfCtx {
  double3 x, v, w;
  Quat q;
  double sc;
  int n0, nn, cl0, ncl;
};

// Contact constants of one pair (contactKernel.cu:99-104 / :176-179 and the damping
// terms of LinearContact, contactKernel.cuh:50-58), evaluated once per pair.
struct PairK {
  double kn, ks, mu, cn, cs;
};

// The SDF side of a test.
struct Partner {
  double3 x;        // centre
  Quat q;
  double r;         // bounding radius (particle partners)
  double3 o;        // grid origin (body frame)
  double invh;
  int3 gs;
  const double* sdf;
  double sc;        // SDF value scale
  int key;          // cell key (walls: wall grid, ghosts: particle grid)
  int real;         // particle index receiving the reaction (-1: none)
  double3 v, w;     // velocity, angular velocity
  double invm, kn, ks, mu, res;
};

template <int KIND>
LD Partner load_partner(const StepArgs& a, int pid) {
  Partner P;
  if (KIND == KIND_WALL) {
    const BodyView& W = a.W;
    P.x = W.pos[pid]; P.q = W.quat[pid]; P.r = W.radius[pid];
    P.o = W.origin[pid]; P.invh = W.invh[pid];
    const int sh = W.shape[pid];
    P.gs = a.S.gsize[sh]; P.sdf = a.S.sdf + a.S.sdf_off[sh]; P.sc = W.scale[pid];
    P.key = W.key[pid]; P.real = -1;
    P.v = W.vel[pid]; P.w = W.angvel[pid];
    P.invm = 0.; P.kn = 0.; P.ks = 0.; P.mu = W.mu[pid]; P.res = W.res[pid];
  } else {
    const BodyView& B = a.P;
    int i = pid, set = 0;
    if (KIND == KIND_GHOST) { i = pid >> 3; set = pid & 7; }
    if (KIND == KIND_GHOST) {
      P.x = a.G.gpos[(size_t)set * B.n + i];
      P.key = a.G.gkey[(size_t)set * B.n + i];
    } else {
      P.x = B.pos[i];
      P.key = B.key[i];
    }
    P.q = B.quat[i]; P.r = B.radius[i];
    P.o = B.origin[i]; P.invh = B.invh[i];
    const int sh = B.shape[i];
    P.gs = a.S.gsize[sh]; P.sdf = a.S.sdf + a.S.sdf_off[sh]; P.sc = B.scale[i];
    P.real = i;
    P.v = B.vel[i]; P.w = B.angvel[i];
    if (KIND == KIND_GHOST && a.G.sector) {
      // rotated image: its own orientation and velocity; the angular velocity stays the
      // particle's (addGhostLevelSetParticleContactForceTorqueKernel, contactKernel.cu:240-242)
      P.q = a.G.gquat[(size_t)set * B.n + i];
      P.v = a.G.gvel[(size_t)set * B.n + i];
    }
    P.invm = B.invmass[i]; P.kn = B.kn[i]; P.ks = B.ks[i]; P.mu = B.mu[i]; P.res = B.res[i];
  }
  return P;
}

LD double3 node_world(const StepArgs& a, const SelfCtx& S, int ni) {
  const double3 nl = a.S.node_pos[S.n0 + ni] * S.sc;
  return rotate(S.q, nl) + S.x;
}

// Trilinear SDF evaluation at world point w (LSParticleContactDetectionKernel.cu:63-115,
// interpolateLevelSetFunctionValue .cuh:4-32). True when inside the grid with overlap >= 0.
LD bool sdf_eval(double3 w, const Partner& P, double& ov, double& fx, double& fy, double& fz, double* c) {
  const double3 l = rotate_inv(w - P.x, P.q);
  const double gx = (l.x - P.o.x) * P.invh;
  const double gy = (l.y - P.o.y) * P.invh;
  const double gz = (l.z - P.o.z) * P.invh;
  const int i0 = (int)floor(gx), j0 = (int)floor(gy), k0 = (int)floor(gz);
  if (i0 < 0 || j0 < 0 || k0 < 0) return false;
  if (i0 >= P.gs.x - 1 || j0 >= P.gs.y - 1 || k0 >= P.gs.z - 1) return false;
  fx = gx - (double)i0;
  fy = gy - (double)j0;
  fz = gz - (double)k0;
  const int sx = 1, sy = P.gs.x, sz = P.gs.x * P.gs.y;
  const double* b = P.sdf + (k0 * sz + j0 * sy + i0);
  c[0] = P.sc * __ldg(b);
  c[1] = P.sc * __ldg(b + sx);
  c[2] = P.sc * __ldg(b + sy);
  c[3] = P.sc * __ldg(b + sy + sx);
  c[4] = P.sc * __ldg(b + sz);
  c[5] = P.sc * __ldg(b + sz + sx);
  c[6] = P.sc * __ldg(b + sz + sy);
  c[7] = P.sc * __ldg(b + sz + sy + sx);
  const double wx0 = 1.0 - fx, wx1 = fx, wy0 = 1.0 - fy, wy1 = fy, wz0 = 1.0 - fz, wz1 = fz;
  const double phi = c[0] * wx0 * wy0 * wz0 + c[1] * wx1 * wy0 * wz0 + c[2] * wx0 * wy1 * wz0 +
                     c[3] * wx1 * wy1 * wz0 + c[4] * wx0 * wy0 * wz1 + c[5] * wx1 * wy0 * wz1 +
                     c[6] * wx0 * wy1 * wz1 + c[7] * wx1 * wy1 * wz1;
  ov = -phi;
  return ov >= 0.;
}

// Gradient in grid units (interpolateLevelSetFunctionGradient, .cuh:34-77).
LD double3 sdf_grad(double fx, double fy, double fz, const double* c, int flags) {
  const double x = (flags & FIX_GRADIENT) ? fx : (double)(int)fx;
  const double wx0 = 1.0 - x, wx1 = x, wy0 = 1.0 - fy, wy1 = fy, wz0 = 1.0 - fz, wz1 = fz;
  const double gx = (c[1] - c[0]) * wy0 * wz0 + (c[3] - c[2]) * wy1 * wz0 + (c[5] - c[4]) * wy0 * wz1 +
                    (c[7] - c[6]) * wy1 * wz1;
  const double gy = (c[2] - c[0]) * wx0 * wz0 + (c[3] - c[1]) * wx1 * wz0 + (c[6] - c[4]) * wx0 * wz1 +
                    (c[7] - c[5]) * wx1 * wz1;
  const double gz = (c[4] - c[0]) * wx0 * wy0 + (c[5] - c[1]) * wx1 * wy0 + (c[6] - c[2]) * wx0 * wy1 +
                    (c[7] - c[3]) * wx1 * wy1;
  return d3(gx, gy, gz);
}

// Exact per-node admission test of the reference for each partner kind.
template <int KIND>
LD bool node_admitted(const StepArgs& a, double3 w, const Partner& P) {
  if (KIND == KIND_PP) {
    const double3 r = w - P.x;
    return !(len2(r) > P.r * P.r);
  } else {
    int3 c, lo, hi;
    node_window(w, KIND == KIND_WALL ? a.wg : a.pg, c, lo, hi);
    return in_window(P.key, KIND == KIND_WALL ? a.wg : a.pg, c, lo, hi);
  }
}

LD double sqrt_damp(double v, int flags) { return (flags & FIX_SQRTF) ? sqrt(v) : (double)sqrtf((float)v); }

template <int KIND>
LD PairK pair_constants(const StepArgs& a, int A, const Partner& P) {
  const double invmA = a.P.invmass[A], knA = a.P.kn[A], ksA = a.P.ks[A], muA = a.P.mu[A], resA = a.P.res[A];
  double kn = 0., ks = 0., effM = 0., mu, res;
  if (KIND == KIND_WALL) {
    kn = knA; ks = ksA;
    if (invmA > 0.) effM = 1. / invmA;
    mu = fmin(muA, P.mu);
    res = fmin(resA, P.res);
  } else {
    if (knA > 0. && P.kn > 0.) kn = knA * P.kn / (knA + P.kn);
    if (ksA > 0. && P.ks > 0.) ks = ksA * P.ks / (ksA + P.ks);
    if (invmA > 0. || P.invm > 0.) effM = 1. / (invmA + P.invm);
    res = fmin(resA, P.res);
    mu = fmin(muA, P.mu);
  }
  const double logRes = log(res);
  const double diss = -logRes / sqrt_damp(logRes * logRes + M_PI * M_PI, a.flags);
  PairK k;
  k.kn = kn; k.ks = ks; k.mu = mu;
  k.cn = 2. * diss * sqrt_damp(effM * kn, a.flags);
  k.cs = 2. * diss * sqrt_damp(effM * ks, a.flags);
  return k;
}

// integrateSlidingSpring + LinearContact (contactKernel.cuh:4-77) with the pair constants.
LD void linear_contact(double3& F, double3& spring, double3 vc, double3 n, double delta, double dt, const PairK& k) {
  if (delta > 0.) {
    const double3 vn = dot(vc, n) * n;
    const double3 fn = k.kn * delta * n - k.cn * vn;
    const double3 vs = vc - vn;
    double3 s = d3(0., 0., 0.);
    if (k.mu > 0. && k.ks > 0.) {
      double3 p1 = spring - dot(spring, n) * n;
      const double a1 = len(p1);
      if (!is_zero(a1)) p1 *= len(spring) / a1;
      s = p1 + vs * dt;
      double3 fs = -k.ks * s - k.cs * vs;
      const double afs = len(fs), afn = len(fn);
      if (!is_zero(afs) && afs > k.mu * afn) {
        const double ratio = k.mu * afn / afs;
        fs *= ratio;
        s = -(fs + k.cs * vs) / k.ks;
      }
    }
    spring = s;
    const double3 fsl = -k.ks * spring - k.cs * vs;
    F = fn + fsl;
  } else {
    spring = d3(0., 0., 0.);
    F = d3(0., 0., 0.);
  }
}

template <int KIND>
LD const SlotView& slots_of(const StepArgs& a, bool old) {
  if (KIND == KIND_PP) return old ? a.pp_old : a.pp;
  if (KIND == KIND_WALL) return old ? a.pw_old : a.pw;
  return old ? a.pgh_old : a.pgh;
}

// Contact geometry, carried-over spring and linear contact force of one
// admitted node (LSParticleContactDetectionKernel.cu:63-115, contactKernel.cu:75-117 /
// :155-190 / :225-270); writes the contact at pos.
LD void contact_node(const StepArgs& a, const SelfCtx& S, const Partner& P, const PairK& K, int ni, int ostart,
                     int ocnt, int rank, int pos, bool can_write, double3& FA, double3& TA, double3& FB, double3& TB) {
  const double3 w = node_world(a, S, ni);
  double ov, fx, fy, fz, cr[8];
  sdf_eval(w, P, ov, fx, fy, fz, cr);
  double3 n = sdf_grad(fx, fy, fz, cr, a.flags);
  n = rotate(P.q, n);
  n = normalize_dev(n);
  const double3 pc = w + 0.5 * ov * n;
  // carried-over spring: search of node ni in the old segment (sorted by node), outwards from its
  // rank in the new one, where it mostly still is, then by halves
  double3 spring = d3(0., 0., 0.);
  int lo = 0, hi = ocnt - 1, mid = min(rank, hi), away = 1;
  bool below = false, above = false;
  while (lo <= hi) {
    const int v = a.C_old.node[ostart + mid];
    if (v == ni) { spring = a.C_old.spring[ostart + mid]; break; }
    if (v < ni) { lo = mid + 1; below = true; } else { hi = mid - 1; above = true; }
    if (below && above) mid = (lo + hi) >> 1;
    else { mid = below ? min(hi, mid + away) : max(lo, mid - away); away *= 4; }
  }
  const double3 vc = S.v + cross(S.w, pc - S.x) - (P.v + cross(P.w, pc - P.x));
  double3 F;
  linear_contact(F, spring, vc, n, ov, a.dt, K);
  if (can_write) {
    a.C.node[pos] = ni;
    a.C.spring[pos] = spring;
    if (a.C.point) {
      a.C.point[pos] = pc;
      a.C.normal[pos] = n;
      a.C.overlap[pos] = ov;
      a.C.en_n[pos] = 0.5 * ov * ov * K.kn;
      a.C.en_s[pos] = 0.5 * len2(spring) * K.ks;
    }
  }
  FA += F;
  TA += cross(pc - S.x, F);
  FB -= F;
  TB += cross(pc - P.x, -F);
}

// ---------------------------------------------------------------------------
// Certified FP32 screening.
//
// Almost every node the narrowphase visits is rejected (outside the partner's
// bounding sphere or cell window, or phi > 0). Those rejections are made in FP32,
// in the precision forms against SDF templates stored as phi / h in FP16 or BF16, in
// the FP64 form against the FP64 templates, and a node is rejected only when error
// bounds prove that the FP64 test (k_contacts_f) rejects it too. Every node the screen
// cannot reject is decided by that test, and every contact is evaluated in FP64. Pair
// lists, contact segments and forces of all forms are therefore the same; the 16-bit
// store only makes the rejections cheaper. (The FP64 form ran its cluster cull and node test
// in FP64, one warp per owner at 255 registers, with no cull by phi: a step of a bed of 20,000
// bodies took 961 us that way and takes 392 us.)
//
// Per pair, the owner's node offsets n (template units) map to the partner's
// frame by l = M n + dB, M = R_B^T R_A scale_A, dB = R_B^T (xA - xB), and to its
// grid by g = l invh + cg, cg = -origin invh. M and dB are formed in FP32 from
// the pair's FP32 rotation matrices (each entry rounded once from FP64) and from
// xA - xB rounded from FP64.
//
// Error bounds (unit roundoff u = 2^-24; |.|_1 norms bound the Euclidean ones):
// l carries at most ~10u (N1 + |d|_1) of rounding, N1 = sqrt(3) x the largest
// node distance x scale_A, and g adds u |g|_1 + invh u |origin|_1; EPS_F = 1.6e-5
// (~270u) bounds all of it with a wide margin: el = EPS_F (N1 + 2 |d|_1) in
// length, eg = invh (el + EPS_F |origin|_1) + EPS_F (sizes summed) in grid units
// per axis. The corners c differ from the FP64 values v by at most
// Q |v| (Q = 2^-11 for FP16, 2^-8 for BF16, round to nearest, plus the FP32
// rounding of phi / h and of the interpolation; these alone, below 16u, from the FP64
// templates); an error eg in the grid point
// moves the piecewise-trilinear phi / h by at most 3 L eg, L = the largest
// difference of neighbouring grid values of the partner's template in spacings;
// and every corner of the cell lies within 3 L of the interpolated value. So
// with Q' = Q / (1 - Q), the FP64 phi at the FP64 point is positive whenever the
// interpolated 16-bit value exceeds
//   T = (3 L Q' + 3 L eg + 1e-7) / (1 - Q'),
// a constant of the pair: a node is rejected by one comparison.
LD float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
LD float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
LD float3 tof(double3 v) { return f3((float)v.x, (float)v.y, (float)v.z); }
LD double3 tod(float3 v) { return d3(v.x, v.y, v.z); }

static constexpr float EPS_F = 1.6e-5f;
static constexpr float PHI_BAND = (float)LIP_BAND;

// relative bound of the 16-bit store and FP32 interpolation error (with margin)
template <int SDFK>
LD constexpr float quant16() {
  return SDFK == PREC_FP32_BF16 ? 3.95e-3f + 1e-6f : (SDFK == PREC_FP32_FP16 ? 4.95e-4f + 1e-6f : 2e-6f);
}

// Constants of one screened pair.
struct PairF {
  float M[9];        // R_B^T R_A scale_A, row-major
  float3 dB;         // R_B^T (xA - xB)
  float3 cg;         // -origin invh
  float invh;
  float ux, uy, uz;  // grid size - 1 per axis
  float R2;          // particle partners: admission radius (with margin), squared
  float rB;          // particle partners: bounding radius
  float el;          // position error bound in the partner frame (length)
  float eg;          // grid-point error bound per axis (grid units)
  float T;           // rejection threshold of phi / h
  float Tq;          // 1 / (1 - Q')
  float gmax;        // gradient-norm bound of phi / h per grid unit
  float gband;       // the same over the cells where phi / h takes values in [0, PHI_BAND]
  int sy, sz;        // cell strides
  const uint4* cells;
  const double* sdf; // FP64 form: grid values, their factor ih to phi / h (strides sy, sz of the grid)
  float ih;
  // the owner
  int A, slot, n0, nn, cl0, ncl;  // particle, slot; first node, nodes, first cluster, clusters
  float scA;
};
// Walls and images: the partner's cell key, R_A scale_A (world offsets of the nodes), their error
// bound, the owner's position.
template <bool WIN>
struct PairWin {};
template <>
struct PairWin<true> {
  int key;
  float RA[9];
  float n1w;
  double3 xA;
};
// Learned SDF: u = l * ms - mc (network input), phi / h = y * mtoh, threshold Tn.
template <bool LRN>
struct PairNet {};
template <>
struct PairNet<true> {
  float ms, mtoh, Tn;
  float3 mc;
  int pshape;
};
template <bool WIN, bool LRN>
struct PairX : PairF, PairWin<WIN>, PairNet<LRN> {};

template <int KIND>
LD int partner_shape(const StepArgs& a, int pid) {
  if (KIND == KIND_WALL) return a.W.shape[pid];
  return a.P.shape[KIND == KIND_GHOST ? (pid >> 3) : pid];
}

template <int KIND, int SDFK, bool WIN, bool LRN>
LD void make_pair_f(const StepArgs& a, int A, int slot, int pid, PairX<WIN, LRN>& F) {
  const Partner P = load_partner<KIND>(a, pid);
  const int pshape = partner_shape<KIND>(a, pid);
  // R_A and R_B (row-major), rotated in FP64 and rounded
  float ra[9], rb[9];
  const Quat qA = a.P.quat[A];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double3 u = d3(j == 0 ? 1. : 0., j == 1 ? 1. : 0., j == 2 ? 1. : 0.);
    const double3 ca = rotate(qA, u), cb = rotate(P.q, u);
    ra[j] = (float)ca.x; ra[3 + j] = (float)ca.y; ra[6 + j] = (float)ca.z;
    rb[j] = (float)cb.x; rb[3 + j] = (float)cb.y; rb[6 + j] = (float)cb.z;
  }
  const int shA = a.P.shape[A];
  const float scA = (float)a.P.scale[A];
  // M = R_B^T R_A scale_A
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j)
      F.M[3 * i + j] = fmaf(rb[i], ra[j], fmaf(rb[3 + i], ra[3 + j], rb[6 + i] * ra[6 + j])) * scA;
  const double3 xA = owner_pos<KIND>(a, A);
  const float3 df = tof(xA - P.x);
  F.dB = f3(fmaf(rb[0], df.x, fmaf(rb[3], df.y, rb[6] * df.z)), fmaf(rb[1], df.x, fmaf(rb[4], df.y, rb[7] * df.z)),
            fmaf(rb[2], df.x, fmaf(rb[5], df.y, rb[8] * df.z)));
  F.invh = (float)P.invh;
  F.cg = tof(-1.0 * P.o * P.invh);
  F.ux = (float)(P.gs.x - 1); F.uy = (float)(P.gs.y - 1); F.uz = (float)(P.gs.z - 1);
  const float N1 = 1.7320508f * (float)a.S.node_box[8 * shA + 6] * scA;
  const float n1d = fabsf(df.x) + fabsf(df.y) + fabsf(df.z);
  const float el = EPS_F * (N1 + 2.0f * n1d);
  F.el = el;
  F.rB = (float)P.r;
  const float R = F.rB * (1.0f + 1e-6f) + el;
  F.R2 = R * R * (1.0f + 1e-6f);
  const float eg = F.invh * (el + EPS_F * (fabsf(F.cg.x) + fabsf(F.cg.y) + fabsf(F.cg.z)) / F.invh) +
                   EPS_F * (float)(P.gs.x + P.gs.y + P.gs.z);
  F.eg = eg;
  const float L = a.S.lip[3 * pshape];
  const float Q = quant16<SDFK>();
  const float Qp = Q / (1.0f - Q);
  F.Tq = 1.0f / (1.0f - Qp);
  F.T = (3.0f * L * Qp + 3.0f * L * eg + 1e-7f) * F.Tq * (1.0f + 1e-5f);
  F.gmax = a.S.lip[3 * pshape + 1];
  F.gband = a.S.lip[3 * pshape + 2];
  if (SDFK == PREC_FP64) {
    F.sy = P.gs.x;
    F.sz = P.gs.x * P.gs.y;
    F.sdf = P.sdf;
    F.ih = (float)(P.invh * P.sc);  // 1 / template spacing
  } else {
    F.sy = P.gs.x - 1;
    F.sz = (P.gs.x - 1) * (P.gs.y - 1);
    F.cells = a.S.cell16 + a.S.cell_off[pshape];
  }
  F.A = A;
  F.slot = slot;
  F.scA = scA;
  F.n0 = a.S.node_off[shA]; F.nn = a.S.node_cnt[shA];
  F.cl0 = a.S.cl_off[shA]; F.ncl = a.S.cl_cnt[shA];
  if constexpr (WIN) {
    F.key = P.key;
    for (int k = 0; k < 9; ++k) F.RA[k] = ra[k] * scA;
    F.n1w = EPS_F * N1;
    F.xA = xA;
  }
  if constexpr (LRN) {
    F.pshape = pshape;
    // partner frame (length) -> template units (/ scale) -> network input
    const MlpNorm nm = a.mlp_norm[pshape];
    const double ht = 1.0 / (P.invh * P.sc);  // template spacing
    F.ms = (float)(1.0 / (P.sc * nm.R));
    F.mc = f3(nm.cx / nm.R, nm.cy / nm.R, nm.cz / nm.R);
    F.mtoh = (float)(nm.R / ht);
    F.Tn = a.mlp_band[pshape];
  }
}

LD float3 mulf(const float* M, float x, float y, float z) {
  return f3(fmaf(M[0], x, fmaf(M[1], y, M[2] * z)), fmaf(M[3], x, fmaf(M[4], y, M[5] * z)),
            fmaf(M[6], x, fmaf(M[7], y, M[8] * z)));
}

// Interpolated phi / h of the 16-bit store at grid point g, which must lie in
// [0, size - 1) on every axis: one 16-byte load of the cell's corners.
template <int SDFK>
LD float2 unpack16(unsigned w) {
  if (SDFK == PREC_FP32_BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <int SDFK>
LD float phi16_interp(uint4 w, float gx, float gy, float gz) {
  const float fx = gx - floorf(gx), fy = gy - floorf(gy), fz = gz - floorf(gz);
  const float2 c01 = unpack16<SDFK>(w.x), c23 = unpack16<SDFK>(w.y);
  const float2 c45 = unpack16<SDFK>(w.z), c67 = unpack16<SDFK>(w.w);
  const float x0 = fmaf(fx, c01.y - c01.x, c01.x), x1 = fmaf(fx, c23.y - c23.x, c23.x);
  const float x2 = fmaf(fx, c45.y - c45.x, c45.x), x3 = fmaf(fx, c67.y - c67.x, c67.x);
  const float y0 = fmaf(fy, x1 - x0, x0), y1 = fmaf(fy, x3 - x2, x2);
  return fmaf(fz, y1 - y0, y0);
}
// The cell's corners (one 16-byte load) and the interpolation, split so that the load
// can be issued early.
LD uint4 phi16_cell(const uint4* cells, int sy, int sz, float gx, float gy, float gz) {
  const int i0 = __float2int_rd(gx), j0 = __float2int_rd(gy), k0 = __float2int_rd(gz);
  return __ldg(cells + (k0 * sz + j0 * sy + i0));
}
template <int SDFK>
LD float phi16_at(const uint4* cells, int sy, int sz, float gx, float gy, float gz) {
  return phi16_interp<SDFK>(phi16_cell(cells, sy, sz, gx, gy, gz), gx, gy, gz);
}
template <int SDFK>
LD float phi16(const PairF& F, float gx, float gy, float gz) {
  if (SDFK == PREC_FP64) {
    const int i0 = __float2int_rd(gx), j0 = __float2int_rd(gy), k0 = __float2int_rd(gz);
    const double* b = F.sdf + (k0 * F.sz + j0 * F.sy + i0);
    const float fx = gx - floorf(gx), fy = gy - floorf(gy), fz = gz - floorf(gz);
    float c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = (float)__ldg(b + (k & 1) + (k & 2 ? F.sy : 0) + (k & 4 ? F.sz : 0));
    const float x0 = fmaf(fx, c[1] - c[0], c[0]), x1 = fmaf(fx, c[3] - c[2], c[2]);
    const float x2 = fmaf(fx, c[5] - c[4], c[4]), x3 = fmaf(fx, c[7] - c[6], c[6]);
    const float y0 = fmaf(fy, x1 - x0, x0), y1 = fmaf(fy, x3 - x2, x2);
    return fmaf(fz, y1 - y0, y0) * F.ih;
  }
  return phi16_at<SDFK>(F.cells, F.sy, F.sz, gx, gy, gz);
}

// Cell-window admission of walls and images from the FP32 world node offset ra
// (error bound e): 0 = certainly rejected, 1 = certainly admitted, 2 = the FP64
// node may lie in a neighbouring cell (within e of a cell boundary).
template <int KIND>
LD int window_state(const StepArgs& a, double3 x, float3 ra, float e0, int key) {
  const GridP& g = KIND == KIND_WALL ? a.wg : a.pg;
  const double3 w = x + tod(ra);
  const double e = (double)e0 + 1e-14 * (fabs(w.x) + fabs(w.y) + fabs(w.z));
  const double ux = (w.x - g.mn.x) * g.inv.x, uy = (w.y - g.mn.y) * g.inv.y, uz = (w.z - g.mn.z) * g.inv.z;
  if (fabs(ux - rint(ux)) <= e * g.inv.x + 1e-9 || fabs(uy - rint(uy)) <= e * g.inv.y + 1e-9 ||
      fabs(uz - rint(uz)) <= e * g.inv.z + 1e-9)
    return 2;
  int3 c, lo, hi;
  node_window(w, g, c, lo, hi);
  return in_window(key, g, c, lo, hi) ? 1 : 0;
}

// FP32 screen of one node (offset nd, template units): false only when the
// FP64 test (k_contacts_f) certainly rejects it.
template <int KIND, int SDFK, class FX>
LD bool node_may_hit_f(const StepArgs& a, const FX& F, float4 nd, bool& looked) {
  const float3 l = mulf(F.M, nd.x, nd.y, nd.z) + F.dB;
  if constexpr (KIND == KIND_PP) {
    if (l.x * l.x + l.y * l.y + l.z * l.z > F.R2) return false;
  } else {
    if (window_state<KIND>(a, F.xA, mulf(F.RA, nd.x, nd.y, nd.z), F.n1w, F.key) == 0) return false;
  }
  const float gx = fmaf(l.x, F.invh, F.cg.x), gy = fmaf(l.y, F.invh, F.cg.y), gz = fmaf(l.z, F.invh, F.cg.z);
  // the FP64 test rejects g < 0 or g >= size - 1 on any axis
  const float lo = fminf(gx, fminf(gy, gz));
  const float hi = fmaxf(gx - F.ux, fmaxf(gy - F.uy, gz - F.uz));
  if (lo < -F.eg || hi >= F.eg) return false;
  if (lo < F.eg || hi >= -F.eg) return true;  // within the error of the grid boundary
  looked = true;
  return !(phi16<SDFK>(F, gx, gy, gz) > F.T);  // NaN never rejects
}

// Cluster cull (sphere of radius rad about the cluster centre cn, template
// units): false only when no node of the cluster can pass the FP64 test.
//  - particle partners: the sphere misses the partner's bounding sphere;
//  - the sphere misses the partner's grid box (nodes outside it fail the SDF test);
//  - phi / h at q, the centre projected into the box shrunk by m >= eg, exceeds
//    the cluster's reach: for a node p inside the box, |p - q| <= |p - c| +
//    sqrt(3) m (projection onto a convex set does not expand distances), the
//    segment p-q lies in the box, and along it phi / h changes by at most gmax
//    per grid unit, so phi(q) - gmax (rad + sqrt(3) m) > 0 proves phi > 0 at
//    every node of the cluster. On the way down to phi = 0 the last stretch from
//    min(phi(q), PHI_BAND) lies in cells where phi / h takes values in [0, PHI_BAND], so
//    when the distance times their bound gband is below PHI_BAND, gband serves in place of
//    gmax, which the medial surface sets (1.73 against 1.15 for a rounded box, 1.14 against
//    1.07 for an ellipsoid).
//  With up != nullptr (learned form), *up receives an estimate of the largest phi / h
//  over the cluster's nodes (phi at q plus gmax times the reach; +inf when phi at q is
//  not looked up): where it is below the network's rejection threshold the network would
//  reject a node only by overestimating phi there, so the nodes are not sent to it (an
//  efficiency choice only: every node the network does not see takes the grid test).
template <int KIND, int SDFK>
LD bool cluster_may_hit_f(const PairF& F, float4 cn, float scA, float* up = nullptr) {
  if (up) *up = INFINITY;
  const float3 l = mulf(F.M, cn.x, cn.y, cn.z) + F.dB;
  const float rad = cn.w * scA * (1.0f + 1e-6f);
  if (KIND == KIND_PP) {
    const float R = F.rB * (1.0f + 1e-6f) + rad + F.el;
    if (l.x * l.x + l.y * l.y + l.z * l.z > R * R * (1.0f + 1e-6f)) return false;
  }
  const float gx = fmaf(l.x, F.invh, F.cg.x), gy = fmaf(l.y, F.invh, F.cg.y), gz = fmaf(l.z, F.invh, F.cg.z);
  const float radh = rad * F.invh;
  const float dx = fmaxf(fmaxf(-gx, gx - F.ux), 0.f), dy = fmaxf(fmaxf(-gy, gy - F.uy), 0.f),
              dz = fmaxf(fmaxf(-gz, gz - F.uz), 0.f);
  const float Rb = (radh + F.eg) * (1.0f + 1e-6f);
  if (dx * dx + dy * dy + dz * dz > Rb * Rb) return false;
  const float m = fmaxf(F.eg, 1e-3f);  // > 0: q stays below size - 1, so its cell is in the grid
  if (F.ux < 4.f * m || F.uy < 4.f * m || F.uz < 4.f * m) return true;
  const float qx = fminf(fmaxf(gx, m), F.ux - m), qy = fminf(fmaxf(gy, m), F.uy - m),
              qz = fminf(fmaxf(gz, m), F.uz - m);
  const float dist = radh + 2.8f * m;
  const float g = F.gband * dist * (1.0f + 1e-6f) < PHI_BAND ? F.gband : F.gmax;
  const float reach = (g * dist + 1e-6f) * F.Tq * (1.0f + 1e-6f);
  const float ph = phi16<SDFK>(F, qx, qy, qz);
  if (up) *up = ph + reach;
  return !(ph > F.T + reach);
}


// Screens one (A, partner) pair: cluster cull, then the node screen over the
// surviving clusters. The nodes the screen cannot reject are written, in node
// order, to the precision-form node buffer and the pair is queued for
// k_contacts_f; a pair without such nodes gets its empty contact segment here.
template <int KIND, int SDFK, bool LRN, bool STATS, class FX>
LD void screen_pair_f(const StepArgs& a, const FX& F, int li, unsigned char* s_cl, unsigned short* s_sub, unsigned* s_mask,
                      unsigned* s_dir, unsigned (&cnt)[8], unsigned& queued) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the previous pair's write pass may still read s_cl / s_mask
  const int A = F.A, slot = F.slot, n0 = F.n0, nn = F.nn, cl0 = F.cl0, ncl = F.ncl;
  const float scA = F.scA;
  int nsurv = 0;
  for (int c0 = 0; c0 < ncl; c0 += 32) {
    const int c = c0 + lane;
    bool keep = false;
    if (c < ncl) keep = cluster_may_hit_f<KIND, SDFK>(F, __ldg(a.S.cl_sphere_f + cl0 + c), scA);
    const unsigned m = __ballot_sync(FULL, keep);
    if (keep) s_cl[nsurv + __popc(m & lanemask_lt())] = (unsigned char)c;
    nsurv += __popc(m);
  }
  __syncwarp();
  // second level: sub-clusters of 8 nodes of the surviving clusters, compacted in
  // ascending order; chunk k of the node loop is sub-clusters 4k .. 4k + 3. Learned
  // form: bit 15 marks a sub-cluster whose phi / h estimate is below the network's
  // threshold; its nodes take the grid test here instead of the network.
  int nsub = 0;
  for (int j0 = 0; j0 < 4 * nsurv; j0 += 32) {
    const int j = j0 + lane;
    bool keep = false;
    int sid = 0;
    if (j < 4 * nsurv) {
      sid = s_cl[j >> 2] * 4 + (j & 3);
      const float4 sp = __ldg(a.S.sub_sphere + 4 * cl0 + sid);
      float up = INFINITY;
      keep = sp.w >= 0.f && cluster_may_hit_f<KIND, SDFK>(F, sp, scA, LRN ? &up : nullptr);
      if constexpr (LRN)
        if (up <= F.Tn) sid |= 0x8000;
    }
    const unsigned m = __ballot_sync(FULL, keep);
    if (keep) s_sub[nsub + __popc(m & lanemask_lt())] = (unsigned short)sid;
    nsub += __popc(m);
  }
  const int nch = (nsub + 3) >> 2;
  if (STATS) { cnt[0] += 1; cnt[1] += ncl; cnt[2] += nsurv; cnt[7] += nsub; }
  __syncwarp();
  // this lane's node in chunk k (nn when none)
  auto node_of = [&](int k) {
    const int j = 4 * k + (lane >> 3);
    if (j >= nsub) return nn;
    const int ni = (s_sub[j] & 0x7fff) * 8 + (lane & 7);
    return ni < nn ? ni : nn;
  };
  int total = 0;
  if constexpr (LRN) {
    // Learned form: the nodes the partner's bounds cannot reject go to the network of the
    // partner's shape (k_net_screen, tensor cores), which decides with the grid test of
    // the nodes it keeps, unless their sub-cluster is marked (then the grid test runs
    // here). A pair with network nodes records all its remaining nodes in node order as
    // pending (the marked ones with a passing verdict already; k_net_compact queues the
    // survivors for the FP64 pass); a pair without takes the plain screen's tail.
    const NetView& Q = a.net[li];
    int tnet = 0, tdir = 0;
    for (int k = 0; k < nch; ++k) {
      const int ni = node_of(k);
      const int j = 4 * k + (lane >> 3);
      const bool marked = j < nsub && (s_sub[j] & 0x8000);
      if (STATS) cnt[4] += __popc(__ballot_sync(FULL, ni < nn));
      bool need = false, may = false, looked = false;
      if (ni < nn) {
        const float4 nd = __ldg(a.S.node_pos_f + n0 + ni);
        if (marked) {
          may = node_may_hit_f<KIND, SDFK>(a, F, nd, looked);
        } else {
          const float3 l = mulf(F.M, nd.x, nd.y, nd.z) + F.dB;
          bool adm;
          if constexpr (KIND == KIND_PP) adm = !(l.x * l.x + l.y * l.y + l.z * l.z > F.R2);
          else adm = window_state<KIND>(a, F.xA, mulf(F.RA, nd.x, nd.y, nd.z), F.n1w, F.key) != 0;
          const float gx = fmaf(l.x, F.invh, F.cg.x), gy = fmaf(l.y, F.invh, F.cg.y), gz = fmaf(l.z, F.invh, F.cg.z);
          const float lo = fminf(gx, fminf(gy, gz));
          const float hi = fmaxf(gx - F.ux, fmaxf(gy - F.uy, gz - F.uz));
          need = adm && !(lo < -F.eg || hi >= F.eg);
        }
      }
      if (STATS) cnt[3] += __popc(__ballot_sync(FULL, looked));
      const unsigned mn = __ballot_sync(FULL, need), md = __ballot_sync(FULL, may);
      if (lane == 0) {
        s_mask[k] = mn;
        s_dir[k] = md;
      }
      tnet += __popc(mn);
      tdir += __popc(md);
    }
    __syncwarp();
    if (tnet == 0) {
      // no node for the network: the marked nodes that passed go to the FP64 pass as in
      // the plain screen
      for (int k = lane; k < nch; k += 32) s_mask[k] = s_dir[k];
      total = tdir;
      __syncwarp();
    } else {
      const SlotView& cur = slots_of<KIND>(a, false);
      const size_t sidx = (size_t)A * cur.cap + slot;
      if (lane == 0) {  // set here; k_contacts_f writes the segment of a pair with contacts
        cur.seg_start[sidx] = 0;
        cur.seg_cnt[sidx] = 0;
      }
      const int tot = tnet + tdir;
      int pstart = 0, pi = 0;
      bool ok = false;
      if (lane == 0) {
        pstart = atomicAdd(&Q.ctr[0], tot);
        pi = atomicAdd(&Q.ctr[1], 1);
        ok = pstart + tot <= Q.pcap && pi < Q.paircap;
        if (!ok) {
          atomicOr(&a.status->flags, OVF_NET);
          const long long need = (long long)pstart + tot;
          atomicMax(&a.status->need_pend, (int)(need < 0x7fffffff ? need : 0x7fffffff));
        }
      }
      pstart = __shfl_sync(FULL, pstart, 0);
      pi = __shfl_sync(FULL, pi, 0);
      ok = __shfl_sync(FULL, ok, 0);
      if (!ok) return;
      const int sh = F.pshape;
      int off = 0;
      for (int k = 0; k < nch; ++k) {
        const unsigned mn = s_mask[k], md = s_dir[k], m = mn | md;
        if (m == 0u) continue;
        const int ni = node_of(k);
        int base = 0;
        if (lane == 0 && mn) base = atomicAdd(&Q.cnt[sh], __popc(mn));
        base = __shfl_sync(FULL, base, 0);
        if ((m >> lane) & 1u) {
          const int idx = pstart + off + __popc(m & lanemask_lt());
          Q.pend_n[idx] = ni;
          if ((md >> lane) & 1u) {
            Q.pend_v[idx] = 1;
          } else {
            const float4 nd = __ldg(a.S.node_pos_f + n0 + ni);
            const float3 l = mulf(F.M, nd.x, nd.y, nd.z) + F.dB;
            const float gx = fmaf(l.x, F.invh, F.cg.x), gy = fmaf(l.y, F.invh, F.cg.y),
                        gz = fmaf(l.z, F.invh, F.cg.z);
            const float lo = fminf(gx, fminf(gy, gz));
            const float hi = fmaxf(gx - F.ux, fmaxf(gy - F.uy, gz - F.uz));
            const bool edge = lo < F.eg || hi >= -F.eg;
            const int r = base + __popc(mn & lanemask_lt());
            if (r < Q.qcap) {
              float4* row = Q.row + 2 * ((size_t)sh * Q.qcap + r);
              row[0] = make_float4(fmaf(l.x, F.ms, -F.mc.x), fmaf(l.y, F.ms, -F.mc.y), fmaf(l.z, F.ms, -F.mc.z),
                                   __int_as_float(idx | (edge ? (int)0x80000000u : 0)));
              row[1] = make_float4(gx, gy, gz, F.T);
            } else {
              atomicOr(&a.status->flags, OVF_NET);
              atomicMax(&a.status->need_netq, r + 1);
            }
          }
        }
        off += __popc(m);
      }
      if (lane == 0) Q.pair[pi] = make_int4(A, (KIND << 24) | slot, pstart, tot);
      return;
    }
  } else {
    for (int k = 0; k < nch; ++k) {
      const int ni = node_of(k);
      if (STATS) cnt[4] += __popc(__ballot_sync(FULL, ni < nn));
      bool may = false, looked = false;
      if (ni < nn) may = node_may_hit_f<KIND, SDFK>(a, F, __ldg(a.S.node_pos_f + n0 + ni), looked);
      if (STATS) cnt[3] += __popc(__ballot_sync(FULL, looked));
      const unsigned m = __ballot_sync(FULL, may);
      if (lane == 0) s_mask[k] = m;
      total += __popc(m);
    }
  }
  if (STATS) { cnt[5] += total; queued += total; }
  __syncwarp();
  const SlotView& cur = slots_of<KIND>(a, false);
  const size_t sidx = (size_t)A * cur.cap + slot;
  if (total == 0) {
    if (lane == 0) {
      cur.seg_start[sidx] = 0;
      cur.seg_cnt[sidx] = 0;
    }
    return;
  }
  int start = 0;
  bool ok = false;
  if (lane == 0) {
    start = atomicAdd(&a.mb.ctr[0], total);
    const int pi = atomicAdd(&a.mb.ctr[1 + li], 1);
    ok = start + total <= a.mb.cap && pi < a.mb.pcap;
    if (ok) {
      a.mb.pair[(size_t)li * a.mb.pcap + pi] = make_int4(A, (KIND << 24) | slot, start, total);
    } else {
      // the pair index is reserved: mark its entry empty so that the contact pass skips it
      // (the node queue is full; the batch re-runs with grown capacities)
      if (pi < a.mb.pcap) a.mb.pair[(size_t)li * a.mb.pcap + pi] = make_int4(-1, 0, 0, 0);
      atomicOr(&a.status->flags, OVF_QUEUE);
      const long long need = start + total > 2LL * (pi + 1) ? start + total : 2LL * (pi + 1);
      atomicMax(&a.status->need_queue, (int)(need < 0x7fffffff ? need : 0x7fffffff));
    }
    cur.seg_start[sidx] = 0;
    cur.seg_cnt[sidx] = 0;
  }
  start = __shfl_sync(FULL, start, 0);
  ok = __shfl_sync(FULL, ok, 0);
  if (!ok) return;
  int off = 0;
  for (int k = 0; k < nch; ++k) {
    const unsigned m = s_mask[k];
    if ((m >> lane) & 1u) a.mb.node[start + off + __popc(m & lanemask_lt())] = node_of(k);
    off += __popc(m);
  }
}

// A warp takes up to SCREEN_PAIRS pairs at a time: its lanes form their constants (about 350
// instructions of a pair's 1,100 when the whole warp formed them for each), then it screens them one by
// one. The flat pair lists of the kinds in KINDS, in
// particle, wall, image order.
// Particle-only screens fit 64 registers (8 blocks per SM); walls and images
// need the window test's FP64 registers.
static constexpr int SCREEN_PAIRS = 8;
template <int KINDS, int SDFK, bool LRN, bool STATS>
__global__ void __launch_bounds__(NP_WARPS * 32, KINDS == 1 ? 8 : 5) k_screen_f(StepArgs a, int li, int kinds) {
  __shared__ unsigned char s_cl[NP_WARPS][MAXCL];
  __shared__ unsigned short s_sub[NP_WARPS][4 * MAXCL];
  __shared__ unsigned s_mask[NP_WARPS][MAXCL];
  __shared__ unsigned s_dir[NP_WARPS][LRN ? MAXCL : 1];
  __shared__ PairX<KINDS != 1, LRN> s_pair[NP_WARPS][SCREEN_PAIRS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (KINDS & 1) ? a.pl.ctr[0] : 0;
  const int n1 = (kinds & KINDS & 2) && a.pw.cap > 0 ? a.pl.ctr[1] : 0;
  const int n2 = (kinds & KINDS & 4) ? a.pl.ctr[2] : 0;
  const int tot = n0 + n1 + n2;
  unsigned cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // warp-uniform screen counters
  unsigned queued[3] = {0, 0, 0};              // nodes queued by partner kind
  const int W = gridDim.x * NP_WARPS;
  const int per = max(1, min(SCREEN_PAIRS, tot / W));
  for (int e0 = (blockIdx.x * NP_WARPS + warp) * per; e0 < tot; e0 += W * per) {
    __syncwarp();  // the previous pairs' records may still be read
    const int e = e0 + lane;
    if (lane < per && e < tot) {
      auto& F = s_pair[warp][lane];
      if ((KINDS & 1) && e < n0) {
        const unsigned idx = __ldg(a.pl.list[0] + e);
        const int A = idx / a.pp.cap;
        make_pair_f<KIND_PP, SDFK>(a, A, idx - (unsigned)A * a.pp.cap, __ldg(a.pp.id + idx), F);
      } else if ((KINDS & 2) && e < n0 + n1) {
        const unsigned idx = a.pl.list[1][e - n0];
        const int A = idx / a.pw.cap;
        make_pair_f<KIND_WALL, SDFK>(a, A, idx - (unsigned)A * a.pw.cap, a.pw.id[idx], F);
      } else if (KINDS & 4) {
        const unsigned idx = __ldg(a.pl.list[2] + e - n0 - n1);
        const int A = idx / a.pgh.cap;
        make_pair_f<KIND_GHOST, SDFK>(a, A, idx - (unsigned)A * a.pgh.cap, __ldg(a.pgh.id + idx), F);
      }
    }
    __syncwarp();
    for (int p = 0; p < per && e0 + p < tot; ++p) {
      const auto& F = s_pair[warp][p];
      if ((KINDS & 1) && e0 + p < n0) {
        screen_pair_f<KIND_PP, SDFK, LRN, STATS>(a, F, li, s_cl[warp], s_sub[warp], s_mask[warp], s_dir[warp], cnt, queued[0]);
      } else if constexpr ((KINDS & 6) != 0) {
        if ((KINDS & 2) && e0 + p < n0 + n1)
          screen_pair_f<KIND_WALL, SDFK, LRN, STATS>(a, F, li, s_cl[warp], s_sub[warp], s_mask[warp], s_dir[warp], cnt, queued[1]);
        else
          screen_pair_f<KIND_GHOST, SDFK, LRN, STATS>(a, F, li, s_cl[warp], s_sub[warp], s_mask[warp], s_dir[warp], cnt, queued[2]);
      }
    }
  }
  if (STATS && (threadIdx.x & 31) == 0) {
    for (int k = 0; k < 8; ++k)
      if (cnt[k]) atomicAdd(&a.screen_stats[k], (unsigned long long)cnt[k]);
    // grid screen: nodes queued for the FP64 test by partner kind
    for (int k = 0; k < 3; ++k)
      if (!LRN && queued[k]) atomicAdd(&a.screen_stats[8 + k], (unsigned long long)queued[k]);
  }
}

// The partner of a pair whose kind is a value.
LD Partner load_partner_of(const StepArgs& a, int kind, int pid) {
  if (kind == KIND_WALL) return load_partner<KIND_WALL>(a, pid);
  return kind == KIND_GHOST ? load_partner<KIND_GHOST>(a, pid) : load_partner<KIND_PP>(a, pid);
}

// Queued pairs of the screen in FP64: the reference's node test on the screened nodes, then
// each pair's contact segment, history and forces.
//
// A warp takes up to 32 pairs and runs their nodes, then their contacts, one lane each, whichever
// pair they are of. A pair of a bed has 1.5 queued nodes and 0.7 contacts, so that a warp per
// pair left 30 of its lanes idle through a chain of dependent loads, eight warps an SM (100k
// bodies with 336k contacts: 2325 us that way, 150 us now). A warp takes fewer where there are
// not 32 for each, or where pairs have many nodes: at least 64 nodes, on the average. In 32s, bodies
// with faces pressed together, hundreds of contacts a pair, left most warps waiting for a few (100k
// bodies, 4.3M contacts of 115k pairs: 2160 us that way, 1190 us; 8,000 cubes, 5.2M contacts: a step
// of 770 us, 925 with the constants formed for each contact and the old segment searched by halves).
// A pair's constants are formed once, by the lane that has the pair, where the contacts take more than
// one round; in one round, with each contact, beside its loads (2,000 bodies on a floor: 38.9 us a
// step with the constants first, 37.7 this way).
// Between the two runs a pair's hits stand at the front of its part of the node queue, in node
// order; one atomic per warp reserves the segments of its pairs.
__global__ void __launch_bounds__(NP_WARPS * 32, 3) k_contacts_f(StepArgs a, int li) {
  __shared__ int4 s_pair[NP_WARPS][32];   // {A, partner, first node, hits}
  __shared__ int4 s_seg[NP_WARPS][32];    // {segment (-1: does not fit), old segment, its length, kind}
  __shared__ PairK s_cst[NP_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int4* pair = s_pair[warp];
  int4* seg = s_seg[warp];
  PairK* cst = s_cst[warp];
  const int np = min(a.mb.ctr[1 + li], a.mb.pcap);
  if (blockIdx.x == 0 && threadIdx.x == 0)  // this step's demand, for the capacity planning
    atomicMax(&a.status->need_queue, max(a.mb.ctr[0], min(np, 0x3fffffff) * 2));
  const int W = gridDim.x * NP_WARPS;
  int per = 1;
  if (np > W) per = max(1, min(min(32, (np + W - 1) / W), (int)fminf(32.f, 64.f * (float)np / (float)max(1, a.mb.ctr[0]))));
  for (int p0 = (blockIdx.x * NP_WARPS + warp) * per; p0 < np; p0 += W * per) {
    __syncwarp();  // the previous pairs' records are still read
    int4 e = make_int4(-1, 0, 0, 0);  // A < 0: reserved by a pair whose nodes did not fit the queue
    if (lane < per && p0 + lane < np) e = a.mb.pair[(size_t)li * a.mb.pcap + p0 + lane];
    const int kind = e.y >> 24, slot = e.y & 0xffffff;
    const SlotView& cur = kind == KIND_PP ? a.pp : (kind == KIND_WALL ? a.pw : a.pgh);
    const SlotView& old = kind == KIND_PP ? a.pp_old : (kind == KIND_WALL ? a.pw_old : a.pgh_old);
    const size_t sidx = e.x >= 0 ? (size_t)e.x * cur.cap + slot : 0;
    const int pid = e.x >= 0 ? cur.id[sidx] : 0;
    const int cnt = e.x >= 0 ? e.w : 0;
    pair[lane] = make_int4(e.x, pid, e.z, 0);
    seg[lane].w = kind;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    int total = __shfl_sync(FULL, incl, 31);
    __syncwarp();
    for (int i0 = 0; i0 < total; i0 += 32) {
      const int i = i0 + lane;
      const int ow = lane_of(incl, i), first = __shfl_sync(FULL, incl - cnt, ow);
      const int4 pr = pair[ow];
      bool hit = false;
      int ni = 0;
      if (i < total) {
        ni = a.mb.node[pr.z + i - first];
        const int k = seg[ow].w;
        SelfCtx S;
        S.x = a.P.pos[pr.x];
        if (k == KIND_GHOST && a.wrap_axes) S.x = wrap_pos(S.x, a.pg, a.wrap_axes);
        S.q = a.P.quat[pr.x];
        S.sc = a.P.scale[pr.x];
        S.n0 = a.S.node_off[a.P.shape[pr.x]];
        const Partner P = load_partner_of(a, k, pr.y);
        const double3 w = node_world(a, S, ni);
        const bool in = k == KIND_PP ? node_admitted<KIND_PP>(a, w, P)
                                     : (k == KIND_WALL ? node_admitted<KIND_WALL>(a, w, P) : node_admitted<KIND_GHOST>(a, w, P));
        double ov, fx, fy, fz, cr[8];
        hit = in && sdf_eval(w, P, ov, fx, fy, fz, cr);
      }
      const unsigned m = __ballot_sync(FULL, hit);
      const int at = pr.w + __popc(m & lanemask_lt() & (~0u << max(min(first - i0, 31), 0)));
      const int nx = __shfl_down_sync(FULL, ow, 1);
      __syncwarp();
      if (hit) a.mb.node[pr.z + at] = ni;
      if (i < total && (lane == 31 || nx != ow || i + 1 == total)) pair[ow].w = at + hit;
      __syncwarp();
    }
    // segments, and the previous step's of the same pairs
    const int h = pair[lane].w;
    incl = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    total = __shfl_sync(FULL, incl, 31);
    const bool many = total > 32;  // contacts fill more than one round of the lanes
    int base = 0;
    if (lane == 0 && total > 0) base = atomicAdd(a.C.count, total);
    base = __shfl_sync(FULL, base, 0) + incl - h;
    if (e.x >= 0) {
      const bool fits = base + h <= a.C.cap;
      int ostart = 0, ocnt = 0;
      if (h > 0 && old.cnt != nullptr) {
        const int on = min(old.cnt[e.x], old.cap);
        for (int j = 0; j < on; ++j) {
          if (old.id[(size_t)e.x * old.cap + j] != pid) continue;
          ostart = old.seg_start[(size_t)e.x * old.cap + j];
          ocnt = old.seg_cnt[(size_t)e.x * old.cap + j];
          break;
        }
      }
      cur.seg_start[sidx] = base;
      cur.seg_cnt[sidx] = fits ? h : 0;
      if (!fits) atomicOr(&a.status->flags, OVF_CONTACT);
      seg[lane] = make_int4(fits ? base : -1, ostart, ocnt, kind);
      if (h > 0 && many) {
        const Partner P = load_partner_of(a, kind, pid);
        cst[lane] = kind == KIND_WALL ? pair_constants<KIND_WALL>(a, e.x, P) : pair_constants<KIND_PP>(a, e.x, P);
      }
    }
    __syncwarp();
    for (int i0 = 0; i0 < total; i0 += 32) {
      const int i = i0 + lane;
      const int ow = lane_of(incl, i), first = __shfl_sync(FULL, incl - h, ow);
      double3 FA = d3(0., 0., 0.), TA = FA, FB = FA, TB = FA;
      int A = -1, real = -1;
      if (i < total) {
        const int4 pr = pair[ow], sg = seg[ow];
        const int k = sg.w;
        A = pr.x;
        SelfCtx S;
        S.x = a.P.pos[A];
        if (k == KIND_GHOST && a.wrap_axes) S.x = wrap_pos(S.x, a.pg, a.wrap_axes);
        S.v = a.P.vel[A]; S.w = a.P.angvel[A]; S.q = a.P.quat[A];
        S.sc = a.P.scale[A];
        S.n0 = a.S.node_off[a.P.shape[A]];
        const Partner P = load_partner_of(a, k, pr.y);
        const PairK K = many ? cst[ow]
                             : (k == KIND_WALL ? pair_constants<KIND_WALL>(a, A, P) : pair_constants<KIND_PP>(a, A, P));
        contact_node(a, S, P, K, a.mb.node[pr.z + i - first], sg.y, sg.z, i - first, sg.x + i - first, sg.x >= 0, FA, TA, FB, TB);
        // an image of the owner itself takes no reaction
        if (!(k == KIND_GHOST && P.real == A)) real = P.real;
      }
      const int ow0 = __shfl_sync(FULL, ow, 0);
      if (__all_sync(FULL, i >= total || ow == ow0)) {  // one pair: one atomic per component
        FA = warp_sum3(FA); TA = warp_sum3(TA); FB = warp_sum3(FB); TB = warp_sum3(TB);
        if (lane > 0) A = real = -1;
      }
      if (A >= 0) {
        atomic_add3(a.P.force, A, FA);
        atomic_add3(a.P.torque, A, TA);
      }
      if (real >= 0) {
        atomic_add3(a.P.force, real, FB);
        atomic_add3(a.P.torque, real, TB);
      }
    }
  }
}

// Learned form, the network pass of launch li: the queued nodes of each partner shape
// in 128-row tiles on the tensor cores (mlp.cuh), one tile per CTA at a time over a
// persistent grid. A node is kept when phi_net does not exceed the shape's network
// threshold (trust band plus the measured one-sided error, in spacings); a kept node
// then takes the 16-bit grid test of the plain screen (skipped within the error of the
// grid boundary), and its verdict goes to the pair's pending list. If a tensor-core wait
// gives up, the tile's nodes are passed on (no rejection) and the batch reports an error.
template <int SDFK>
__global__ void __launch_bounds__(MLP_TILE) k_net_screen(StepArgs a, int li) {
  extern __shared__ unsigned char dyn[];
  MlpTcSmem* T = mlp_tc_smem(dyn);
  int* s_pre = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(T) + sizeof(MlpTcSmem));
  const NetView& Q = a.net[li];
  const int ns = a.nshapes;
  if (threadIdx.x == 0) {
    int t = 0, mx = 0;
    for (int s = 0; s < ns; ++s) {
      const int c = Q.cnt[s];
      mx = max(mx, c);
      s_pre[s] = t;
      t += (min(c, Q.qcap) + MLP_TILE - 1) / MLP_TILE;
    }
    s_pre[ns] = t;
    if (blockIdx.x == 0) {  // this step's demands, for the capacity planning
      atomicMax(&a.status->need_netq, mx);
      atomicMax(&a.status->need_pend, Q.ctr[0]);
    }
  }
  __syncthreads();
  const int tiles = s_pre[ns];
  if ((int)blockIdx.x >= tiles) return;  // no tensor memory taken
  mlp_tc_setup(T);
  unsigned evals = 0, looks = 0;
  bool ok = true;
  // tile t's shape and this thread's row; the row of the CTA's next tile is loaded while
  // the current one runs
  auto shape_of = [&](int t) {
    int sh = 0;
    while (s_pre[sh + 1] <= t) ++sh;
    return sh;
  };
  auto load_row = [&](int t, int sh, float4& u, float4& g) {
    const int r = (t - s_pre[sh]) * MLP_TILE + threadIdx.x;
    if (t < tiles && r < min(Q.cnt[sh], Q.qcap)) {
      const float4* row = Q.row + 2 * ((size_t)sh * Q.qcap + r);
      u = row[0];
      g = row[1];
    } else {
      u = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
      g = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  int t = blockIdx.x, sh = shape_of(t);
  float4 u, g;
  load_row(t, sh, u, g);
  while (t < tiles && ok) {
    if (T->staged != sh) mlp_tc_stage(T, a.mlp_inf[sh], sh);
    const int tag = __float_as_int(u.w);
    const bool act = tag != -1;
    const bool edge = act && tag < 0;
    const int idx = tag & 0x7fffffff;
    // the grid test's 16-byte cell load is in flight during layer 1 and the MMA; the
    // test is applied only to the nodes the network keeps
    uint4 cell = make_uint4(0u, 0u, 0u, 0u);
    if (act && !edge) {
      const int3 gs = a.S.gsize[sh];
      cell = phi16_cell(a.S.cell16 + a.S.cell_off[sh], gs.x - 1, (gs.x - 1) * (gs.y - 1), g.x, g.y, g.z);
    }
    mlp_tc_layer1(T, u.x, u.y, u.z);
    const float4 gc = g;
    const int tn = t + gridDim.x;
    const int shn = tn < tiles ? shape_of(tn) : sh;
    load_row(tn, shn, u, g);
    ok = mlp_tc_mma(T);
    const float y = mlp_tc_output(T);
    if (act) {
      unsigned char may = 1;
      if (ok && !(y * __ldg(&a.mlp_norm[sh].r_over_h) > __ldg(&a.mlp_band[sh]))) {
        // kept by the network: the plain screen's grid test decides (not within the error
        // of the grid boundary, where the FP64 test decides)
        if (!edge) {
          may = !(phi16_interp<SDFK>(cell, gc.x, gc.y, gc.z) > gc.w);
          ++looks;
        }
      } else if (ok) {
        may = 0;
      }
      Q.pend_v[idx] = may;
      ++evals;
    }
    t = tn;
    sh = shn;
  }
  if (!ok && threadIdx.x == 0) atomicAdd(&a.status->errors, 1);
  if (a.screen_stats) {
    evals = __reduce_add_sync(FULL, evals);
    looks = __reduce_add_sync(FULL, looks);
    if ((threadIdx.x & 31) == 0) {
      if (evals) atomicAdd(&a.screen_stats[6], (unsigned long long)evals);
      if (looks) atomicAdd(&a.screen_stats[3], (unsigned long long)looks);
    }
  }
  mlp_tc_teardown(T, ok);
}

// Learned form, after the network pass of launch li: one warp per pair record, its
// pending nodes with a passing verdict compacted in node order into the FP64 pass's
// node queue, and the pair queued for k_contacts_f (the screen's tail for the plain
// screen).
__global__ void __launch_bounds__(NP_WARPS * 32) k_net_compact(StepArgs a, int li) {
  __shared__ unsigned s_mask[NP_WARPS][MAXCL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const NetView& Q = a.net[li];
  const int np = min(Q.ctr[1], Q.paircap);
  unsigned queued = 0;
  for (int p = blockIdx.x * NP_WARPS + warp; p < np; p += gridDim.x * NP_WARPS) {
    const int4 e = Q.pair[p];
    const int nch = (e.w + 31) >> 5;
    __syncwarp();  // the previous pair may still read s_mask
    int total = 0;
    for (int k = 0; k < nch; ++k) {
      const int j = k * 32 + lane;
      const bool may = j < e.w && Q.pend_v[e.z + j] != 0;
      const unsigned m = __ballot_sync(FULL, may);
      if (lane == 0) s_mask[warp][k] = m;
      total += __popc(m);
    }
    __syncwarp();
    if (total == 0) continue;
    queued += total;
    int start = 0;
    bool ok = false;
    if (lane == 0) {
      start = atomicAdd(&a.mb.ctr[0], total);
      const int pi = atomicAdd(&a.mb.ctr[1 + li], 1);
      ok = start + total <= a.mb.cap && pi < a.mb.pcap;
      if (ok) {
        a.mb.pair[(size_t)li * a.mb.pcap + pi] = make_int4(e.x, e.y, start, total);
      } else {
        if (pi < a.mb.pcap) a.mb.pair[(size_t)li * a.mb.pcap + pi] = make_int4(-1, 0, 0, 0);
        atomicOr(&a.status->flags, OVF_QUEUE);
        const long long need = start + total > 2LL * (pi + 1) ? start + total : 2LL * (pi + 1);
        atomicMax(&a.status->need_queue, (int)(need < 0x7fffffff ? need : 0x7fffffff));
      }
    }
    start = __shfl_sync(FULL, start, 0);
    ok = __shfl_sync(FULL, ok, 0);
    if (!ok) continue;
    int off = 0;
    for (int k = 0; k < nch; ++k) {
      const unsigned m = s_mask[warp][k];
      if ((m >> lane) & 1u) a.mb.node[start + off + __popc(m & lanemask_lt())] = Q.pend_n[e.z + k * 32 + lane] & 0x7fffffff;
      off += __popc(m);
    }
  }
  if (a.screen_stats && lane == 0 && queued) atomicAdd(&a.screen_stats[5], (unsigned long long)queued);
}

bool one_screen(const StepArgs& a) { return a.P.n <= num_sms() * 20; }

template <int KINDS, int SDFK, bool LRN>
void launch_screen_k(const StepArgs& a, int li, int kinds, dim3 g, dim3 b, cudaStream_t s) {
  // the counters' ballots are compiled in only where they are asked for
  if (a.screen_stats) k_screen_f<KINDS, SDFK, LRN, true><<<g, b, 0, s>>>(a, li, kinds);
  else k_screen_f<KINDS, SDFK, LRN, false><<<g, b, 0, s>>>(a, li, kinds);
}

// Learned form: the network pass and the compaction after the screen of launch li.
template <int SDFK>
void launch_net_k(const StepArgs& a, int li, cudaStream_t s) {
  const int smem = (int)(MLP_TC_SMEM + sizeof(int) * (a.nshapes + 1));
  static int attr = 0;  // per kernel instance: the largest dynamic shared memory set so far
  if (smem > attr) {
    cudaFuncSetAttribute(k_net_screen<SDFK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = smem;
  }
  // eight CTAs per SM (8 x 64 = all 512 tensor-memory columns, 8 x 27 KB of shared
  // memory): a CTA that finds no free columns (the other launch's pass beside it) waits
  // in tcgen05.alloc until a CTA on its SM has finished
  k_net_screen<SDFK><<<num_sms() * 8, MLP_TILE, smem, s>>>(a, li);
}
void launch_net_screen(const StepArgs& a, int li, cudaStream_t s) {
  if (!a.mlp_inf || a.P.n <= 0) return;
  if (a.precision == PREC_FP32_FP16) launch_net_k<PREC_FP32_FP16>(a, li, s);
  else launch_net_k<PREC_FP32_BF16>(a, li, s);
}
void launch_net_compact(const StepArgs& a, int li, cudaStream_t s) {
  if (!a.mlp_inf || a.P.n <= 0) return;
  k_net_compact<<<num_sms() * 16, NP_WARPS * 32, 0, s>>>(a, li);
}

// Particle pairs, and wall and image pairs, in two launches: the particle-only screen fits 64
// registers (8 blocks per SM); the others (few) take the window test's FP64 registers.
// A system of no more particles than the warps that are resident at 96 registers takes one
// launch: there a launch counts more than occupancy (2,000 ellipsoids on a floor: 54.3 us per step
// with two, 46.1 us with one).
template <int SDFK, bool LRN>
void launch_screen(const StepArgs& a, int kinds, int li, dim3 g, dim3 b, cudaStream_t s) {
  if ((kinds & 1) && (kinds & 6) && one_screen(a)) {
    launch_screen_k<7, SDFK, LRN>(a, li, kinds, g, b, s);
    return;
  }
  if (kinds & 1) launch_screen_k<1, SDFK, LRN>(a, li, kinds, g, b, s);
  if (kinds & 6) launch_screen_k<6, SDFK, LRN>(a, li, kinds, g, b, s);
}

// The screen over the flat pair lists (launch_contact_pass, in the learned form after
// launch_net_screen and _compact, follows it); the grid is sized for the device, the list length
// is on it.
void launch_narrowphase(const StepArgs& a, int kinds, cudaStream_t s) {
  if (a.P.n <= 0) return;
  // walls and images come on top of a small system's particle pairs
  const dim3 g(std::min((2 * a.P.n + NP_WARPS - 1) / NP_WARPS, num_sms() * 16)), b(NP_WARPS * 32);
  const int li = kinds == 4 && !a.gl.list ? 1 : 0;
  if (a.precision == PREC_FP64) launch_screen<PREC_FP64, false>(a, kinds, li, g, b, s);
  else if (a.precision == PREC_FP32_FP16 && a.mlp_inf) launch_screen<PREC_FP32_FP16, true>(a, kinds, li, g, b, s);
  else if (a.precision == PREC_FP32_FP16) launch_screen<PREC_FP32_FP16, false>(a, kinds, li, g, b, s);
  else if (a.mlp_inf) launch_screen<PREC_FP32_BF16, true>(a, kinds, li, g, b, s);
  else launch_screen<PREC_FP32_BF16, false>(a, kinds, li, g, b, s);
}

void launch_contact_pass(const StepArgs& a, int li, cudaStream_t s) {
  if (a.P.n <= 0) return;
  k_contacts_f<<<num_sms() * 3, NP_WARPS * 32, 0, s>>>(a, li);
}

// ---------------------------------------------------------------------------
// Periodic boundary: wrap along each periodic axis in x, y, z order, each
// single-axis image set taken right after its own axis is wrapped, the
// multi-axis sets after all wraps (mySpatialGrid.cu:28-56, 87-152 and the order
// of PeriodicBoundaryXY2D::updateGhostSpatialGrid, PeriodicBoundary.h:215-288).
// Ghost keys follow calculateGhostHashKernel (mySpatialGrid.cu:214-240),
// including its z-upper test against the y bound.
// Sector periodicity about the z axis through the domain minimum m: a particle
// left of x = m.x (with y >= m.y) is turned by -90 degrees about that axis, one
// below y = m.y (with x >= m.x) by +90 degrees: position about m, velocity and
// orientation (updateVelocityPositionOrientationOutOfSectorKernel, mySpatialGrid.cu:58-85;
// the angular velocity is left as it is, as there). The particle and wall forces of
// the step were evaluated before the wrap with the pre-wrap state, so its force and
// torque turn with it (the reference evaluates them after the wrap, which mixes the
// frames as for translations). Images: a copy per set, turned by 90 degrees when the
// particle is in the first cell row along y, by 270 (-90) degrees when in the first
// cell column along x, and by 180 degrees when in both
// (calculateSectorGhostVelocityPositionOrientationKernel, mySpatialGrid.cu:154-212).
LD void sector_wrap_images(const StepArgs& a, int i, double3& p) {
  const GridP& g = a.pg;
  const int n = a.P.n;
  const double hp = 0.5 * 3.14159265358979323846;
  double3 v = a.P.vel[i];
  Quat q = a.P.quat[i];
  bool turned = false;
  double3 om = d3(0., 0., 0.);
  if (p.x < g.mn.x && p.y >= g.mn.y) {
    om = d3(0., 0., -hp);
    v = rotate_vector_dev(v, om);
    p = g.mn + rotate_vector_dev(p - g.mn, om);
    q = rotate_quaternion_dev(q, om);
    a.P.force[i] = rotate_vector_dev(a.P.force[i], om);
    a.P.torque[i] = rotate_vector_dev(a.P.torque[i], om);
    turned = true;
  }
  if (p.y < g.mn.y && p.x >= g.mn.x) {
    om = d3(0., 0., hp);
    v = rotate_vector_dev(v, om);
    p = g.mn + rotate_vector_dev(p - g.mn, om);
    q = rotate_quaternion_dev(q, om);
    a.P.force[i] = rotate_vector_dev(a.P.force[i], om);
    a.P.torque[i] = rotate_vector_dev(a.P.torque[i], om);
    turned = true;
  }
  if (turned) {
    a.P.vel[i] = v;
    a.P.quat[i] = q;
  }
  double3 gp[3] = {p, p, p}, gv[3] = {v, v, v};
  Quat gq[3] = {q, q, q};
  const double ang[3] = {hp, 2.0 * hp, -hp};  // sets R90, R180, R270
  const int3 c = cell_of(p, g);
  const bool row = c.y == 0, col = c.x == 0;
  for (int s = 0; s < 3; ++s) {
    const bool on = s == 0 ? row : (s == 1 ? row && col : col);
    if (!on) continue;
    const double3 o = d3(0., 0., ang[s]);
    gv[s] = rotate_vector_dev(v, o);
    gp[s] = g.mn + rotate_vector_dev(p - g.mn, o);
    gq[s] = rotate_quaternion_dev(q, o);
  }
  for (int s = 0; s < 3; ++s) {
    a.G.gpos[(size_t)s * n + i] = gp[s];
    a.G.gvel[(size_t)s * n + i] = gv[s];
    a.G.gquat[(size_t)s * n + i] = gq[s];
  }
}

__global__ void k_periodic(StepArgs a, int axes, double3* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.P.n) return;
  const GridP& g = a.pg;
  double3 p = a.P.pos[i];
  const int n = a.P.n;
  for (int ax = 0; ax < 3; ++ax) {
    if (!((axes >> ax) & 1)) continue;
    p = wrap_axis(p, g, ax);
    for (int s = 0; s < a.G.nsets; ++s)
      if (a.G.mask[s] == (1 << ax)) ghost_image(p, g, a.G.mask[s], a.G.gpos[(size_t)s * n + i]);
  }
  if (a.G.sector) {
    sector_wrap_images(a, i, p);
  } else {
    for (int s = 0; s < a.G.nsets; ++s)
      if (__popc(a.G.mask[s]) >= 2) ghost_image(p, g, a.G.mask[s], a.G.gpos[(size_t)s * n + i]);
  }
  for (int s = 0; s < a.G.nsets; ++s) a.G.gkey[(size_t)s * n + i] = ghost_key(a.G.gpos[(size_t)s * n + i], g);
  out[i] = p;
}

// out: where the wrapped positions go (the particles' own positions, or a separate array
// when the images run beside the particle narrowphase, which still reads the pre-wrap ones)
void launch_periodic(const StepArgs& a, int axes, double3* out, cudaStream_t s) {
  if (a.P.n > 0) k_periodic<<<(a.P.n + 255) / 256, 256, 0, s>>>(a, axes, out);
}

// Clamped cell of every particle after the wrap (search grid for ghost partners).
__global__ void k_clamped_keys(StepArgs a, int* key2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.P.n) return;
  key2[i] = lin3(clamp_cell(cell_of(a.P.pos[i], a.pg), a.pg.size), a.pg.size);
}
void launch_clamped_keys(const StepArgs& a, int* key2, cudaStream_t s) {
  if (a.P.n > 0) k_clamped_keys<<<(a.P.n + 255) / 256, 256, 0, s>>>(a, key2);
}

// Visible images (ghost key >= 0) are compacted into a list first: only a
// few percent of (set, particle) pairs are images, so a thread per pair would
// leave almost every lane idle.
__global__ void k_ghost_compact(StepArgs a) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool vis = t < (long long)a.G.nsets * a.P.n && a.G.gkey[t] >= 0;
  const unsigned m = __ballot_sync(FULL, vis);
  if (m == 0) return;
  int base = 0;
  const int lane = threadIdx.x & 31;
  if (lane == __ffs(m) - 1) base = atomicAdd(a.G.count, __popc(m));
  base = __shfl_sync(FULL, base, __ffs(m) - 1);
  if (vis) a.G.list[base + __popc(m & lanemask_lt())] = (int)t;
}

// Ghost partners, searched with one warp per visible image G: a node of A can
// only reach G's cell window when A's clamped cell is within 2 cells of G's
// cell, and only when A's bounding sphere reaches G's SDF grid box. The lanes
// walk the occupants of those cells.
__global__ void k_ghost_candidates(StepArgs a, const int* __restrict__ g2_idx, const int* __restrict__ g2_off) {
  const int lane = threadIdx.x & 31;
  const int nvis = *a.G.count;
  const int n = a.P.n;
  const GridP& g = a.pg;
  int need = 0;  // largest per-particle image count seen by this lane
  for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nvis; v += (gridDim.x * blockDim.x) >> 5) {
    const int t = a.G.list[v];
    const int s = t / n, i = t % n;
    const int gk = a.G.gkey[t];
    const double3 xg = a.G.gpos[t];
    const int cx = gk % g.size.x, cy = (gk / g.size.x) % g.size.y, cz = gk / (g.size.x * g.size.y);
    // circumradius of the image's SDF grid box about its centre
    const double Rg = grid_reach(a, i);
    const int pid = (i << 3) | s;
    // A candidate lies within rmax + Rg of the image, so its clamped cell lies in
    // the per-axis cell range of that ball (edge cells are open outward: they
    // also hold clamped bodies outside the domain), intersected with the 2-cell
    // window.
    const double reach = (a.rmax + Rg) * (1.0 + 1e-6) + coord_slack(xg, xg);
    const int x0 = axis_lo(xg.x, g.mn.x, g.inv.x, g.size.x, reach, cx), x1 = axis_hi(xg.x, g.mn.x, g.inv.x, g.size.x, reach, cx);
    const int y0 = axis_lo(xg.y, g.mn.y, g.inv.y, g.size.y, reach, cy), y1 = axis_hi(xg.y, g.mn.y, g.inv.y, g.size.y, reach, cy);
    const int z0 = axis_lo(xg.z, g.mn.z, g.inv.z, g.size.z, reach, cz), z1 = axis_hi(xg.z, g.mn.z, g.inv.z, g.size.z, reach, cz);
    const float3 xgf = make_float3((float)xg.x, (float)xg.y, (float)xg.z);
    const float Rgf = (float)Rg, n1g = fabsf(xgf.x) + fabsf(xgf.y) + fabsf(xgf.z);
    // separation test of the pair (owner A, image), as for
    // particle pairs: a translated image has the particle's orientation, shape and scale
    // (turned sector images are not tested)
    const bool sep = !a.G.sector;
    const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
    const Quat qi = a.P.quat[i];
    const float4 qbf = make_float4((float)qi.q0, (float)qi.q1, (float)qi.q2, (float)qi.q3);
    const float4 pbf = make_float4(xgf.x, xgf.y, xgf.z, 0.f);
    const int shB = a.P.shape[i];
    const float scB = (float)a.P.scale[i];
    for (int z = z0; z <= z1; ++z) {
      for (int y = y0; y <= y1; ++y) {
        // the cells x0..x1 of a row are contiguous in the sorted order
        const int h0 = lin3(make_int3(x0, y, z), g.size);
        const int st = g2_off[h0 + 1], en = g2_off[h0 + (x1 - x0) + 2];
        {
          for (int k0 = st; k0 < en; k0 += 32) {
            const int k = k0 + lane;
            int slot = -1, A = 0;
            if (k < en) {
              // superset test on the FP32 copies (margin covers their rounding)
              const float4 pa = __ldg(a.cell_pk + k);
              const float dx = pa.x - xgf.x, dy = pa.y - xgf.y, dz = pa.z - xgf.z;
              const float R = (pa.w + Rgf) * (1.0f + 1e-5f) + 1e-6f * (n1g + fabsf(pa.x) + fabsf(pa.y) + fabsf(pa.z));
              bool cand = !(dx * dx + dy * dy + dz * dz > R * R);
              if (cand) A = __ldg(g2_idx + k);
              if (cand && sep) {
                const Quat qa = a.P.quat[A];
                const float4 qaf = make_float4((float)qa.q0, (float)qa.q1, (float)qa.q2, (float)qa.q3);
                const float n1a = __fadd_rn(__fadd_rn(fabsf(pa.x), fabsf(pa.y)), fabsf(pa.z));
                cand = !pair_separated(sup, pa, n1a, qaf, (float)a.P.scale[A], a.P.shape[A], pbf, qbf, scB, shB);
              }
              if (cand) {
                slot = atomicAdd(&a.pgh.cnt[A], 1);
                if (slot < a.pgh.cap) a.pgh.id[(size_t)A * a.pgh.cap + slot] = pid;
                else atomicOr(&a.status->flags, OVF_GHOST);
              }
            }
            need = max(need, slot + 1);
            {  // flat pair list
              const bool ok = slot >= 0 && slot < a.pgh.cap;
              const unsigned m = __ballot_sync(FULL, ok);
              int base = 0;
              if (lane == 0 && m) base = atomicAdd(&a.pl.ctr[2], __popc(m));
              base = __shfl_sync(FULL, base, 0);
              if (ok) a.pl.list[2][base + __popc(m & lanemask_lt())] = pair_code(A, a.pgh.cap, slot);
            }
          }
        }
      }
    }
  }
  need = __reduce_max_sync(FULL, need);
  if (lane == 0 && need > 0) atomicMax(&a.status->need_ghost, need);
}

// Image partners from the image list (k_rebuild, neighbours.cu): one thread per listed pair of
// an owner A and an image, which stands at the particle moved by the domain or at the particle
// itself (entry's high bit: moved). The pair is a candidate of this step when the image is
// visible and stands so now, A's clamped cell is among the cells that k_ghost_candidates
// walks for it, the spheres reach and no direction separates the two. Positions are the wrapped
// ones. Writes the position and the cell of the images it passes on. (The image search of a step
// was a wrap of all particles, a second cell sort and a walk, 18 launches beside the particles'
// own: a step of 100k polydisperse particles took 199 us with them and takes 146 us now, one of
// 2M settling particles 1105 and 665 us.)
__global__ void __launch_bounds__(128) k_image_candidates(StepArgs a) {
  const int lane = threadIdx.x & 31;
  const int m = min(*a.gl.count, a.gl.cap), n = a.P.n;
  const GridP& g = a.pg;
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  int need = 0;
  for (int e0 = (blockIdx.x * blockDim.x + threadIdx.x) - lane; e0 < m; e0 += gridDim.x * blockDim.x) {
    int slot = -1, A = 0;
    if (e0 + lane < m) {
      const int2 e = a.gl.list[e0 + lane];
      A = e.x & 0x7fffffff;
      const int i = e.y >> 3, s = e.y & 7;
      const double3 base = image_base(a.P.pos[i], g, a.wrap_axes, a.G.mask[s]);
      const bool hit = image_hit(base, g, a.G.mask[s]);
      const double3 xg = hit ? base + image_offset(g, a.G.mask[s]) : base;
      const int key = ghost_key(xg, g);
      bool cand = key >= 0 && hit == (e.x < 0);
      if (cand) {
        const double3 xA = wrap_pos(a.P.pos[A], g, a.wrap_axes);
        const int3 c = make_int3(key % g.size.x, (key / g.size.x) % g.size.y, key / (g.size.x * g.size.y));
        const int3 cA = clamp_cell(cell_of(xA, g), g.size);
        const double Rg = grid_reach(a, i);
        const double reach = (a.rmax + Rg) * (1.0 + 1e-6) + coord_slack(xg, xg);
        cand = cA.x >= axis_lo(xg.x, g.mn.x, g.inv.x, g.size.x, reach, c.x) &&
               cA.x <= axis_hi(xg.x, g.mn.x, g.inv.x, g.size.x, reach, c.x) &&
               cA.y >= axis_lo(xg.y, g.mn.y, g.inv.y, g.size.y, reach, c.y) &&
               cA.y <= axis_hi(xg.y, g.mn.y, g.inv.y, g.size.y, reach, c.y) &&
               cA.z >= axis_lo(xg.z, g.mn.z, g.inv.z, g.size.z, reach, c.z) &&
               cA.z <= axis_hi(xg.z, g.mn.z, g.inv.z, g.size.z, reach, c.z);
        if (cand) {
          int kA, kB;
          CandRec ra = cand_rec(a, A, kA), rb = cand_rec(a, i, kB);
          ra.p = make_float4((float)xA.x, (float)xA.y, (float)xA.z, ra.p.w);
          rb.p = make_float4((float)xg.x, (float)xg.y, (float)xg.z, 0.f);
          const float R = (ra.p.w + (float)Rg) * (1.0f + 1e-5f) + 1e-6f * (n1_f(rb.p) + n1_f(ra.p));
          cand = !(dist2_f(ra.p, rb.p) > R * R) &&
                 !pair_separated(sup, ra.p, n1_f(ra.p), ra.q, ra.sc, ra.sh, rb.p, rb.q, rb.sc, rb.sh);
        }
        if (cand) {
          a.G.gpos[(size_t)s * n + i] = xg;  // the same from every entry of the image
          a.G.gkey[(size_t)s * n + i] = key;
          slot = atomicAdd(&a.pgh.cnt[A], 1);
          if (slot < a.pgh.cap) a.pgh.id[(size_t)A * a.pgh.cap + slot] = e.y;
          else atomicOr(&a.status->flags, OVF_GHOST);
        }
      }
    }
    need = max(need, slot + 1);
    {  // flat pair list
      const bool ok = slot >= 0 && slot < a.pgh.cap;
      const unsigned mk = __ballot_sync(FULL, ok);
      int at = 0;
      if (lane == 0 && mk) at = atomicAdd(&a.pl.ctr[2], __popc(mk));
      at = __shfl_sync(FULL, at, 0);
      if (ok) a.pl.list[2][at + __popc(mk & lanemask_lt())] = pair_code(A, a.pgh.cap, slot);
    }
  }
  need = __reduce_max_sync(FULL, need);
  if (lane == 0 && need > 0) atomicMax(&a.status->need_ghost, need);
}

void launch_image_candidates(const StepArgs& a, cudaStream_t s) {
  if (a.P.n > 0) k_image_candidates<<<std::min((a.P.n + 127) / 128, num_sms() * 4), 128, 0, s>>>(a);
}

// The step's wrap, in place after everything that reads the positions before it. A body beyond a
// periodic face has set the rebuild flag (k_integrate_first), so most steps return at once.
__global__ void k_wrap(StepArgs a) {
  if (*a.reuse == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.P.n) return;
  const double3 x = a.P.pos[i], p = wrap_pos(x, a.pg, a.wrap_axes);
  if (p.x != x.x || p.y != x.y || p.z != x.z) a.P.pos[i] = p;
}
void launch_wrap(const StepArgs& a, cudaStream_t s) {
  if (a.P.n > 0) k_wrap<<<(a.P.n + 255) / 256, 256, 0, s>>>(a);
}

void launch_ghost_candidates(const StepArgs& a, const int* g2_idx, const int* g2_off, cudaStream_t s) {
  long long n = (long long)a.G.nsets * a.P.n;
  if (n <= 0) return;
  k_ghost_compact<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
  StepArgs g = a;
  g.pk_meta = nullptr;  // the particle records stay in the particle grid's order
  k_pack_cells<<<(a.P.n + 255) / 256, 256, 0, s>>>(g, g2_idx);  // the candidate walk's copy is spent
  int blocks = num_sms() * 16;
  k_ghost_candidates<<<blocks, 128, 0, s>>>(a, g2_idx, g2_off);
}

// ---------------------------------------------------------------------------
// V-bond forces, one thread per bond.
__global__ void k_bonds(StepArgs a, BondView b) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= b.n) return;
  double* st = b.state + 9 * (size_t)k;
  if (b.bonded[k] == 0) {
    for (int q = 0; q < 6; ++q) st[q] = 0.;
    return;
  }
  const int i = b.ids[2 * k], j = b.ids[2 * k + 1];
  const Quat qi = a.P.quat[i], qj = a.P.quat[j];
  const double3* fr = b.frames + 8 * (size_t)k;
  const double3 n1i = rotate(qi, fr[0]), n2i = rotate(qi, fr[1]), n3i = rotate(qi, fr[2]);
  const double3 n1j = rotate(qj, fr[4]), n2j = rotate(qj, fr[5]), n3j = rotate(qj, fr[6]);
  const double3 ri = a.P.pos[i], rj = a.P.pos[j];
  const double3 rbi = rotate(qi, fr[3]) + ri;
  const double3 rbj = rotate(qj, fr[7]) + rj;
  const double3 bp = 0.5 * (rbi + rbj);
  st[6] = bp.x; st[7] = bp.y; st[8] = bp.z;
  const double B1 = b.B[4 * k], B2 = b.B[4 * k + 1], B3 = b.B[4 * k + 2], B4 = b.B[4 * k + 3];
  const double Rb = b.geo[5 * k], D0 = b.geo[5 * k + 1], ten = b.geo[5 * k + 2], coh = b.geo[5 * k + 3],
               fmu = b.geo[5 * k + 4];
  double3 F = d3(0., 0., 0.), Mij = d3(0., 0., 0.), Mji = d3(0., 0., 0.);
  int ok = 1;
  const double3 rbij = rbi - rbj;
  const double D = len(rbij);
  if (!is_zero(D)) {
    const double3 nij = normalize_dev(rbij);
    const double3 e = -nij;
    st[0] = 0.5 * B1 * (D - D0) * (D - D0);
    st[1] = B2 * (0.5 * dot((n1j - n1i), e) - 0.25 * dot(n1i, n1j) + 0.75);
    st[2] = (0.25 * B2 + B3 + 0.5 * B4) * (dot(n1i, n1j) + 1.);
    st[3] = -0.5 * B4 * (dot(n1i, n1j) + dot(n2i, n2j) + dot(n3i, n3j) - 1);
    F = B1 * (D - D0) * e + B2 / (2 * D) * ((n1j - n1i) - dot((n1j - n1i), e) * e);
    const double3 MTB = B3 * cross(n1j, n1i) - 0.5 * B4 * (cross(n2j, n2i) + cross(n3j, n3i));
    Mij = -0.5 * B2 * cross(e, n1i) + MTB;
    Mji = 0.5 * B2 * cross(e, n1j) - MTB;
    const double fnb = dot(F, nij);
    const double3 fsb = F - fnb * nij;
    const double tt = dot(MTB, nij);
    const double3 tb = MTB - tt * nij;
    const double Ab = Rb * Rb * M_PI;
    const double Ib = Ab * Rb * Rb / 4.;
    const double Jb = 2 * Ib;
    st[4] = -fnb / Ab + len(tb) / Ib * Rb;
    st[5] = len(fsb) / Ab + fabs(tt) / Jb * Rb;
    if (ten > 0. && st[4] > ten) ok = 0;
    else if (coh > 0. && st[5] > coh - fmu * st[4]) ok = 0;
  }
  b.bonded[k] = ok;
  atomic_add3(a.P.force, i, F);
  atomic_add3(a.P.torque, i, Mij + cross(rbi - ri, F));
  atomic_add3(a.P.force, j, -F);
  atomic_add3(a.P.torque, j, Mji + cross(rbj - rj, -F));
}

void launch_bonds(const StepArgs& a, const BondView& b, cudaStream_t s) {
  if (b.n > 0) k_bonds<<<(b.n + 127) / 128, 128, 0, s>>>(a, b);
}

}  // namespace lsdem
