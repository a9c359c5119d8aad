// The separating-axis test of candidate pairs and the bounding-sphere test before it, shared by
// the candidate search of a step (step.cu) and the neighbour lists' rebuild (neighbours.cu).
#pragma once
#include "kernels.h"

namespace lsdem {

// The separation test runs in FP32 on the packed records of the candidate search, with
// explicitly rounded operations, so that every place it is inlined at decides a pair alike.
LD float3 rot_f(float3 v, float w, float a, float b, float c) {
  const float tx = __fmul_rn(2.0f, __fmaf_rn(b, v.z, -__fmul_rn(c, v.y)));
  const float ty = __fmul_rn(2.0f, __fmaf_rn(c, v.x, -__fmul_rn(a, v.z)));
  const float tz = __fmul_rn(2.0f, __fmaf_rn(a, v.y, -__fmul_rn(b, v.x)));
  return make_float3(__fadd_rn(__fmaf_rn(w, tx, v.x), __fmaf_rn(b, tz, -__fmul_rn(c, ty))),
                     __fadd_rn(__fmaf_rn(w, ty, v.y), __fmaf_rn(c, tx, -__fmul_rn(a, tz))),
                     __fadd_rn(__fmaf_rn(w, tz, v.z), __fmaf_rn(a, ty, -__fmul_rn(b, tx))));
}
LD float dot_f(float3 a, float3 b) { return __fmaf_rn(a.x, b.x, __fmaf_rn(a.y, b.y, __fmul_rn(a.z, b.z))); }

// Upper bound of the support h(u) from the table of one shape, and the bound's gradient g:
// on the cone of a cell's triangle the bound is linear in u, so g is the point it is reached
// at (a point near the shape's support point along u). 0 when u = 0.
LD float sup_bound_f(const float4* __restrict__ tab, float3 u, float3& g) {
  const float ax = fabsf(u.x), ay = fabsf(u.y), az = fabsf(u.z);
  int f;
  float p, q, m;
  if (ax >= ay && ax >= az) { f = u.x >= 0.f ? 0 : 1; m = ax; p = u.y; q = u.z; }
  else if (ay >= az) { f = u.y >= 0.f ? 2 : 3; m = ay; p = u.z; q = u.x; }
  else { f = u.z >= 0.f ? 4 : 5; m = az; p = u.x; q = u.y; }
  g = make_float3(0.f, 0.f, 0.f);
  if (!(m > 0.f)) return 0.f;
  const float r = __frcp_rn(m);
  p = __fmul_rn(p, r);
  q = __fmul_rn(q, r);
  const float x = __fmul_rn(__fadd_rn(p, 1.0f), 0.5f * SUP_M);
  const float y = __fmul_rn(__fadd_rn(q, 1.0f), 0.5f * SUP_M);
  const int i = min(max((int)floorf(x), 0), SUP_M - 1), j = min(max((int)floorf(y), 0), SUP_M - 1);
  const float s = fminf(fmaxf(__fsub_rn(x, (float)i), 0.f), 1.f), t = fminf(fmaxf(__fsub_rn(y, (float)j), 0.f), 1.f);
  const float4 c = __ldg(tab + (f * SUP_M + j) * SUP_M + i);
  const bool low = __fadd_rn(s, t) <= 1.0f;
  const float ds = low ? __fsub_rn(c.y, c.x) : __fsub_rn(c.w, c.z), dt = low ? __fsub_rn(c.z, c.x) : __fsub_rn(c.w, c.y);
  const float v = low ? __fmaf_rn(s, ds, __fmaf_rn(t, dt, c.x))
                      : __fmaf_rn(__fsub_rn(s, 1.0f), ds, __fmaf_rn(__fsub_rn(t, 1.0f), dt, c.w));
  const float gp = __fmul_rn(ds, 0.5f * SUP_M), gq = __fmul_rn(dt, 0.5f * SUP_M);
  const float g0 = __fmaf_rn(-gp, p, __fmaf_rn(-gq, q, v)), gm = (f & 1) ? -g0 : g0;
  g = f < 2 ? make_float3(gm, gp, gq) : (f < 4 ? make_float3(gq, gm, gp) : make_float3(gp, gq, gm));
  return __fmul_rn(m, v);
}

struct SupTabs {
  const float4* n;  // nodes
  const float4* s;  // solid
  const float* r;   // largest |p| of the solid's points
};

// Separating-axis test of the pair (A, B). For a direction s, every node of A projects onto s
// at most scale_A h_n(A, R_A^T s) beyond x_A, and every point where B's interpolated phi is
// <= 0 at least scale_B h_s(B, -R_B^T s) before x_B; if the two reaches sum to less than
// s . (x_B - x_A) for any s, no node of A can be inside B and the pair has no contact.
// The first direction is the line of centres. While a direction does not separate, the two
// support points it gives, delta = (B's) - (A's), give the next: s + 1.75 (e / |delta|^2) delta,
// e what s . delta lacks of the margin, over-relaxed towards the half space that s must lie in
// (the separating vector step of K. Chung and W. Wang, "Quick collision detection of polytopes in
// virtual environments", 1996, with 1.75 in place of its reflection's 2). Of the pairs of a
// random packing of superquadrics that some direction separates, the line of centres finds
// four fifths, one more direction 97 %, SEP_DIRS directions 99.7 %. The bodies of a pair that
// is kept are within a few per cent of their size of touching, so this test sets the work of
// everything after it: settling configuration of 2M particles, candidate pairs per step
// 490k -> 225k; bonded lattice of 12,000, 43.8k -> 6.8k
// (25k and none with the tables of k_support_vertices).
// Margins: the FP32 centres differ from the FP64 ones by at most 2^-24 of each
// coordinate, so the distance by 1.2e-7 (n1 + D); 2e-6 for the FP32 orientation and
// rotation, and 2e-6 for the rounding of the face
// coordinates and of the interpolation (the interpolated plane point moves by a few
// 1e-7, and the values, at most sqrt(3) times the set's largest |p|, round by a few
// ulps); a direction error e moves a support by at most e times the set's largest |p|
// (the bounding radius for A's nodes, scale_B sup_r for B's solid). |s| = 1 and the rotation
// keeps it within 1e-6, and s . (x_B - x_A) rounds by less than 1e-6 D, covered by the relative
// 1e-5. Each margin is taken several times over, and they are the same for every direction: a
// direction is exact by itself, whichever way it was found.
// gap > 0: the bodies must be at least that far apart along the direction.
static constexpr int SEP_DIRS = 5;
template <int DIRS = SEP_DIRS>
LD bool pair_separated(const SupTabs& S, float4 pa, float n1a, float4 qA, float scA, int shA, float4 pb, float4 qb,
                       float scB, int shB, float gap = 0.f) {
  const float3 d = make_float3(__fsub_rn(pb.x, pa.x), __fsub_rn(pb.y, pa.y), __fsub_rn(pb.z, pa.z));
  const float D2 = dot_f(d, d);
  if (!(D2 > 0.f)) return false;
  const float D = __fsqrt_rn(D2), Di = __frcp_rn(D);
  const float n1 = __fadd_rn(n1a, __fadd_rn(__fadd_rn(fabsf(pb.x), fabsf(pb.y)), fabsf(pb.z)));
  const float eps = __fadd_rn(__fmul_rn(__fmul_rn(4e-7f, __fadd_rn(n1, D)), Di), 8e-6f);
  const float rho = __fadd_rn(pa.w, __fmul_rn(scB, __ldg(S.r + shB)));
  const float slack = __fadd_rn(gap, __fmaf_rn(eps, rho, __fmaf_rn(1e-6f, n1, __fmul_rn(1e-5f, D))));
  const float4* tA = S.n + (size_t)shA * SUP_CELLS;
  const float4* tB = S.s + (size_t)shB * SUP_CELLS;
  float3 s = make_float3(__fmul_rn(d.x, Di), __fmul_rn(d.y, Di), __fmul_rn(d.z, Di));
#pragma unroll 1
  for (int k = 0;; ++k) {
    float3 gA, gB;
    const float hA = __fmul_rn(scA, sup_bound_f(tA, rot_f(s, qA.x, -qA.y, -qA.z, -qA.w), gA));
    const float hB = __fmul_rn(scB, sup_bound_f(tB, rot_f(make_float3(-s.x, -s.y, -s.z), qb.x, -qb.y, -qb.z, -qb.w), gB));
    const float sd = dot_f(s, d), need = __fmul_rn(__fadd_rn(__fadd_rn(hA, hB), slack), 1.0f + 1e-5f);
    if (need < sd) return true;
    if (k == DIRS - 1) return false;
    const float3 wA = rot_f(gA, qA.x, qA.y, qA.z, qA.w), wB = rot_f(gB, qb.x, qb.y, qb.z, qb.w);
    const float3 dl = make_float3(__fmaf_rn(scB, wB.x, __fmaf_rn(-scA, wA.x, d.x)),
                                  __fmaf_rn(scB, wB.y, __fmaf_rn(-scA, wA.y, d.y)),
                                  __fmaf_rn(scB, wB.z, __fmaf_rn(-scA, wA.z, d.z)));
    const float dd = dot_f(dl, dl);
    if (!(dd > __fmul_rn(1e-10f, D2))) return false;
    const float c = __fdiv_rn(__fmul_rn(1.75f, __fsub_rn(need, sd)), dd);
    s = make_float3(__fmaf_rn(c, dl.x, s.x), __fmaf_rn(c, dl.y, s.y), __fmaf_rn(c, dl.z, s.z));
    const float i = __frsqrt_rn(dot_f(s, s));
    s = make_float3(__fmul_rn(s.x, i), __fmul_rn(s.y, i), __fmul_rn(s.z, i));
  }
}

// Bounding-sphere test of the candidate search on the FP32 copies (centre and
// bounding radius): the reach carries a margin that covers their rounding
// (relative 1e-5 plus 1e-6 of the coordinates). Written with explicitly rounded
// operations so that every caller evaluates it to the same bits.
LD float reach_f(float4 pa, float n1a, float4 pb) {
  const float n1 = __fadd_rn(n1a, __fadd_rn(__fadd_rn(fabsf(pb.x), fabsf(pb.y)), fabsf(pb.z)));
  return __fmaf_rn(1e-6f, n1, __fmul_rn(__fadd_rn(pa.w, pb.w), 1.0f + 1e-5f));
}
LD float dist2_f(float4 pa, float4 pb) {
  const float dx = __fsub_rn(pb.x, pa.x), dy = __fsub_rn(pb.y, pa.y), dz = __fsub_rn(pb.z, pa.z);
  return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmul_rn(dz, dz)));
}

// Cell index along one axis of the point v, by floor and clamped to [0, n - 1]:
// monotone in v and equal to the key's int() cell for points inside the grid.
LD int ball_axis(double v, double mn, double inv, int n) {
  const double f = floor((v - mn) * inv);
  return f <= 0.0 ? 0 : (f >= (double)(n - 1) ? n - 1 : (int)f);
}
LD int3 ball_cell(double3 p, const GridP& g) {
  return make_int3(ball_axis(p.x, g.mn.x, g.inv.x, g.size.x), ball_axis(p.y, g.mn.y, g.inv.y, g.size.y),
                   ball_axis(p.z, g.mn.z, g.inv.z, g.size.z));
}


// The lane that owns entry i of the warp's entries, given every lane's inclusive count of them
// (all lanes call it; 31 for an i past the last).
LD int lane_of(int incl, int i) {
  int ow = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int v = __shfl_sync(0xffffffffu, incl, ow + o - 1);
    if (v <= i) ow += o;
  }
  return ow;
}

// FP32 record of one particle for the two tests.
struct CandRec {
  float4 p;  // centre, bounding radius
  float4 q;
  float sc;
  int sh;
};
LD CandRec cand_rec(const StepArgs& a, int i, int& key) {
  const float4 x = a.rec[2 * i], q = a.rec[2 * i + 1], s = __ldg(a.rec_s + i);
  key = __float_as_int(x.w);
  return CandRec{make_float4(x.x, x.y, x.z, s.x), q, s.y, __float_as_int(s.z)};
}
// Record of body B at sorted position k (the sorted order of the walks).
LD void pack_cell(const StepArgs& a, int k, int B) {
  const double3 x = a.P.pos[B];
  a.cell_pk[k] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)a.P.radius[B]);
  if (a.pk_meta) {
    a.pk_meta[k] = make_int4(a.P.key[B], B, a.P.shape[B], __float_as_int((float)a.P.scale[B]));
    const Quat q = a.P.quat[B];
    a.pk_q[k] = make_float4((float)q.q0, (float)q.q1, (float)q.q2, (float)q.q3);
  }
}
LD float n1_f(float4 p) { return __fadd_rn(__fadd_rn(fabsf(p.x), fabsf(p.y)), fabsf(p.z)); }

}  // namespace lsdem
