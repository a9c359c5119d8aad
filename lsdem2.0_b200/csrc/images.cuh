// Periodic wrap and images of one particle (mySpatialGrid.cu:28-56, 87-152, 214-240), shared by
// the image search of a step (step.cu) and the neighbour lists' rebuild (neighbours.cu).
#pragma once
#include "kernels.h"

namespace lsdem {

LD double3 wrap_axis(double3 p, const GridP& g, int ax) {
  if (ax == 0) { const double L = g.mx.x - g.mn.x; if (p.x < g.mn.x) p.x += L; else if (p.x >= g.mx.x) p.x -= L; }
  if (ax == 1) { const double L = g.mx.y - g.mn.y; if (p.y < g.mn.y) p.y += L; else if (p.y >= g.mx.y) p.y -= L; }
  if (ax == 2) { const double L = g.mx.z - g.mn.z; if (p.z < g.mn.z) p.z += L; else if (p.z >= g.mx.z) p.z -= L; }
  return p;
}
LD double3 wrap_pos(double3 p, const GridP& g, int axes) {
  for (int ax = 0; ax < 3; ++ax)
    if ((axes >> ax) & 1) p = wrap_axis(p, g, ax);
  return p;
}

// Position that the image of set `mask` is taken from: a single-axis set right after its own
// axis is wrapped, the others after all wraps.
LD double3 image_base(double3 p, const GridP& g, int axes, int mask) {
  const int upto = mask == 1 ? 1 : (mask == 2 ? 3 : 7);
  return wrap_pos(p, g, axes & upto);
}
LD double3 image_offset(const GridP& g, int mask) {
  return d3(mask & 1 ? g.mx.x - g.mn.x : 0., mask & 2 ? g.mx.y - g.mn.y : 0., mask & 4 ? g.mx.z - g.mn.z : 0.);
}
// True when p is in the first cell along every axis of the set: then the image is p moved by
// the domain, otherwise it stays at p.
LD bool image_hit(double3 p, const GridP& g, int mask) {
  const int3 c = cell_of(p, g);
  return (!(mask & 1) || c.x == 0) && (!(mask & 2) || c.y == 0) && (!(mask & 4) || c.z == 0);
}
LD void ghost_image(double3 p, const GridP& g, int mask, double3& out) {
  out = p;
  if (image_hit(p, g, mask)) out += image_offset(g, mask);
}
LD int ghost_key(double3 p, const GridP& g) {
  int3 c = cell_of(p, g);
  bool out = false;
  if (p.x < g.mn.x) { c.x = 0; out = true; } else if (p.x >= g.mx.x) { c.x = g.size.x - 1; out = true; }
  if (p.y < g.mn.y) { c.y = 0; out = true; } else if (p.y >= g.mx.y) { c.y = g.size.y - 1; out = true; }
  if (p.z < g.mn.z) { c.z = 0; out = true; } else if (p.z >= g.mx.y) { c.z = g.size.z - 1; out = true; }
  return out ? lin3(c, g.size) : -1;
}

// Circumradius of a particle's SDF grid box about its centre.
LD double grid_reach(const StepArgs& a, int i) {
  const double3 o = a.P.origin[i];
  const int3 gs = a.S.gsize[a.P.shape[i]];
  const double invh = a.P.invh[i];
  const double3 hi = d3(o.x + (gs.x - 1) / invh, o.y + (gs.y - 1) / invh, o.z + (gs.z - 1) / invh);
  return len(d3(fmax(fabs(o.x), fabs(hi.x)), fmax(fabs(o.y), fabs(hi.y)), fmax(fabs(o.z), fabs(hi.z))));
}

// Cell range along one axis of a ball (centre p, radius r) on the clamped grid,
// intersected with [c - 2, c + 2].
LD int axis_lo(double p, double mn, double inv, int size, double r, int c) {
  int v = (int)floor((p - mn - r) * inv);
  v = v < 0 ? 0 : (v > size - 1 ? size - 1 : v);
  return v > c - 2 ? v : c - 2;
}
LD int axis_hi(double p, double mn, double inv, int size, double r, int c) {
  int v = (int)floor((p - mn + r) * inv);
  v = v < 0 ? 0 : (v > size - 1 ? size - 1 : v);
  return v < c + 2 ? v : c + 2;
}

}  // namespace lsdem
