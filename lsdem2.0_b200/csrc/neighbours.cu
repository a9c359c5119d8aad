// Rebuild of the neighbour lists: cell sort, packed records and lists in one cooperative launch.
//
// A step launches it after its drift; between rebuilds every block returns at once. As separate
// launches the sort alone was ten that returned at once, 1.9 us each of the 58 us that a step of
// 2,000 particles took; a rebuild's phases, one grid barrier apart, take no longer than those
// launches did.
//
// A list holds, per particle A, the bodies B > A that some step may find before the next
// rebuild: bounding spheres within reach + skin, and no direction found along which the two are
// 0.8 skin apart. Until the next rebuild no point of a body moves by more than 0.4 skin
// (k_integrate_first, the turn of the body included), so bodies that were 0.8 skin apart have no
// contact. Listing only what is that near, a twelfth of the bodies within reach + skin in the
// settling configuration, is what makes the steps between rebuilds cheap.
#include <cooperative_groups.h>

#include <algorithm>

#include "cell_sort.cuh"
#include "images.cuh"
#include "separation.cuh"

namespace lsdem {

namespace cg = cooperative_groups;

static constexpr unsigned FULL = 0xffffffffu;
static constexpr int RB_THREADS = 256;
static constexpr int RB_BUF = 12;  // bodies within reach + skin a lane gathers before the warp tests them

// The stable cell sort of bucket_sort (sort_scan.cu), phase by phase; the members of a cell in any
// order where ORDERED is false (the images' search, whose list has none).
template <bool ORDERED>
LD void grid_cell_sort(cg::grid_group& grid, const int* key, int n, int ncells, const BucketScratch& w, int* sorted_idx,
                       int* sums, int* sw) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
  const int nb = ncells + 2, m = nb + 1;
  for (int i = tid; i < m; i += T) w.counts[i] = w.fill[i] = 0;
  if (tid == 0) w.big_count[0] = w.big_count[1] = 0;
  grid.sync();
  for (int i = tid; i < n; i += T) atomicAdd(&w.counts[bucket_of(key[i], ncells)], 1);
  grid.sync();
  // exclusive scan over nb + 1 entries: each block a chunk
  const int chunk = (m + gridDim.x - 1) / gridDim.x, c0 = min(m, (int)blockIdx.x * chunk), c1 = min(m, c0 + chunk);
  int sum = 0, tot;
  for (int i = c0 + threadIdx.x; i < c1; i += blockDim.x) sum += __ldcg(w.counts + i);
  block_exclusive_scan<int>(sum, sw, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
  grid.sync();
  sum = 0;
  for (int i = threadIdx.x; i < (int)blockIdx.x; i += blockDim.x) sum += __ldcg(sums + i);
  int base;
  block_exclusive_scan<int>(sum, sw, &base);
  for (int i0 = c0; i0 < c1; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    const int v = i < c1 ? __ldcg(w.counts + i) : 0;
    const int ex = block_exclusive_scan<int>(v, sw, &tot);
    if (i < c1) w.offs[i] = base + ex;
    base += tot;
  }
  grid.sync();
  // scatter; a special bucket longer than a warp can rank is placed in index order instead
  const int n0 = __ldcg(w.offs + 1), nL = n - __ldcg(w.offs + ncells + 1);
  for (int i = tid; i < n; i += T) {
    const int b = bucket_of(key[i], ncells);
    if ((b == 0 && n0 > 64) || (b == ncells + 1 && nL > 64)) continue;
    sorted_idx[__ldcg(w.offs + b) + atomicAdd(&w.fill[b], 1)] = i;
  }
  if (n0 > 64 || nL > 64) {
    // in index order: a chunk of bodies per block, behind the chunks before it (1M bodies, 900k of
    // them outside, rebuilt in every step: 4450 us a step with one block for all of them, 1560 this way)
    const int part = (n + gridDim.x - 1) / gridDim.x, i0 = min(n, (int)blockIdx.x * part), i1 = min(n, i0 + part);
    int f0 = 0, fL = 0;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
      const int b = bucket_of(key[i], ncells);
      f0 += b == 0;
      fL += b == ncells + 1;
    }
    block_exclusive_scan<int>(f0, sw, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
    block_exclusive_scan<int>(fL, sw, &tot);
    if (threadIdx.x == 0) sums[REBUILD_SUMS / 2 + blockIdx.x] = tot;
    grid.sync();
    f0 = fL = 0;
    for (int i = threadIdx.x; i < (int)blockIdx.x; i += blockDim.x) {
      f0 += __ldcg(sums + i);
      fL += __ldcg(sums + REBUILD_SUMS / 2 + i);
    }
    int base0, baseL;
    block_exclusive_scan<int>(f0, sw, &base0);
    block_exclusive_scan<int>(fL, sw, &baseL);
    special_buckets(key, i0, i1, ncells, w.offs, base0, n - nL + baseL, sorted_idx, sw);
  }
  grid.sync();
  if (!ORDERED) return;
  for (int b = tid; b < nb; b += T) {
    const int s = w.offs[b], L = w.offs[b + 1] - s;
    if (L <= 1 || (b == 0 && L > 64)) continue;
    if (L > 64) w.big_list[atomicAdd(&w.big_count[0], 1)] = b;
    else if (L > 8) w.tmp[atomicAdd(&w.big_count[1], 1)] = b;
    else small_bucket(key, b == ncells + 1, s, L, sorted_idx);
  }
  grid.sync();
  const int nbig = __ldcg(w.big_count), nmid = __ldcg(w.big_count + 1);
  for (int q = tid >> 5; q < nmid; q += T >> 5) {
    const int b = __ldcg(w.tmp + q), s = w.offs[b];
    mid_bucket(key, b == ncells + 1, s, w.offs[b + 1] - s, sorted_idx);
  }
  if (nbig > 0) {
    grid.sync();  // tmp held the list of the buckets above
    for (int q = blockIdx.x; q < nbig; q += gridDim.x) {
      const int b = __ldcg(w.big_list + q), s = w.offs[b];
      big_bucket(key, b == ncells + 1, s, w.offs[b + 1] - s, sorted_idx, w.tmp);
      __syncthreads();
    }
  }
  if (nbig > 0 || nmid > 0) grid.sync();
}

// Bounding spheres within reach + skin, with a margin beyond the FP32 rounding of the step's test.
LD bool in_reach(const StepArgs& a, float4 pa, float n1a, float4 pb) {
  const float Rs = __fmul_rn(__fmaf_rn(1e-5f, __fadd_rn(n1a, n1_f(pb)), __fadd_rn(reach_f(pa, n1a, pb), a.skin)),
                             1.0f + 1e-4f);
  return !(dist2_f(pa, pb) > __fmul_rn(Rs, Rs));
}

// Bodies that crossed a periodic face in this step: they stand in no cell, and from the next step
// on at their wrapped position, in the domain or outside it along another axis. Their pairs there
// are added to the lists now, so that the next step, which finds them moved by the domain, needs no
// rebuild of its own. The partners of such a body are bodies in a cell, and the crossers that
// will be; it is itself a partner, of any body of smaller index, once it is in a cell, so that the
// bodies in no cell are looked through, too. list[0, m) holds them.
// (Only where the domain is wide enough that a body cannot be near both positions: a.cross.)
//
// A warp walks the cells of one crosser; the crossers and the bodies in no cell are tested against
// each crosser in chunks of 32, spread over the warps (100k bodies with 30k of them above the domain,
// one or two crossers a step: 660 us a step with all of it by the crosser's warp, 333 this way). The
// work is the product of two counts: above CROSS_PAIRS the next step rebuilds instead (bodies that
// are handed over a domain's length off all cross at once).
static constexpr long long CROSS_PAIRS = 1ll << 24;
LD void grid_cross_lists(const StepArgs& a, const BucketScratch& w, const int* idx, const int* list, int m) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
  const int n = a.P.n;
  const int n0 = __ldcg(w.offs + 1), nL = n - __ldcg(w.offs + a.pg.ncells + 1);  // in no cell
  if ((long long)m * (m + n0 + nL) > CROSS_PAIRS) {
    if (tid == 0) *a.reuse_next = 2;
    return;
  }
  const GridP& g = a.pg;
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  const float gap = 0.8f * a.skin * (1.0f + 1e-5f);
  // crosser v at its next position
  int W = 0;
  double3 xw = d3(0., 0., 0.);
  CandRec rw;
  float n1w = 0.f;
  auto take = [&](int v) {
    W = __ldcg(list + v);
    xw = wrap_pos(a.P.pos[W], g, a.wrap_axes);
    int key;
    rw = cand_rec(a, W, key);
    rw.p = make_float4((float)xw.x, (float)xw.y, (float)xw.z, rw.p.w);
    n1w = n1_f(rw.p);
  };
  auto add = [&](int B, float4 pB) {
    if (!__ldcg(a.kin + max(W, B)) || !in_reach(a, rw.p, n1w, pB)) return;
    int key;
    CandRec rb = cand_rec(a, B, key);
    rb.p = pB;
    const bool first = W < B;
    const CandRec &r0 = first ? rw : rb, &r1 = first ? rb : rw;
    if (pair_separated<2>(sup, r0.p, n1_f(r0.p), r0.q, r0.sc, r0.sh, r1.p, r1.q, r1.sc, r1.sh, gap)) return;
    const int A = first ? W : B, at = atomicAdd(&a.nbr_cnt[A], 1);
    if (at >= 0 && at < a.nbr_cap) a.nbr[(size_t)at * n + A] = first ? B : W;
    if (at >= a.nbr_cap) {
      atomicMax(&a.status->need_nbr, at + 1);
      atomicOr(&a.status->flags, OVF_NBR);
    }
  };
  for (int v = tid >> 5; v < m; v += T >> 5) {
    take(v);
    const double R = a.P.radius[W] + a.rmax + (double)a.skin;
    const double ext = 1.001 * R + 1e-4 * (fabs(xw.x) + fabs(xw.y) + fabs(xw.z) + 4.0 * R);
    const int3 lo = ball_cell(xw - d3(ext, ext, ext), g), hi = ball_cell(xw + d3(ext, ext, ext), g);
    for (int z = lo.z; z <= hi.z; ++z)
      for (int y = lo.y; y <= hi.y; ++y) {
        const int h0 = lin3(make_int3(lo.x, y, z), g.size);
        const int st = __ldcg(w.offs + h0 + 1), en = __ldcg(w.offs + h0 + (hi.x - lo.x) + 2);
        for (int k = st + lane; k < en; k += 32) add(a.pk_meta[k].y, a.cell_pk[k]);
      }
  }
  const int chunks = (m + n0 + nL + 31) / 32;
  for (int q = tid >> 5; q < m * chunks; q += T >> 5) {
    const int v = q / chunks, u = (q - v * chunks) * 32 + lane;
    take(v);
    if (u < m) {  // the other crossers, once
      const int B = __ldcg(list + u);
      const double3 x = wrap_pos(a.P.pos[B], g, a.wrap_axes);
      if (u > v) add(B, make_float4((float)x.x, (float)x.y, (float)x.z, __ldg(a.rec_s + B).x));
    } else if (u < m + n0 + nL) {  // the bodies in no cell that did not cross
      const int k = u - m < n0 ? u - m : n - nL + u - m - n0, B = __ldcg(idx + k);
      const double3 x = a.P.pos[B], p = wrap_pos(x, g, a.wrap_axes);
      if (p.x == x.x && p.y == x.y && p.z == x.z) add(B, a.cell_pk[k]);
    }
  }
}

// The image list: owners A and images that some step before the next rebuild may find as
// partners. An image is listed where it stands if its particle may be found in the first cell
// along the set's axes (moved by the domain), and, not moved, if it is visible in place (a body
// outside the domain, or above the y bound, which the image keys test z against); in between,
// bodies keep their side of the domain's faces, or the lists are rebuilt. The search is that of
// k_ghost_candidates with the list's margin.
LD void grid_image_list(cg::grid_group& grid, const StepArgs& a, const BucketScratch& w1, const int* idx1,
                        const ImageSort& im, int* sums, int* sw) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
  const int n = a.P.n;
  const GridP& g = a.pg;
  if (tid == 0) *a.G.count = *a.gl.count = 0;
  // The owners are searched in the cells of their wrapped positions. Those of bodies in a cell are
  // the particle sort's own; the bodies in no cell are tested one by one with every image while
  // they are few (the crossers of a step), and all bodies sorted again otherwise (a second sort
  // was a third of a rebuild of 100k particles).
  const int n0 = __ldcg(w1.offs + 1), nL = n - __ldcg(w1.offs + g.ncells + 1);
  const bool resort = n0 + nL > 64;
  grid.sync();
  if (resort) {
    for (int i = tid; i < n; i += T)
      im.key[i] = lin3(clamp_cell(cell_of(wrap_pos(a.P.pos[i], g, a.wrap_axes), g), g.size), g.size);
    grid.sync();
    grid_cell_sort<false>(grid, im.key, n, g.ncells, im.w, im.idx, sums, sw);
    for (int k = tid; k < n; k += T) {
      const int B = __ldcg(im.idx + k);
      const double3 p = wrap_pos(a.P.pos[B], g, a.wrap_axes);
      im.pk[k] = make_float4((float)p.x, (float)p.y, (float)p.z, (float)a.P.radius[B]);
    }
  }
  const int* offs = resort ? im.w.offs : w1.offs;
  const int* idx = resort ? im.idx : idx1;
  const float4* pk = resort ? im.pk : a.cell_pk;
  const double m = 0.4 * (double)a.skin * 1.01;
  for (int i0 = tid - lane; i0 < n; i0 += T) {
    const int i = i0 + lane;
    double3 x = d3(0., 0., 0.);
    if (i < n) x = a.P.pos[i];
    for (int s = 0; s < a.G.nsets; ++s) {
      bool on[2] = {false, false};  // in place, moved
      // (with a.cross also where a body beyond a face stands from the next step on)
      for (int q = 0; i < n && q < (a.cross ? 2 : 1); ++q) {
        const int mask = a.G.mask[s];
        const double3 p = q == 0 ? image_base(x, g, a.wrap_axes, mask) : wrap_pos(x, g, a.wrap_axes);
        const double ux = fabs((p.x - g.mn.x) * g.inv.x), uy = fabs((p.y - g.mn.y) * g.inv.y),
                     uz = fabs((p.z - g.mn.z) * g.inv.z);
        const double ex = m * g.inv.x + 1e-9, ey = m * g.inv.y + 1e-9, ez = m * g.inv.z + 1e-9;
        on[1] = on[1] || ((!(mask & 1) || ux < 1.0 + ex) && (!(mask & 2) || uy < 1.0 + ey) && (!(mask & 4) || uz < 1.0 + ez));
        const bool stays = ((mask & 1) && ux >= 1.0 - ex) || ((mask & 2) && uy >= 1.0 - ey) || ((mask & 4) && uz >= 1.0 - ez);
        on[0] = on[0] || (stays && (ghost_key(p, g) >= 0 || p.z >= g.mx.y - m));
      }
      for (int v = 0; v < 2; ++v) {
        const unsigned b = __ballot_sync(FULL, on[v]);
        int at = 0;
        if (lane == 0 && b) at = atomicAdd(a.G.count, __popc(b));
        at = __shfl_sync(FULL, at, 0);
        if (on[v]) a.G.list[at + __popc(b & ((1u << lane) - 1u))] = 2 * (s * n + i) + v;
      }
    }
  }
  grid.sync();
  const int nimg = __ldcg(a.G.count);
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  const float gap = 0.8f * a.skin * (1.0f + 1e-5f);
  for (int v = tid >> 5; v < nimg; v += T >> 5) {  // one warp per image
    const int t = __ldcg(a.G.list + v), moved = t & 1, s = (t >> 1) / n, i = (t >> 1) % n;
    const double3 base = image_base(a.P.pos[i], g, a.wrap_axes, a.G.mask[s]), xw = wrap_pos(a.P.pos[i], g, a.wrap_axes);
    const double Rg = grid_reach(a, i);
    int kB;
    CandRec rb = cand_rec(a, i, kB);
    const float Rgs = (float)Rg + a.skin;
    // the second position only where the body crosses a face of an axis the set does not wrap
    const int places = a.cross && (base.x != xw.x || base.y != xw.y || base.z != xw.z) ? 2 : 1;
    for (int q = 0; q < places; ++q) {
      double3 xg = q == 0 ? base : xw;
      if (moved) xg += image_offset(g, a.G.mask[s]);
      const double r = (a.rmax + Rg + (double)a.skin) * 1.001 + 1e-4 * (fabs(xg.x) + fabs(xg.y) + fabs(xg.z));
      const int3 lo = ball_cell(xg - d3(r, r, r), g), hi = ball_cell(xg + d3(r, r, r), g);
      rb.p = make_float4((float)xg.x, (float)xg.y, (float)xg.z, 0.f);
      const float n1g = n1_f(rb.p);
      // one owner per lane (A < 0: none)
      auto add = [&](int A, float4 pa) {
        bool keep = false;
        const float R = (pa.w + Rgs) * (1.0f + 1e-4f) + 1e-5f * (n1g + n1_f(pa));
        if (A >= 0 && !(dist2_f(pa, rb.p) > R * R)) {
          int kA;
          const CandRec ra = cand_rec(a, A, kA);
          keep = !pair_separated<2>(sup, pa, n1_f(pa), ra.q, ra.sc, ra.sh, rb.p, rb.q, rb.sc, rb.sh, gap);
        }
        const unsigned b = __ballot_sync(FULL, keep);
        int at = 0;
        if (lane == 0 && b) at = atomicAdd(a.gl.count, __popc(b));
        at = __shfl_sync(FULL, at, 0) + __popc(b & ((1u << lane) - 1u));
        if (keep && at < a.gl.cap) a.gl.list[at] = make_int2(A | (moved ? (int)0x80000000u : 0), (i << 3) | s);
      };
      for (int z = lo.z; z <= hi.z; ++z) {
        for (int y = lo.y; y <= hi.y; ++y) {
          const int h0 = lin3(make_int3(lo.x, y, z), g.size);
          const int st = __ldcg(offs + h0 + 1), en = __ldcg(offs + h0 + (hi.x - lo.x) + 2);
          for (int k0 = st; k0 < en; k0 += 32) {
            const int k = min(k0 + lane, en - 1);
            add(k0 + lane < en ? __ldcg(idx + k) : -1, pk[k]);
          }
        }
      }
      for (int k0 = 0; !resort && k0 < n0 + nL; k0 += 32) {  // the bodies in no cell
        const int k = min(k0 + lane, n0 + nL - 1), A = __ldcg(idx1 + (k < n0 ? k : n - nL + k - n0));
        const double3 x = wrap_pos(a.P.pos[A], g, a.wrap_axes);
        add(k0 + lane < n0 + nL ? A : -1, make_float4((float)x.x, (float)x.y, (float)x.z, __ldg(a.rec_s + A).x));
      }
    }
  }
  grid.sync();
  if (tid == 0) {
    const int c = __ldcg(a.gl.count);
    atomicMax(&a.status->need_img, c);
    if (c > a.gl.cap) atomicOr(&a.status->flags, OVF_IMG);  // the batch re-runs with a longer list
  }
}

__global__ void __launch_bounds__(RB_THREADS, 2) k_rebuild(StepArgs a, BucketScratch w, ImageSort im,
                                                           int* __restrict__ sorted_idx, int* __restrict__ sums) {
  if (*a.reuse == 0) return;
  __shared__ int sw[32];
  __shared__ int s_buf[RB_THREADS / 32][32 * RB_BUF], s_cnt[RB_THREADS / 32][32];
  cg::grid_group grid = cg::this_grid();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
  const int n = a.P.n;
  int* cross_n = sums + REBUILD_SUMS;
  int* cross_list = w.tmp;  // the sort's, free after it
  if (tid == 0) *cross_n = 0;
  grid_cell_sort<true>(grid, a.P.key, n, a.pg.ncells, w, sorted_idx, sums, sw);
  if (tid == 0) atomicAdd(&a.status->builds, 1);
  for (int k = tid; k < n; k += T) pack_cell(a, k, __ldcg(sorted_idx + k));
  grid.sync();
  // Lists, threads in cell-sorted order (the lanes of a warp walk the same cells in step). A lane
  // walks until its shared buffer of bodies within reach + skin is full; the warp's buffers are
  // then tested one lane per pair, since a lane testing as it walks would leave most of the
  // warp idle (2M settling particles: 2.5 ms a rebuild that way, 1.7 ms now).
  // Where the bodies do not fill the grid's threads, 2 to 8 lanes share a body, each with its part of
  // the rows (3,000 polydisperse bodies at 5 m/s, rebuilt in 46 of 80 steps: 133 us a step with one
  // lane a body, 100 this way).
  const SupTabs sup{a.S.sup_n, a.S.sup_s, a.S.sup_r};
  const float gap = 0.8f * a.skin * (1.0f + 1e-5f);
  const int lane = threadIdx.x & 31;
  int* buf = s_buf[threadIdx.x >> 5];
  int* cnt = s_cnt[threadIdx.x >> 5];
  int sh = 0;  // 1 << sh lanes per body
  while (sh < 3 && (long long)n << (sh + 1) <= T) ++sh;
  const int body = lane >> sh, part = lane & ((1 << sh) - 1);
  int need = 0;
  for (int t0 = (tid >> 5) * (32 >> sh); t0 < n; t0 += (T >> 5) * (32 >> sh)) {
    const int t = t0 + body;
    float4 pa = make_float4(0.f, 0.f, 0.f, 0.f);
    float n1a = 0.f;
    int A = 0, r = 0, rows = 0, ny = 1, k = 0, en = 0;
    int3 lo = make_int3(0, 0, 0), hi = lo;
    double3 xA = d3(0., 0., 0.);
    if (t < n) {
      pa = a.cell_pk[t];
      n1a = n1_f(pa);
      A = a.pk_meta[t].y;
      xA = a.P.pos[A];
      // A's ball of reach + skin can reach past the 27 cells (cells are only 2 rmax wide;
      // reach + skin is up to 2.1 rmax): every cell it overlaps is walked (at most two more per
      // side), with a rounding margin far beyond the FP32 test's
      const double R = a.P.radius[A] + a.rmax + (double)a.skin;
      const double ext = 1.001 * R + 1e-4 * (fabs(xA.x) + fabs(xA.y) + fabs(xA.z) + 4.0 * R);
      const int3 c = clamp_cell(cell_of(xA, a.pg), a.pg.size);
      lo = ball_cell(xA - d3(ext, ext, ext), a.pg);
      hi = ball_cell(xA + d3(ext, ext, ext), a.pg);
      lo = make_int3(min(lo.x, max(c.x - 1, 0)), min(lo.y, max(c.y - 1, 0)), min(lo.z, max(c.z - 1, 0)));
      hi = make_int3(max(hi.x, min(c.x + 1, a.pg.size.x - 1)), max(hi.y, min(c.y + 1, a.pg.size.y - 1)),
                     max(hi.z, min(c.z + 1, a.pg.size.z - 1)));
      ny = hi.y - lo.y + 1;
      rows = ny * (hi.z - lo.z + 1);
      r = (rows * part) >> sh;
      rows = (rows * (part + 1)) >> sh;
    }
    cnt[lane] = 0;
    while (__any_sync(FULL, r < rows || k < en)) {
      int m = 0;
      while (m <= RB_BUF - 4) {
        if (k >= en) {
          if (r >= rows) break;
          // the cells of a row are contiguous in the sorted order
          const int h0 = lin3(make_int3(lo.x, lo.y + r % ny, lo.z + r / ny), a.pg.size);
          k = __ldcg(w.offs + h0 + 1);
          en = __ldcg(w.offs + h0 + (hi.x - lo.x) + 2);
          ++r;
          continue;
        }
        float4 pb[4];  // four bodies' loads in flight
#pragma unroll
        for (int u = 0; u < 4; ++u) pb[u] = a.cell_pk[min(k + u, en - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k + u < en && in_reach(a, pa, n1a, pb[u]) && a.pk_meta[k + u].y > A) buf[32 * m++ + lane] = k + u;
        k += 4;
      }
      int incl = m;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(FULL, incl, 31);
      __syncwarp();
      for (int i0 = 0; i0 < total; i0 += 32) {
        const int i = i0 + lane;
        const int ow = lane_of(incl, i);
        const int first = __shfl_sync(FULL, incl - m, ow), oA = __shfl_sync(FULL, A, ow);
        const int ob = ow >> sh, fb = __shfl_sync(FULL, incl - m, ob << sh);  // the body, its first entry
        bool keep = false;
        int B = 0;
        if (i < total) {
          const int kB = buf[32 * (i - first) + ow], to = t0 + ob;
          const int4 mA = a.pk_meta[to], mB = a.pk_meta[kB];
          const float4 po = a.cell_pk[to];
          B = mB.y;
          keep = !pair_separated<2>(sup, po, n1_f(po), a.pk_q[to], __int_as_float(mA.w), mA.z, a.cell_pk[kB],
                                    a.pk_q[kB], __int_as_float(mB.w), mB.z, gap);
        }
        const unsigned mk = __ballot_sync(FULL, keep);
        const int at = cnt[ob] + __popc(mk & ((1u << lane) - 1u) & (~0u << max(fb - i0, 0)));
        if (keep && at < a.nbr_cap) a.nbr[(size_t)at * n + oA] = B;
        const int nx = __shfl_down_sync(FULL, ob, 1);
        __syncwarp();
        if (i < total && (lane == 31 || nx != ob || i + 1 == total)) cnt[ob] = at + keep;
        __syncwarp();
      }
    }
    if (t < n && part == 0) {
      const int nl = cnt[body];
      // an overflowed list: the batch re-runs with longer lists
      a.nbr_cnt[A] = nl <= a.nbr_cap ? nl : -1;
      if (nl > a.nbr_cap) atomicOr(&a.status->flags, OVF_NBR);
      need = max(need, nl);
      // where the body stands from the next step on
      const double3 xw = a.cross ? wrap_pos(xA, a.pg, a.wrap_axes) : xA;
      a.xb[A] = xw;
      const int k0 = a.pk_meta[t].x, kw = a.cross && k0 < 0 ? hash_key(xw, a.pg) : k0;
      a.kin[A] = kw >= 0;
      if (k0 < 0 && (xw.x != xA.x || xw.y != xA.y || xw.z != xA.z)) cross_list[atomicAdd(cross_n, 1)] = A;
      const Quat q = a.P.quat[A];
      a.qb[A] = make_float4((float)q.q0, (float)q.q1, (float)q.q2, (float)q.q3);
    }
    __syncwarp();
  }
  need = __reduce_max_sync(FULL, need);
  if (lane == 0 && need > 0) atomicMax(&a.status->need_nbr, need);
  if (a.cross) {
    grid.sync();
    grid_cross_lists(a, w, sorted_idx, cross_list, __ldcg(cross_n));
  }
  if (a.gl.list) grid_image_list(grid, a, w, sorted_idx, im, sums, sw);
}

void launch_rebuild(const StepArgs& a, const BucketScratch& w, const ImageSort& img, int* sorted_idx, int* sums,
                    cudaStream_t s) {
  static int blocks = 0;  // resident at once, the same on every B200
  if (blocks == 0) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rebuild, RB_THREADS, 0);
    blocks = std::min(std::max(1, sms * per), REBUILD_SUMS / 2);
  }
  if (a.P.n <= 0) return;
  // One thread per two buckets; four per body, or one block, whose barriers are the cheapest; with
  // images, a block per 64 pairs of a set and a body (201 bodies in a narrow box that rebuild in two of
  // three steps: 190 us a step with one block, 99 with 22)
  int want = (a.pg.ncells / 2 + RB_THREADS) / RB_THREADS;
  if (a.P.n > RB_THREADS) want = (int)std::max<long long>(want, (4ll * a.P.n + RB_THREADS - 1) / RB_THREADS);
  if (a.gl.list) want = (int)std::max<long long>(want, ((long long)a.G.nsets * a.P.n + 63) / 64);
  StepArgs aa = a;
  BucketScratch ww = w;
  ImageSort im = img;
  void* args[] = {&aa, &ww, &im, &sorted_idx, &sums};
  cudaLaunchCooperativeKernel((const void*)k_rebuild, dim3(std::min(want, blocks)), dim3(RB_THREADS), args, 0, s);
}

}  // namespace lsdem
