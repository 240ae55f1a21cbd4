// Lane-parallel search of one mesh for one point (sm_100a): all 32 lanes of a warp work on the same
// query, each on another child of the tree or another triangle.
//
// A packet of 32 queries (mesh_sdf.cu) shares its node and triangle reads, which pays when the 32
// points are neighbours.  A few scattered points are not: their packet opens what any of them
// needs, and a call of n points fills only n / 32 warps.  Here a round takes up to eight nodes off
// the stack and tests their 32 children at once, four leaves' triangles go through the 32 lanes
// together, and a call of n points fills n warps.
//
// The pruning bound does not wait for the first triangles: a tight axis-aligned box has a triangle
// touching each of its faces, so the nearest of the faces' farthest corners (the "min-max" distance)
// bounds the distance to the surface from above, and the search can go breadth-first without opening
// much that a best-first order would not.
#ifndef EBG_MESH_POINT_CUH
#define EBG_MESH_POINT_CUH

#include <cfloat>

#include "ebg_device.cuh"
#include "mesh_traverse.cuh"

namespace ebg {

// Node entries per warp.  A round of eight nodes starts only at or below POINT_WIDE entries and so
// ends with at most POINT_WIDE + 24; above it a round takes one node, which adds at most 3 entries
// per tree level, and the builder accepts at most (EBG_STACK_DEPTH - 1) / 3 levels.
constexpr int POINT_WIDE   = 64;
constexpr int POINT_NODES  = POINT_WIDE + 24 + EBG_STACK_DEPTH;
constexpr int POINT_LEAVES = 64; // a round adds at most 32 to at most 32

struct PointMem
{
  uint32_t ref[POINT_NODES];
  float    key[POINT_NODES];
  uint32_t leafRef[POINT_LEAVES];
  uint32_t leafCount[POINT_LEAVES];
  float    leafKey[POINT_LEAVES];
};

// Squared min-max distance: the smallest over the box's faces of the distance to the face's
// farthest point, for the face of each axis nearest to p.
__device__ __forceinline__ float boxMinMax2(float lx, float ly, float lz, float hx, float hy, float hz, float px,
                                            float py, float pz)
{
  const float ax = fabsf(px - lx), bx = fabsf(px - hx), nx = fminf(ax, bx), fx = fmaxf(ax, bx);
  const float ay = fabsf(py - ly), by = fabsf(py - hy), ny = fminf(ay, by), fy = fmaxf(ay, by);
  const float az = fabsf(pz - lz), bz = fabsf(pz - hz), nz = fminf(az, bz), fz = fmaxf(az, bz);
  const float qx = fx * fx, qy = fy * fy, qz = fz * fz;
  return fminf(fmaf(nx, nx, qy + qz), fminf(fmaf(ny, ny, qx + qz), fmaf(nz, nz, qx + qy)));
}

// Runs `tris(active, triangle)` -- all 32 lanes together -- over the triangles of every leaf whose
// boxes lie within `bound` (squared, warp-uniform; the callback lowers it).  With UPPER, boxes lower
// it too: an upper bound r of the distance becomes r * 1.00001 + slack, which covers the FP32 error
// of the triangle distances that are compared with it.  With FIRST the search ends after the first
// leaves, the nearest found so far: a near triangle, not always the nearest.  Returns ST_* bits.
template <bool UPPER, bool FIRST = false, class TriFn>
__device__ __forceinline__ int pointSearch(const EbgMeshView& m, float px, float py, float pz, float& bound, float slack,
                                           PointMem& w, TriFn&& tris)
{
  const int      lane = threadIdx.x & 31;
  const unsigned lt   = (1u << lane) - 1u;
  const float    inf  = __int_as_float(0x7f800000);
  int            sp = 0, nl = 0;
  if (m.root_ref & EBG_LEAF_BIT) {
    if (lane == 0) {
      w.leafRef[0]   = m.root_ref;
      w.leafCount[0] = m.root_count;
      w.leafKey[0]   = 0.f;
    }
    nl = 1;
  }
  else {
    if (lane == 0) {
      w.ref[0] = m.root_ref;
      w.key[0] = boxDist2(m.root_lo[0], m.root_lo[1], m.root_lo[2], m.root_hi[0], m.root_hi[1], m.root_hi[2], px, py, pz);
    }
    sp = 1;
  }
  __syncwarp();
  uint32_t iters = 0;
#pragma unroll 1
  while (sp > 0 || nl > 0) {
    if (++iters > MAX_ITERS) {
      return ST_ITERS;
    }
    if (nl > POINT_LEAVES - 32 || sp == 0) {
      // keep the leaves still within the bound, put the nearest on top, take the top four
      const float    k0 = lane < nl ? w.leafKey[lane] : inf, k1 = lane + 32 < nl ? w.leafKey[lane + 32] : inf;
      const bool     keep0 = k0 <= bound, keep1 = k1 <= bound;
      const unsigned b0 = __ballot_sync(FULL, keep0), b1 = __ballot_sync(FULL, keep1);
      const int      n0 = __popc(b0), total = n0 + __popc(b1);
      if (total == 0) {
        nl = 0;
        continue;
      }
      const float    mine = fminf(keep0 ? k0 : inf, keep1 ? k1 : inf);
      const uint32_t least = __reduce_min_sync(FULL, __float_as_uint(mine));
      const int      r0 = __popc(b0 & lt), r1 = n0 + __popc(b1 & lt);
      int            at = total; // the compacted place of the nearest leaf
      at                = keep1 && __float_as_uint(k1) == least ? r1 : at;
      at                = keep0 && __float_as_uint(k0) == least ? r0 : at;
      at                = int(__reduce_min_sync(FULL, uint32_t(at)));
      uint32_t ref0 = 0, cnt0 = 0, ref1 = 0, cnt1 = 0;
      if (keep0) {
        ref0 = w.leafRef[lane];
        cnt0 = w.leafCount[lane];
      }
      if (keep1) {
        ref1 = w.leafRef[lane + 32];
        cnt1 = w.leafCount[lane + 32];
      }
      __syncwarp(); // every entry is read before any is overwritten
      // the nearest and the last change places
      auto place = [&](int r) { return r == at ? total - 1 : (r == total - 1 ? at : r); };
      if (keep0) {
        const int p    = place(r0);
        w.leafRef[p]   = ref0;
        w.leafCount[p] = cnt0;
        w.leafKey[p]   = k0;
      }
      if (keep1) {
        const int p    = place(r1);
        w.leafRef[p]   = ref1;
        w.leafCount[p] = cnt1;
        w.leafKey[p]   = k1;
      }
      __syncwarp();
      const int      g = lane >> 3, idx = total - 1 - g;
      const uint32_t t0  = idx >= 0 ? w.leafRef[idx] & ~EBG_LEAF_BIT : 0u;
      const int      cnt = idx >= 0 ? int(w.leafCount[idx] & EBG_COUNT_MASK) : 0;
      nl                 = total > 4 ? total - 4 : 0;
      const int most     = int(__reduce_max_sync(FULL, uint32_t(cnt)));
      __syncwarp(); // the next round may overwrite the taken entries
      for (int t = 0; t < most; t += 8) {
        const int j = t + (lane & 7);
        tris(j < cnt, t0 + uint32_t(j < cnt ? j : 0));
      }
      if (FIRST) {
        return 0;
      }
      continue;
    }
    const int  take = sp <= POINT_WIDE ? (sp < 8 ? sp : 8) : 1;
    const int  g    = lane >> 2, k = lane & 3;
    bool       need = g < take && w.key[g < take ? sp - 1 - g : 0] <= bound;
    uint32_t   child = 0, cw = 0;
    float      d2 = inf, up = inf;
    if (need) {
      const float4* sl = reinterpret_cast<const float4*>(m.children + 4 * size_t(w.ref[sp - 1 - g]) + k);
      const float4  lo = __ldg(sl), hi = __ldg(sl + 1);
      child = __float_as_uint(lo.w);
      cw    = __float_as_uint(hi.w);
      need  = (child | cw) != 0u; // an empty slot
      if (need) {
        d2 = boxDist2(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, px, py, pz);
        up = boxMinMax2(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, px, py, pz);
      }
    }
    sp -= take;
    if (UPPER) {
      const float u = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(up)));
      const float r = sqrtf(u) * 1.00001f + slack;
      bound         = fminf(bound, r * r);
    }
    need            = need && d2 <= bound;
    const bool leaf = (child & EBG_LEAF_BIT) != 0u;
    if (need && (leaf || (cw & EBG_NODE_HAS_OBB))) {
      const float4* ob = reinterpret_cast<const float4*>(leaf ? m.obb + (cw >> EBG_COUNT_BITS) : m.node_obb + child);
      d2   = fmaxf(d2, obbDist2(__ldg(ob), __ldg(ob + 1), __ldg(ob + 2), __ldg(ob + 3), px, py, pz));
      need = d2 <= bound;
    }
    const unsigned ml = __ballot_sync(FULL, need && leaf), mn = __ballot_sync(FULL, need && !leaf);
    __syncwarp(); // the taken entries are read before they are overwritten
    if (need && leaf) {
      const int p    = nl + __popc(ml & lt);
      w.leafRef[p]   = child;
      w.leafCount[p] = cw;
      w.leafKey[p]   = d2;
    }
    if (need && !leaf) {
      const int p = sp + __popc(mn & lt);
      w.ref[p]    = child;
      w.key[p]    = d2;
    }
    nl += __popc(ml);
    sp += __popc(mn);
    __syncwarp();
    if (sp > POINT_NODES - 4) { // never for trees the builder accepts
      return ST_STACK;
    }
  }
  return 0;
}

// The nearest triangle (FP32, ties to the lower leaf position, as in the packet traversal) of one point among
// those nearer than the root of bd2; bt stays as it is if there is none.  FIRST as for pointSearch.
// The boxes' upper bounds hold for exact distances.  Where every FP32 distance is above them by more than
// `slack` (squares that underflow, triangles that FP32 cannot tell from a line) the search runs again
// without them.
template <bool FIRST = false>
__device__ __forceinline__ int pointNearest(const EbgMeshView& m, float px, float py, float pz, float slack, PointMem& w,
                                            float& bd2, int& bt)
{
  const float inf   = __int_as_float(0x7f800000);
  float       bound = bd2;
  int         err   = 0;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    err |= pointSearch<true, FIRST>(m, px, py, pz, bound, slack, w, [&](bool active, uint32_t tri) {
      float dd = inf;
      if (active) {
        const float4* h  = reinterpret_cast<const float4*>(m.hot + tri);
        const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
        float         s, t;
        int           r;
        dd = triDist2<false>(h0, h1, h2, px, py, pz, s, t, r);
      }
      const uint32_t mb = __reduce_min_sync(FULL, __float_as_uint(dd));
      const uint32_t mt = __reduce_min_sync(FULL, __float_as_uint(dd) == mb ? tri : 0x7fffffffu);
      const float    md = __uint_as_float(mb);
      if (md < bd2 || (md == bd2 && int(mt) < bt)) {
        bd2   = md;
        bt    = int(mt);
        bound = fminf(bound, bd2);
      }
    });
    if (FIRST || bound >= bd2) {
      break;
    }
    slack = inf; // shrinks nothing
    bound = bd2;
  }
  return err;
}

// ---- eight lanes per point ---------------------------------------------------------------------------
//
// With more points than warps the 32 lanes of pointSearch are too many for one point: most rounds
// have fewer than 32 children worth testing.  Here four points share a warp, each with eight lanes:
// a round takes the two entries on top of the group's stack, pushes the children in order of
// distance (nearest on top) and then tests the leaf on top, if one is.

// Entries per group: a round of two nodes starts at or below GROUP_WIDE entries and adds at most 6;
// above it a round takes one node, which adds at most 3 entries per tree level.
constexpr int GROUP_WIDE  = 24;
constexpr int GROUP_STACK = GROUP_WIDE + 6 + EBG_STACK_DEPTH;

struct GroupMem
{
  uint32_t ref[GROUP_STACK], count[GROUP_STACK];
  float    key[GROUP_STACK];
};

// The least value of x over the eight lanes of each group.
__device__ __forceinline__ float groupMin(float x)
{
  x = fminf(x, __shfl_xor_sync(FULL, x, 1));
  x = fminf(x, __shfl_xor_sync(FULL, x, 2));
  return fminf(x, __shfl_xor_sync(FULL, x, 4));
}

// Runs `leaf(test, t0, cnt, most)` for the leaves of each group's point whose boxes lie within the group's
// `bound` (squared; the callback lowers it): triangles [t0, t0 + cnt) where `test`, `most` the warp's
// largest cnt.  Groups without a point pass on = false.  UPPER and slack as for pointSearch.  All 32
// lanes call it together; `g` is the group's memory.  Returns ST_* bits.
template <bool UPPER, class LeafFn>
__device__ __forceinline__ int groupSearch(const EbgMeshView& m, bool on, float px, float py, float pz, float& bound,
                                           float slack, GroupMem& g, LeafFn&& leaf)
{
  const int      lane = threadIdx.x & 31, sub = lane & 7, base = lane & 24;
  const unsigned mine = 0xffu << base;
  const float    inf  = __int_as_float(0x7f800000);
  int            sp   = on ? 1 : 0;
  if (on && sub == 0) {
    g.ref[0]   = m.root_ref;
    g.count[0] = m.root_count;
    g.key[0]   = boxDist2(m.root_lo[0], m.root_lo[1], m.root_lo[2], m.root_hi[0], m.root_hi[1], m.root_hi[2], px, py, pz);
  }
  __syncwarp();
  uint32_t iters = 0;
#pragma unroll 1
  while (true) {
    // down to the topmost entry still within the bound, eight at a time
    {
      const int      i   = sp - 1 - sub;
      const unsigned ok  = (__ballot_sync(FULL, i >= 0 && g.key[i >= 0 ? i : 0] <= bound) & mine) >> base;
      sp                 = ok != 0u ? sp - (__ffs(int(ok)) - 1) : (sp > 8 ? sp - 8 : 0);
      if (!__any_sync(FULL, sp > 0)) {
        return 0;
      }
      if (++iters > MAX_ITERS) {
        return ST_ITERS;
      }
    }
    // the node on top and the entry below it, if that is a node as well
    const uint32_t top  = sp > 0 ? g.ref[sp - 1] : EBG_LEAF_BIT;
    const bool     node = !(top & EBG_LEAF_BIT) && (sp > 0 && g.key[sp > 0 ? sp - 1 : 0] <= bound);
    if (__any_sync(FULL, node)) {
      const uint32_t below = node && sp > 1 && sp <= GROUP_WIDE ? g.ref[sp - 2] : EBG_LEAF_BIT;
      const bool     two   = !(below & EBG_LEAF_BIT);
      const uint32_t ref   = sub < 4 ? top : below;
      bool           need  = node && (sub < 4 || two);
      uint32_t       child = 0, cw = 0;
      float          d2 = inf, up = inf;
      if (need) {
        const float4* sl = reinterpret_cast<const float4*>(m.children + 4 * size_t(ref) + (sub & 3));
        const float4  lo = __ldg(sl), hi = __ldg(sl + 1);
        child = __float_as_uint(lo.w);
        cw    = __float_as_uint(hi.w);
        need  = (child | cw) != 0u; // an empty slot
        if (need) {
          d2 = boxDist2(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, px, py, pz);
          if (UPPER) {
            up = boxMinMax2(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, px, py, pz);
          }
        }
      }
      if (UPPER) {
        const float r = sqrtf(groupMin(up)) * 1.00001f + slack;
        bound         = fminf(bound, r * r);
      }
      need             = need && d2 <= bound;
      const bool isLeaf = (child & EBG_LEAF_BIT) != 0u;
      if (need && (isLeaf || (cw & EBG_NODE_HAS_OBB))) {
        const float4* ob = reinterpret_cast<const float4*>(isLeaf ? m.obb + (cw >> EBG_COUNT_BITS) : m.node_obb + child);
        d2   = fmaxf(d2, obbDist2(__ldg(ob), __ldg(ob + 1), __ldg(ob + 2), __ldg(ob + 3), px, py, pz));
        need = d2 <= bound;
      }
      // farther children deeper (ties by lane)
      const float mk   = need ? d2 : -1.f;
      int         rank = 0, all = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float ok = __shfl_sync(FULL, mk, i, 8);
        rank += int(ok > mk || (ok == mk && i < sub));
        all += int(ok >= 0.f);
      }
      sp -= node ? (two ? 2 : 1) : 0;
      __syncwarp(); // the taken entries are read before they are overwritten
      if (need) {
        g.ref[sp + rank]   = child;
        g.count[sp + rank] = cw;
        g.key[sp + rank]   = d2;
      }
      sp += all;
      __syncwarp();
      if (__any_sync(FULL, sp > GROUP_STACK - 8)) { // never for trees the builder accepts
        return ST_STACK;
      }
    }
    // the leaf on top
    const uint32_t lr   = sp > 0 ? g.ref[sp - 1] : 0u;
    const bool     test = (lr & EBG_LEAF_BIT) && g.key[sp > 0 ? sp - 1 : 0] <= bound;
    if (__any_sync(FULL, test)) {
      const uint32_t t0  = lr & ~EBG_LEAF_BIT;
      const int      cnt = test ? int(g.count[sp - 1] & EBG_COUNT_MASK) : 0;
      sp -= test ? 1 : 0;
      __syncwarp(); // read before it is overwritten
      leaf(test, t0, cnt, int(__reduce_max_sync(FULL, uint32_t(cnt))));
    }
  }
}

// The nearest triangle of each group's point, as pointNearest finds it.
__device__ __forceinline__ int groupNearest(const EbgMeshView& m, bool on, float px, float py, float pz, float slack,
                                            GroupMem& g, float& bd2, int& bt)
{
  const int   sub   = threadIdx.x & 7;
  const float inf   = __int_as_float(0x7f800000);
  float       bound = FLT_MAX, b = FLT_MAX;
  int         best  = -1, err = 0;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    err |= groupSearch<true>(m, on, px, py, pz, bound, slack, g, [&](bool test, uint32_t t0, int cnt, int most) {
      float dd  = inf;
      int   tri = 0x7fffffff;
      for (int t = sub; t < most; t += 8) {
        if (t < cnt) {
          const float4* h  = reinterpret_cast<const float4*>(m.hot + t0 + t);
          const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
          float         s_, t_;
          int           r_;
          const float   d = triDist2<false>(h0, h1, h2, px, py, pz, s_, t_, r_);
          if (d < dd) {
            dd  = d;
            tri = int(t0) + t;
          }
        }
      }
      const float dm = groupMin(dd);
      tri            = dd == dm ? tri : 0x7fffffff;
      tri            = min(tri, __shfl_xor_sync(FULL, tri, 1));
      tri            = min(tri, __shfl_xor_sync(FULL, tri, 2));
      tri            = min(tri, __shfl_xor_sync(FULL, tri, 4));
      if (test && (dm < b || (dm == b && tri < best))) {
        b     = dm;
        best  = tri;
        bound = fminf(bound, b);
      }
    });
    on = on && bound < b;
    if (!__any_sync(FULL, on)) {
      break;
    }
    slack = inf; // shrinks nothing
    bound = b;
  }
  bd2 = b;
  bt  = best;
  return err;
}

// Lower bound of the distance from p to a triangle from the closest point that triDist2 found: with
// w the unit vector from it to p, no point of the triangle is nearer than the least of
// w . (p - vertex).  It holds for any w, so an inexact closest point (a sliver) only makes it lower.
__device__ __forceinline__ float triLower(const float4 h0, const float4 h1, const float4 h2, float px, float py, float pz,
                                          float s, float t, float d2)
{
  const float apx = px - h0.x, apy = py - h0.y, apz = pz - h0.z;
  const float dx = fmaf(-t, h2.x, fmaf(-s, h1.x, apx));
  const float dy = fmaf(-t, h2.y, fmaf(-s, h1.y, apy));
  const float dz = fmaf(-t, h2.z, fmaf(-s, h1.z, apz));
  const float a  = fmaf(dx, apx, fmaf(dy, apy, dz * apz));
  const float b  = fmaf(dx, h1.x, fmaf(dy, h1.y, dz * h1.z));
  const float c  = fmaf(dx, h2.x, fmaf(dy, h2.y, dz * h2.z));
  return (a - fmaxf(0.f, fmaxf(b, c))) * rsqrtf(d2);
}

} // namespace ebg

#endif
