// FP32 mesh signed distance of many points (sm_100a): packets of 32 neighbouring queries whose tree
// search runs once per packet, on the packet's box, with the 32 lanes on 32 different children.
//
// A packet's depth-first walk (mesh_sdf.cu) tests every node, oriented box and leaf with all 32
// points, one after another: about 37,000 warp instructions per packet of the 512^3 grid on 1.3 M
// triangles, most of them for entries that no lane turns out to need.  Here a lane decides for one
// entry whether ANY point of the packet can need it:
//   - `a` is a point of the mesh near the packet, so a query p is at most |p - a| from the mesh;
//   - e is the entry's point nearest to the packet's centre c, u the unit vector from e to c; the
//     entry (convex) lies behind the plane through e with normal u, so it is at least u . (p - e)
//     from p;
//   - |p - a| - u . (p - e) is convex in p, so over the packet's box it is largest at a corner: where it
//     is negative at all eight corners, no query of the packet needs the entry.
// Unlike a bound from two radii, this keeps what lies beside the packet's own patch only as far as
// the directions to it and to `a` differ.  What is left is a list of leaves for the lanes to test with
// their own bounds.
//
// Packets come off the work counter in groups of up to eight neighbours.  A group's box is taken
// down the tree once, as far as at most 32 entries reach; its packets start there.  The winners of one
// packet give the next its `a` and its lanes' first bounds (a query that passes an attached model takes
// both from its cells instead: the anchors, and the model's radius where that is smaller).
//
// The list is tested in three steps.  The two leaves nearest to c go through all lanes, which brings
// the bounds near their final values; then a lane per leaf tests its oriented box against the 32
// points and bounds, which gives the (lane, leaf) pairs that are left; 32 pairs at a time, a lane per
// pair, test their triangles, and the results meet in a 64-bit minimum of (d2, triangle) per query.
//
// A packet too wide for one box is divided at its widest step.  What stays too wide, holds too few
// points or reaches too many leaves (points few against the tree's leaves, or near the medial axis) is
// put aside for kMeshAside: eight lanes search for each such point, or, where a packet is too wide as a whole
// but its points share what they reach, the walk for all of them (sharesReach).
//
// Bound by the L1's data stage (89 % of its wavefronts) and by instruction issue (69 %): per packet of
// the 512^3 grid 10 rounds of 32 children, 104 listed leaves, 27 of them with a pair, 7 passes over
// pairs, about 19,000 warp instructions.  B200, 151 M points on 1.3 M triangles, the walk -> here:
// traversal 172.6 -> 79.0 ms, with a model 92.3 -> 70.6 ms; 1 M uniform points on 20,480 triangles
// 1.42 -> 0.73 ms, 8 M on 327,680 11.6 -> 7.4 ms; 8 M about two spheres 12.5 -> 13.1 ms.
#include <algorithm>
#include <cfloat>

#include "ebg_device.cuh"
#include "mesh_kernels.h"
#include "mesh_packet.cuh"
#include "mesh_point.cuh"
#include "mesh_traverse.cuh"

namespace ebg {

namespace {

constexpr int PACKET_WARPS = 4;
constexpr int PACKET_PAIRS = 256; // (lane, leaf) pairs waiting for their triangle tests

// A mesh triangle near a point (all lanes on the same point; -1 if none is found).
__device__ __noinline__ int nearTriangle(const EbgMeshView& m, float px, float py, float pz, float delta, PointMem& w, int& bt)
{
  float bd2 = FLT_MAX;
  bt        = -1;
  return pointNearest<true>(m, px, py, pz, delta, w, bd2, bt);
}

constexpr int PACKET_FRONT = 32; // entries of a group's frontier

// Leaves per point up to which a wide packet takes the walk.  8 M uniform points, 0.05, 0.1, 0.2 and 0.5: about
// two spheres of 81,920 triangles each 15.7, 13.8, 13.4 and 13.1 ms, about a 5:1 ellipsoid of 327,680 19.9, 17.9,
// 16.7 and 16.5, about a round body of 327,680 7.9, 7.8, 8.1 and 8.3.
constexpr float WALK_LEAVES = 0.2f;

struct PacketMem
{
  float4             query[32]; // the lanes' points and bounds
  unsigned long long key[32];   // the lanes' best (d2, triangle)
  float4             corner[2]; // the corners' bounds
  float4             last;      // centre and half-extent of the box before
  uint32_t           front[PACKET_FRONT], frontCount[PACKET_FRONT]; // child and count words
  uint32_t           pairTri[PACKET_PAIRS];                         // (lane, leaf) pairs: first triangle,
  uint16_t           pairLane[PACKET_PAIRS];                        // triangle count and lane
  PointMem           w;
};

// A query's results from its winning triangle (-1: none).
__device__ __forceinline__ void store(const MeshQueryArgs& a, const EbgMeshView& m, int tri, float px, float py, float pz,
                                      uint32_t id, int64_t pos)
{
  const float dist = tri >= 0 ? signedFromWinner(m, uint32_t(tri), px, py, pz) : FLT_MAX;
  a.out_d[id]      = dist;
  if (a.out_tri) {
    a.out_tri[id] = tri >= 0 ? (a.tri_leaf ? tri : __ldg(m.tri_id + tri)) : -1;
  }
  if (a.out_d64 && tri < 0) {
    a.out_d64[id] = double(FLT_MAX); // not among the FP64 pass's queries
  }
  if (a.band_flag) {
    // one flag per sorted position; the list is compacted from them in position order
    a.band_flag[pos] = uint8_t(tri >= 0 && fabsf(dist) <= a.band);
  }
}

// What kMeshPacket32 put aside: first the packets (each a long chain of reads), then the points, eight lanes
// each; a warp takes what is next.
__global__ void __launch_bounds__(32 * PACKET_WARPS, 8) kMeshAside(const __grid_constant__ MeshQueryArgs a, float delta)
{
  union Mem
  {
    float4   stack[2 * EBG_STACK_DEPTH + 32];
    GroupMem group[4];
  };
  __shared__ Mem     mem[PACKET_WARPS];
  Mem&               w    = mem[threadIdx.x >> 5];
  const EbgMeshView& m    = a.mesh;
  const int          lane = threadIdx.x & 31;
  const uint32_t     np   = a.later_count[1];
  while (np != 0u) {
    uint32_t i = 0;
    if (lane == 0) {
      i = atomicAdd(a.later_count + 2, 1u);
    }
    i = __shfl_sync(FULL, i, 0);
    if (i >= np) {
      break;
    }
    const uint32_t* e    = a.point_list + (a.n - 2 * (int64_t(i) + 1));
    const int64_t   pos  = int64_t(__ldg(e)) * 32 + lane;
    const bool      mine = (__ldg(e + 1) >> lane) & 1u;
    const int64_t   src  = pos < a.n ? pos : a.n - 1;
    const uint32_t  id   = a.order ? __ldg(a.order + src) : uint32_t(src);
    const float     px = __ldg(a.points + 3 * size_t(id)), py = __ldg(a.points + 3 * size_t(id) + 1),
                pz = __ldg(a.points + 3 * size_t(id) + 2);
    float             best = mine ? FLT_MAX : -1.f; // a lane that was not left needs nothing
    int               bt = -1, err = 0;
    uint32_t          iters = 0;
    TraversalCounters tc;
    traverseMesh<false, EBG_STACK_DEPTH>(m, px, py, pz, best, bt, w.stack, w.stack + 2 * EBG_STACK_DEPTH, iters, err, tc);
    if (err && lane == 0) {
      atomicOr(a.status, err);
    }
    if (mine) {
      store(a, m, bt, px, py, pz, id, pos);
    }
    __syncwarp();
  }
  const uint32_t n   = a.band_count[1];
  const uint32_t grp = uint32_t(lane) >> 3;
  while (n != 0u) {
    uint32_t i0 = 0;
    if (lane == 0) {
      i0 = atomicAdd(a.later_count + 3, 4u);
    }
    i0 = __shfl_sync(FULL, i0, 0);
    if (i0 >= n) {
      break;
    }
    const uint32_t i   = i0 + grp;
    const bool     on  = i < n;
    const uint32_t pos = __ldg(a.point_list + (on ? i : i0));
    const uint32_t id  = a.order ? __ldg(a.order + pos) : pos;
    const float    px = __ldg(a.points + 3 * size_t(id)), py = __ldg(a.points + 3 * size_t(id) + 1),
                pz = __ldg(a.points + 3 * size_t(id) + 2);
    float     bd2;
    int       bt;
    const int err = groupNearest(m, on, px, py, pz, delta, w.group[grp], bd2, bt);
    if (on && (lane & 7) == 0) {
      if (err) {
        atomicOr(a.status, err);
      }
      store(a, m, bt, px, py, pz, id, pos);
    }
    __syncwarp();
  }
}

// 32 waiting pairs (or the last ones): a lane per pair tests its leaf's triangles.
__device__ __forceinline__ void testPairs(const EbgMeshView& m, PacketMem& pm, int first, int count)
{
  const int      lane = threadIdx.x & 31;
  const bool     on   = lane < count;
  uint32_t       tt = on ? pm.pairTri[first + lane] : 0u;
  const uint32_t v  = on ? pm.pairLane[first + lane] : 0u;
  const uint32_t te = tt + (v >> 5), ql = v & 31u;
  const float4   q  = pm.query[ql];
  float          d  = __int_as_float(0x7f800000);
  uint32_t       di = 0u;
#pragma unroll 1
  for (; tt < te; tt++) {
    const float4* h  = reinterpret_cast<const float4*>(m.hot + tt);
    const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
    float         s, t;
    int           r;
    const float   dd = triDist2<false>(h0, h1, h2, q.x, q.y, q.z, s, t, r);
    if (dd < d) { // the lower position on ties
      d  = dd;
      di = tt;
    }
  }
  if (on && d <= q.w) {
    atomicMin(pm.key + ql, (unsigned long long)__float_as_uint(d) << 32 | di);
  }
}

// The cell of an attached model that holds a point (nearest cell outside the grid).
__device__ __forceinline__ int64_t cellOf(const SeedCellsView& cv, float px, float py, float pz)
{
  const float gm = float(cv.g - 1);
  const int   ix = int(fminf(fmaxf((px - cv.lo[0]) * cv.inv[0], 0.f), gm));
  const int   iy = int(fminf(fmaxf((py - cv.lo[1]) * cv.inv[1], 0.f), gm));
  const int   iz = int(fminf(fmaxf((pz - cv.lo[2]) * cv.inv[2], 0.f), gm));
  return (int64_t(iz) * cv.g + iy) * cv.g + ix;
}

// A cell's anchor, the triangle nearest to its centre, or -1.
__device__ __forceinline__ int cellAnchor(const SeedCellsView& cv, int64_t cell)
{
  return cv.anchor ? __ldg(cv.anchor + cell) : -1;
}

// The model's bound of |d| in the cell that holds a point: FLT_MAX outside the grid, where it says nothing.
__device__ __forceinline__ float cellRadius(const SeedCellsView& cv, int64_t cell, float px, float py, float pz)
{
  const float fx = (px - cv.lo[0]) * cv.inv[0], fy = (py - cv.lo[1]) * cv.inv[1], fz = (pz - cv.lo[2]) * cv.inv[2];
  const float g  = float(cv.g);
  const float R  = __ldg(cv.radius + cell);
  return fx >= 0.f && fx < g && fy >= 0.f && fy < g && fz >= 0.f && fz < g ? fminf(R, FLT_MAX) : FLT_MAX;
}

// Whether a packet too wide for one box takes the walk as a whole: where its points (lanes `in`) share what they
// reach.  The walk opens what any of them needs: about as many leaves as lie within the span of their
// nearest points, (span / diagonal)^2 of all.  Points outside the mesh's box count from where they would
// enter it (the ordering lines them up one behind the other), and the span shrinks with their distance.
__device__ __noinline__ bool sharesReach(const EbgMeshView& m, bool in, float px, float py, float pz, float diagonal,
                                         float leaves)
{
  const float inf = __int_as_float(0x7f800000);
  const int   n   = __popc(__ballot_sync(FULL, in));
  const float qx = fminf(fmaxf(px, m.root_lo[0]), m.root_hi[0]), qy = fminf(fmaxf(py, m.root_lo[1]), m.root_hi[1]),
              qz = fminf(fmaxf(pz, m.root_lo[2]), m.root_hi[2]);
  const float ex = warpMax(in ? qx : -inf) - warpMin(in ? qx : inf);
  const float ey = warpMax(in ? qy : -inf) - warpMin(in ? qy : inf);
  const float ez = warpMax(in ? qz : -inf) - warpMin(in ? qz : inf);
  const float dx = px - qx, dy = py - qy, dz = pz - qz;
  const float far = diagonal + 3.f * sqrtf(warpMin(in ? fmaf(dx, dx, fmaf(dy, dy, dz * dz)) : inf));
  return n > 4 && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) * leaves < WALK_LEAVES * float(n) * far * far;
}

// CELLS: the query passes an attached model, and its cells give the lanes' first bounds (the smaller of the
// model's radius and the distance to the anchor) and, by their anchors, the mesh points `a`.
template <bool CELLS>
__global__ void __launch_bounds__(32 * PACKET_WARPS, 8) kMeshPacket32(const __grid_constant__ MeshQueryArgs a, float delta,
                                                                     float split, float diagonal, float leaves)
{
  __shared__ PacketMem mem[PACKET_WARPS];
  const EbgMeshView&   m    = a.mesh;
  PacketMem&           pm   = mem[threadIdx.x >> 5];
  PointMem&            w    = pm.w;
  const int            lane = threadIdx.x & 31;
  const unsigned       lt   = (1u << lane) - 1u;
  const float          inf  = __int_as_float(0x7f800000);
  const uint64_t       numPackets = (uint64_t(a.n) + 31) / 32;
  const bool           sparse     = float(numPackets) < leaves;
  unsigned long long   pk = 0, pkEnd = 0;
  int                  besttri = -1, frontN = 0;
  int                  limit = 0; // leaves per point that a range may reach
  while (true) {
    if (pk == pkEnd) {
      // fewer at a time towards the end (a stale count only shifts that)
      unsigned long long take = 0;
      if (lane == 0) {
        const unsigned long long done = *reinterpret_cast<volatile unsigned long long*>(a.work);
        take = done < numPackets ? (numPackets - done) / (gridDim.x * (2ull * PACKET_WARPS)) : 0ull;
        take = take < 1ull ? 1ull : (take > (unsigned long long)a.chunk ? (unsigned long long)a.chunk : take);
        pk   = atomicAdd(a.work, take);
      }
      pk    = __shfl_sync(FULL, pk, 0);
      pkEnd = pk + __shfl_sync(FULL, take, 0);
      if (pk >= numPackets) {
        break;
      }
      // the group of packets: its box, a mesh point near it, and the frontier of the tree that it
      // reaches -- at most PACKET_FRONT entries -- where its packets start
      // (found from one of the points: the centre of a wide group may be equally far from everything)
      float lx = inf, ly = inf, lz = inf, ux = -inf, uy = -inf, uz = -inf, qx = 0.f, qy = 0.f, qz = 0.f;
      bool  got = false;
      for (unsigned long long i = pk; i < pkEnd && i < numPackets; i++) {
        const int64_t  pos = int64_t(i) * 32 + lane;
        const uint32_t id  = pos < a.n ? (a.order ? __ldg(a.order + pos) : uint32_t(pos)) : 0u;
        const float    px = __ldg(a.points + 3 * size_t(id)), py = __ldg(a.points + 3 * size_t(id) + 1),
                    pz = __ldg(a.points + 3 * size_t(id) + 2);
        const bool     ok  = pos < a.n && fabsf(px) + fabsf(py) + fabsf(pz) < 1e12f;
        const unsigned mk  = __ballot_sync(FULL, ok);
        if (!got && mk != 0u) {
          const int j = (mk >> 16) & 1u ? 16 : __ffs(int(mk)) - 1;
          qx          = __shfl_sync(FULL, px, j);
          qy          = __shfl_sync(FULL, py, j);
          qz          = __shfl_sync(FULL, pz, j);
          got         = true;
        }
        if (ok) {
          lx = fminf(lx, px), ly = fminf(ly, py), lz = fminf(lz, pz);
          ux = fmaxf(ux, px), uy = fmaxf(uy, py), uz = fmaxf(uz, pz);
        }
      }
      lx = warpMin(lx), ly = warpMin(ly), lz = warpMin(lz), ux = warpMax(ux), uy = warpMax(uy), uz = warpMax(uz);
      Reach r;
      r.cx = 0.5f * lx + 0.5f * ux, r.cy = 0.5f * ly + 0.5f * uy, r.cz = 0.5f * lz + 0.5f * uz;
      r.hx = fmaxf(ux - r.cx, r.cx - lx), r.hy = fmaxf(uy - r.cy, r.cy - ly), r.hz = fmaxf(uz - r.cz, r.cz - lz);
      besttri = -1;
      frontN  = 1;
      __syncwarp();
      if (lane == 0) {
        pm.last          = make_float4(qx, qy, qz, fmaxf(split, 0.f)); // (the first packet's anchor is found below)
        pm.front[0]      = m.root_ref;
        pm.frontCount[0] = m.root_count;
      }
      __syncwarp();
      limit = numPackets - pk > gridDim.x * (8ull * PACKET_WARPS) ? 32 : 12;
      if (got) {
        int err = 0;
        if (CELLS) {
          besttri = cellAnchor(a.cells, cellOf(a.cells, qx, qy, qz));
        }
        if (besttri < 0) {
          err = nearTriangle(m, qx, qy, qz, delta, w, besttri);
        }
        if (err && lane == 0) {
          atomicOr(a.status, err);
        }
        if (besttri >= 0 && pkEnd - pk > 1 && !(m.root_ref & EBG_LEAF_BIT)) {
          const float4* h  = reinterpret_cast<const float4*>(m.hot + besttri);
          const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
          float         s, t, ax, ay, az;
          int           reg;
          triDist2<false>(h0, h1, h2, qx, qy, qz, s, t, reg);
          triPoint(h0, h1, h2, s, t, ax, ay, az);
          setCorners(pm.corner, r, ax, ay, az, delta);
          // level by level while the next level fits
          for (int level = 0; level < EBG_STACK_DEPTH; level++) {
            int  nn = 0; // the next level's entries, gathered in w
            bool any = false;
            for (int f = 0; f < frontN && nn <= PACKET_FRONT; f += 8) {
              const int      g = lane >> 2, i = f + g;
              const uint32_t ref = i < frontN ? pm.front[i] : EBG_LEAF_BIT;
              const bool     leaf = (ref & EBG_LEAF_BIT) != 0u;
              uint32_t       child = ref, cw = i < frontN ? pm.frontCount[i] : 0u;
              float          d2;
              bool           keep = i < frontN && leaf && (lane & 3) == 0;
              if (!leaf) {
                keep = childReach(m, pm.corner, r, ref, lane & 3, child, cw, d2);
              }
              any |= __any_sync(FULL, !leaf) != 0;
              const unsigned mk = __ballot_sync(FULL, keep);
              if (keep && nn + __popc(mk) <= PACKET_FRONT) {
                w.leafRef[nn + __popc(mk & lt)]   = child;
                w.leafCount[nn + __popc(mk & lt)] = cw;
              }
              nn += __popc(mk);
            }
            __syncwarp();
            if (nn > PACKET_FRONT || nn == 0 || !any) {
              break;
            }
            if (lane < nn) {
              pm.front[lane]      = w.leafRef[lane];
              pm.frontCount[lane] = w.leafCount[lane];
            }
            frontN = nn;
            __syncwarp();
          }
        }
      }
    }
    if (pk >= numPackets) {
      break;
    }
    const int64_t  pos   = int64_t(pk) * 32 + lane;
    const bool     valid = pos < a.n;
    const int64_t  src   = valid ? pos : a.n - 1;
    const uint32_t id    = a.order ? __ldg(a.order + src) : uint32_t(src);
    const float    px = __ldg(a.points + 3 * size_t(id)), py = __ldg(a.points + 3 * size_t(id) + 1),
                pz = __ldg(a.points + 3 * size_t(id) + 2);
    const bool finite = isfinite(px) && isfinite(py) && isfinite(pz);
    const bool live   = valid && finite;
    if (valid && !finite) {
      atomicOr(a.status, ST_INPUT);
    }
    float best  = -1.f; // a lane without a live point needs nothing
    int   prev  = besttri, err = 0;
    bool  later = false; // the lane's point is put aside,
    bool  walk  = false; // as part of a packet for the walk
    besttri     = -1;
    // ranges [b, e) of lanes, each compact enough for one box
    int  b = 0, e = 32;
    while (b < 32 && err == 0) {
      const bool  in  = live && lane >= b && lane < e;
      const float mnx = warpMin(in ? px : inf), mny = warpMin(in ? py : inf), mnz = warpMin(in ? pz : inf);
      const float mxx = warpMax(in ? px : -inf), mxy = warpMax(in ? py : -inf), mxz = warpMax(in ? pz : -inf);
      Reach       r;
      r.cx = 0.5f * mnx + 0.5f * mxx, r.cy = 0.5f * mny + 0.5f * mxy, r.cz = 0.5f * mnz + 0.5f * mxz;
      r.hx = fmaxf(mxx - r.cx, r.cx - mnx), r.hy = fmaxf(mxy - r.cy, r.cy - mny), r.hz = fmaxf(mxz - r.cz, r.cz - mnz);
      const float hm  = fmaxf(r.hx, fmaxf(r.hy, r.hz));
      bool        box = hm <= split && !__any_sync(FULL, in && !(fabsf(px) + fabsf(py) + fabsf(pz) < 1e12f));
      if (!box && e - b == 32 && sharesReach(m, in, px, py, pz, diagonal, leaves)) {
        walk  = true;
        later = in;
        break;
      }
      if (!box && e - b > 4 && hm <= 16.f * split) {
        // divide at the widest step from one point to the next
        const float ux = __shfl_up_sync(FULL, px, 1), uy = __shfl_up_sync(FULL, py, 1), uz = __shfl_up_sync(FULL, pz, 1);
        const float dx = px - ux, dy = py - uy, dz = pz - uz;
        const float step = lane > b && lane < e ? fmaf(dx, dx, fmaf(dy, dy, dz * dz)) : -1.f;
        const float most = warpMax(step);
        e                = most >= 0.f ? __ffs(int(__ballot_sync(FULL, step == most))) - 1 : b + 1;
        continue;
      }
      box = box && e - b > 2;
      if (box) {
        // the mesh point `a` nearest to c among the winners of the packet before and of the ranges
        // before; the lane's own one is its first bound
        int            cand = besttri >= 0 ? besttri : prev;
        const int64_t  cell = CELLS ? cellOf(a.cells, px, py, pz) : 0;
        const int      own  = CELLS ? cellAnchor(a.cells, cell) : -1;
        cand                = CELLS && own >= 0 ? own : cand;
        const float4   last = pm.last;
        if (!__any_sync(FULL, own >= 0) && fmaxf(fabsf(r.cx - last.x), fmaxf(fabsf(r.cy - last.y), fabsf(r.cz - last.z))) > 4.f * (hm + last.w)) {
          // a step of the ordering to somewhere else: those winners are far from nearest here
          err |= nearTriangle(m, __shfl_sync(FULL, px, b), __shfl_sync(FULL, py, b), __shfl_sync(FULL, pz, b), delta, w, cand);
        }
        const unsigned have = __ballot_sync(FULL, cand >= 0);
        const int      alt  = __shfl_sync(FULL, cand, have ? __ffs(int(have)) - 1 : 0);
        cand                = cand >= 0 ? cand : alt;
        float ax = inf, ay = inf, az = inf;
        if (in) {
          best = FLT_MAX;
        }
        if (cand >= 0) {
          const float4* h  = reinterpret_cast<const float4*>(m.hot + cand);
          const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
          float         s, t;
          int           reg;
          const float   dd = triDist2<false>(h0, h1, h2, px, py, pz, s, t, reg);
          if (in && dd <= FLT_MAX) {
            best    = dd;
            besttri = cand;
          }
          triPoint(h0, h1, h2, s, t, ax, ay, az);
          const float ex = r.cx - ax, ey = r.cy - ay, ez = r.cz - az, dc = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
          const int from = (__ffs(int(__ballot_sync(FULL, dc == warpMin(dc)))) - 1) & 31;
          ax             = __shfl_sync(FULL, ax, from);
          ay             = __shfl_sync(FULL, ay, from);
          az             = __shfl_sync(FULL, az, from);
        }
        setCorners(pm.corner, r, ax, ay, az, delta);
        if (CELLS) {
          // The model's radius, where it is the smaller bound: of a lane (a lane that then finds nothing is
          // put aside), and without anchors of the packet.
          const float R = cellRadius(a.cells, cell, px, py, pz), R2 = __fmul_rd(__fmul_rd(R, R), 0.99998f);
          if (in && R2 < best) {
            best    = R2;
            besttri = -1;
          }
          if (a.cells.anchor == nullptr) {
            const float  most = warpMax(in ? R : 0.f) * 1.00001f + delta;
            const float4 A0 = pm.corner[0], A1 = pm.corner[1];
            const bool   nearer = most < fmaxf(fmaxf(fmaxf(A0.x, A0.y), fmaxf(A0.z, A0.w)), fmaxf(fmaxf(A1.x, A1.y), fmaxf(A1.z, A1.w)));
            __syncwarp();
            if (nearer && lane < 2) {
              pm.corner[lane] = make_float4(most, most, most, most);
            }
            __syncwarp();
          }
        }
        pm.key[lane] = (unsigned long long)__float_as_uint(best) << 32 | uint32_t(besttri);
        if (lane == 0) {
          pm.last = make_float4(r.cx, r.cy, r.cz, hm);
        }
        int sp = 0, nl = 0, np = 0, listed = 0;
        {
          // the group's frontier, one entry per lane
          uint32_t child = EBG_LEAF_BIT, cw = 0u;
          float    d2    = 0.f;
          bool     need  = lane < frontN;
          if (need) {
            child = pm.front[lane];
            cw    = pm.frontCount[lane];
          }
          const bool leaf = (child & EBG_LEAF_BIT) != 0u;
          if (need && (leaf || (cw & EBG_NODE_HAS_OBB))) {
            need = cornersReachObb(
              pm.corner[0], pm.corner[1], r.hx, r.hy, r.hz,
              reinterpret_cast<const float4*>(leaf ? m.obb + (cw >> EBG_COUNT_BITS) : m.node_obb + child), r.cx, r.cy, r.cz, d2);
          }
          const unsigned ml = __ballot_sync(FULL, need && leaf), mn = __ballot_sync(FULL, need && !leaf);
          if (need && leaf) {
            const int p    = __popc(ml & lt);
            w.leafRef[p]   = child;
            w.leafCount[p] = cw;
            w.leafKey[p]   = d2;
          }
          if (need && !leaf) {
            w.ref[__popc(mn & lt)] = child;
          }
          nl = __popc(ml);
          sp = __popc(mn);
          __syncwarp();
        }
        uint32_t iters = 0;
#pragma unroll 1
        while (sp > 0 || nl > 0) {
          if (++iters > MAX_ITERS) {
            err |= ST_ITERS;
            break;
          }
          if (nl >= 32 || sp == 0) {
            if (listed == 0) {
              // the two leaves nearest to c first: they bring the lanes' bounds near their final values
              const int reps = sp == 0 && nl <= 3 ? nl : 2; // all of a short list
              for (int rep = 0; rep < reps && nl > 0; rep++) {
                const float k0 = lane < nl ? w.leafKey[lane] : inf, k1 = lane + 32 < nl ? w.leafKey[lane + 32] : inf;
                const float kk = fminf(k0, k1);
                const int   from = (__ffs(int(__ballot_sync(FULL, kk == warpMin(kk)))) - 1) & 31;
                const int   at   = __shfl_sync(FULL, k0 <= k1 ? lane : lane + 32, from);
                const uint32_t t0 = w.leafRef[at] & ~EBG_LEAF_BIT, cw = w.leafCount[at];
                const float4*  ob = reinterpret_cast<const float4*>(m.obb + (cw >> EBG_COUNT_BITS));
                const bool     nd = obbDist2(__ldg(ob), __ldg(ob + 1), __ldg(ob + 2), __ldg(ob + 3), px, py, pz) <= best;
                const uint32_t te = t0 + (__any_sync(FULL, in && nd) ? cw & EBG_COUNT_MASK : 0u);
#pragma unroll 1
                for (uint32_t tt = t0; tt < te; tt++) {
                  const float4* h  = reinterpret_cast<const float4*>(m.hot + tt);
                  const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
                  float         s, t;
                  int           reg;
                  const float   dd = triDist2<false>(h0, h1, h2, px, py, pz, s, t, reg);
                  if (in && (dd < best || (dd == best && int(tt) < besttri))) {
                    best    = dd;
                    besttri = int(tt);
                  }
                }
                nl--;
                __syncwarp();
                if (lane == 0) {
                  w.leafRef[at]   = w.leafRef[nl];
                  w.leafCount[at] = w.leafCount[nl];
                  w.leafKey[at]   = w.leafKey[nl];
                }
                __syncwarp();
                listed++;
              }
              pm.key[lane] = (unsigned long long)__float_as_uint(best) << 32 | uint32_t(besttri);
              if (nl == 0) {
                __syncwarp();
                continue;
              }
            }
            // 32 leaves (or the last ones): a lane per leaf finds the lanes that need it
            __syncwarp();
            pm.query[lane] = make_float4(px, py, pz, in ? __uint_as_float(uint32_t(pm.key[lane] >> 32)) : -1.f);
            __syncwarp();
            const int take = nl < 32 ? nl : 32;
            uint32_t  ref = 0, cw = 0;
            unsigned  mask = 0u;
            if (lane < take) {
              ref = w.leafRef[nl - 1 - lane] & ~EBG_LEAF_BIT;
              cw  = w.leafCount[nl - 1 - lane];
              mask = lanesReach(reinterpret_cast<const float4*>(m.obb + (cw >> EBG_COUNT_BITS)), pm.query, b, e);
            }
            nl -= take;
            listed += take;
            // their pairs join the waiting ones, as many leaves at a time as there is room for, and
            // go 32 at a time
            const uint32_t cnt5 = (cw & EBG_COUNT_MASK) << 5;
            while (__any_sync(FULL, mask != 0u)) {
              const int mine = __popc(mask);
              int       at   = mine;
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, at, o);
                at += lane >= o ? v : 0;
              }
              const bool fits = np + at <= PACKET_PAIRS;
              const int  end  = np + int(__reduce_max_sync(FULL, fits ? uint32_t(at) : 0u));
              if (fits) {
                at += np - mine;
                while (mask != 0u) {
                  pm.pairTri[at]    = ref;
                  pm.pairLane[at++] = uint16_t(cnt5 | uint32_t(__ffs(int(mask)) - 1));
                  mask &= mask - 1u;
                }
              }
              np = end;
              __syncwarp();
              while (np >= 32) {
                np -= 32;
                testPairs(m, pm, np, 32);
              }
              __syncwarp();
            }
            if (listed > limit * (e - b)) {
              box   = false;
              limit = sparse ? limit : (limit > 12 ? 16 : 8);
              break;
            }
            continue;
          }
          const int take = sp <= POINT_WIDE ? (sp < 8 ? sp : 8) : 1;
          const int  g = lane >> 2;
          uint32_t   child = 0, cw = 0;
          float      d2;
          const bool need = g < take && childReach(m, pm.corner, r, w.ref[g < take ? sp - 1 - g : 0], lane & 3, child, cw, d2);
          const bool leaf = (child & EBG_LEAF_BIT) != 0u;
          sp -= take;
          const unsigned ml = __ballot_sync(FULL, need && leaf), mn = __ballot_sync(FULL, need && !leaf);
          __syncwarp(); // the taken entries are read before they are overwritten
          if (need && leaf) {
            const int p    = nl + __popc(ml & lt);
            w.leafRef[p]   = child;
            w.leafCount[p] = cw;
            w.leafKey[p]   = d2;
          }
          if (need && !leaf) {
            w.ref[sp + __popc(mn & lt)] = child;
          }
          nl += __popc(ml);
          sp += __popc(mn);
          __syncwarp();
          if (sp > POINT_NODES - 4) { // never for trees the builder accepts
            err |= ST_STACK;
            break;
          }
        }
        if (np > 0) {
          testPairs(m, pm, 0, np);
        }
        __syncwarp();
        const unsigned long long kb = pm.key[lane];
        if (in) {
          best    = __uint_as_float(uint32_t(kb >> 32));
          besttri = int(uint32_t(kb));
        }
        later = later || (CELLS && box && in && besttri < 0);
      }
      if (!box) {
        // too wide, far away, very few points or too many leaves in reach
        later = later || in;
      }
      b = e;
      e = 32;
    }

    const unsigned todo = __ballot_sync(FULL, later);
    if (todo != 0u) {
      // packets from the list's end, two words each (for at least five points, so that the two never meet)
      uint32_t at = 0;
      if (lane == 0) {
        at = walk ? a.n - 2 * (atomicAdd(a.later_count + 1, 1u) + 1u) : atomicAdd(a.band_count + 1, uint32_t(__popc(todo)));
      }
      at = __shfl_sync(FULL, at, 0) + (walk ? uint32_t(lane) : uint32_t(__popc(todo & lt)));
      if (walk ? lane < 2 : later) {
        a.point_list[at] = walk ? (lane == 0 ? uint32_t(pk) : todo) : uint32_t(pos);
      }
    }
    if (err && lane == 0) {
      atomicOr(a.status, err);
    }
    if (valid && !later) {
      store(a, m, besttri, px, py, pz, id, pos);
    }
    if (besttri < 0) {
      besttri = prev; // still a mesh triangle nearby
    }
    __syncwarp();
    pk++;
  }
}

} // namespace

namespace {
__global__ void kNodeChildren(const EbgNode4* __restrict__ nodes, int64_t slots, EbgChild* __restrict__ out)
{
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < slots; i += int64_t(gridDim.x) * blockDim.x) {
    const EbgNode4& n = nodes[i >> 2];
    const int       k = int(i & 3);
    out[i]            = EbgChild{n.lox[k], n.loy[k], n.loz[k], n.child[k], n.hix[k], n.hiy[k], n.hiz[k], n.count[k]};
  }
}

// sums[0], sums[1]: the leaf boxes' diagonals and their squares, in units of the mesh's diagonal as 32.32
// fixed-point numbers (whose sum does not depend on the order).
__global__ void kLeafSizes(const EbgChild* __restrict__ children, int64_t slots, float invDiagonal,
                           unsigned long long* __restrict__ sums)
{
  unsigned long long s1 = 0, s2 = 0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < slots; i += int64_t(gridDim.x) * blockDim.x) {
    const float4 lo = __ldg(reinterpret_cast<const float4*>(children + i)), hi = __ldg(reinterpret_cast<const float4*>(children + i) + 1);
    if (__float_as_uint(lo.w) & EBG_LEAF_BIT) {
      const float x = (hi.x - lo.x) * invDiagonal, y = (hi.y - lo.y) * invDiagonal, z = (hi.z - lo.z) * invDiagonal;
      const float l2 = fmaf(x, x, fmaf(y, y, z * z));
      s1 += (unsigned long long)(sqrtf(l2) * 4294967296.f);
      s2 += (unsigned long long)(l2 * 4294967296.f);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(FULL, s1, o);
    s2 += __shfl_xor_sync(FULL, s2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(sums, s1);
    atomicAdd(sums + 1, s2);
  }
}
} // namespace

void launchLeafSizes(const EbgChild* children, int64_t numNodes, double diagonal, unsigned long long* sums, cudaStream_t s)
{
  cudaMemsetAsync(sums, 0, 2 * sizeof(unsigned long long), s);
  const int64_t blocks = (4 * numNodes + 255) / 256;
  if (blocks > 0) {
    kLeafSizes<<<unsigned(blocks < 1024 ? blocks : 1024), 256, 0, s>>>(children, 4 * numNodes,
                                                                        float(1.0 / std::max(diagonal, 1e-300)), sums);
  }
}

void launchNodeChildren(const EbgNode4* nodes, int64_t numNodes, EbgChild* children, cudaStream_t s)
{
  const int64_t blocks = (4 * numNodes + 255) / 256;
  if (blocks > 0) {
    kNodeChildren<<<unsigned(blocks < 4096 ? blocks : 4096), 256, 0, s>>>(nodes, 4 * numNodes, children);
  }
}

cudaError_t launchMeshPacket32(const MeshQueryArgs& a, float delta, float split, float diagonal, int64_t numLeaves, int numSms,
                               cudaStream_t s)
{
  const int64_t packets = (a.n + 31) / 32;
  const int64_t need    = (packets + PACKET_WARPS - 1) / PACKET_WARPS;
  const int64_t most    = int64_t(numSms) * 8;
  const int64_t grid    = need < most ? need : most;
  if (a.cells.count != nullptr) {
    kMeshPacket32<true><<<unsigned(grid), 32 * PACKET_WARPS, 0, s>>>(a, delta, split, diagonal, float(numLeaves));
  }
  else {
    kMeshPacket32<false><<<unsigned(grid), 32 * PACKET_WARPS, 0, s>>>(a, delta, split, diagonal, float(numLeaves));
  }
  kMeshAside<<<unsigned(grid), 32 * PACKET_WARPS, 0, s>>>(a, delta);
  return cudaGetLastError();
}

} // namespace ebg
