// FP64 near-surface re-evaluation (sm_100a).  Compiled with -fmad=false: the point-triangle
// arithmetic below keeps the reference's separate multiplies and adds in the reference's order.
//
// Queries whose FP32 distance fell inside the band |d| <= band (default 1e-4 x the mesh's bounding
// box diagonal, where the sign is ill-conditioned) are re-evaluated here with the reference's own
// FP64 triangle test -- a lane-by-lane restatement of the AVX W=4 double path of
// TriangleSoAT::signedDistance (TriangleSoAImplem.hpp:1029-1180) -- over every triangle whose FP32
// (outward-rounded) box lies within |d32| + delta of the point, keeping the value of smallest
// magnitude with strict < (MeshDistanceFunctionsImplem.hpp:492-502).  delta covers the FP32
// distance error, so the FP64 winner is never pruned; leaves and nodes are also pruned by their
// oriented boxes, which bound the exact distance to every triangle inside from below.  Of needle-like
// triangles an FP32 distance can be too small by more than delta: a winner outside the radius, or none,
// shows it, and the query is searched again with the winner's own distance (none: without a bound).
// An FP64 call evaluates all its queries here, with FP32 distances that only bound the search.
//
// Bound by the L1's wavefronts and the FP64 pipe together: an FP64 test is about 200 instructions at
// half rate, so it is spent only on triangles whose FP32 lower bound (triLower) reaches the radius --
// one to a few per query, 32 queries' worth at a time -- where the walk that shared one stack per
// packet evaluated every triangle of every leaf that any lane needed.  B200, that walk -> here: 1.4 M
// band points of 4 M within 1e-3 of 1.3 M triangles 2.40 -> 0.83 ms, of 20,480 triangles 0.57 -> 0.35 ms;
// the band of 1 M uniform points 0.44 -> 0.02 ms; FP64 end to end, 1 M uniform points on 20,480
// triangles, 3.62 -> 0.85 ms; DCEL faces, 250,007 points on 81,920 triangles, 5.14 -> 0.72 ms.
#include <cfloat>

#include <math_constants.h>

#include "band64.cuh"
#include "ebg_device.cuh"
#include "mesh_kernels.h"
#include "mesh_packet.cuh"
#include "mesh_point.cuh"
#include "mesh_traverse.cuh"

namespace ebg {

namespace {

constexpr int BAND_WARPS = 4;
constexpr int BAND_CAND  = 16; // triangles waiting for their FP64 test, per group

struct BandMem
{
  GroupMem g;
  uint32_t cand[BAND_CAND];
};

// One FP64 evaluation of the triangle at leaf position tt (EVAL 0: the reference's Triangle/TriangleSoA
// test, TriMeshSDF; 1: the DCEL face, MeshSDF); DBL_MAX for a degenerate one, which never wins.
template <int EVAL>
__device__ __forceinline__ double triEval64(const EbgMeshView& m, uint32_t tt, D3 P)
{
  const double d = EVAL == 0 ? triSd64(m.tri64 + 30 * size_t(tt), P)
                             : dcelFaceSd(m.tri64 + 30 * size_t(tt), m.dcel_n + 3 * size_t(tt), P);
  return fabs(d) < DBL_MAX ? d : DBL_MAX;
}

// A band query's search radius at its FP32 point, `shift` from its FP64 point P.  Boxes are tested at
// the FP32 point.  The mesh is within |d32| + delta of it (delta covers the FP32 distance error near
// the surface, the relative term far from it), so the FP64 winner is within |d32| + delta + shift of
// P and within |d32| + delta + 2 shift of the FP32 point.
__device__ __forceinline__ float bandRadius(D3 P, float px, float py, float pz, float d32, float delta, float& shift)
{
  const double ex = P.x - double(px), ey = P.y - double(py), ez = P.z - double(pz);
  shift           = float(sqrt(ex * ex + ey * ey + ez * ez)) * 1.0001f;
  return (fabsf(d32) * 1.00001f + delta + 2.f * shift) * 1.000001f;
}

// A query's FP64 point: the caller's own when it passed FP64, else its FP32 point.
__device__ __forceinline__ D3 bandPoint(const MeshQueryArgs& a, uint32_t id, float px, float py, float pz)
{
  return a.points64 ? D3{a.points64[3 * size_t(id)], a.points64[3 * size_t(id) + 1], a.points64[3 * size_t(id) + 2]}
                    : D3{double(px), double(py), double(pz)};
}

// The results of a query whose FP64 winner is bt (-1: none within the radius).
__device__ __forceinline__ void bandStore(const MeshQueryArgs& a, const EbgMeshView& m, uint32_t id, float d32, double best,
                                          int bt)
{
  if (a.out_d64 != nullptr) {
    a.out_d64[id] = bt >= 0 ? best : double(d32);
  }
  if (bt >= 0) {
    a.out_d[id] = float(best);
    if (a.out_tri) {
      a.out_tri[id] = m.tri_id[bt];
    }
  }
}

// Whether a triangle may hold the FP64 winner of a query with squared bound `bound`: its lower bound
// in FP32 from the closest point that triDist2 finds.
__device__ __forceinline__ bool bandCandidate(const EbgMeshView& m, uint32_t tt, float px, float py, float pz, float bound,
                                              float delta)
{
  const float4* h  = reinterpret_cast<const float4*>(m.hot + tt);
  const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
  float         s, t;
  int           r;
  const float   dd = triDist2<false>(h0, h1, h2, px, py, pz, s, t, r);
  return mayReach(triLower(h0, h1, h2, px, py, pz, s, t, dd), dd, sqrtf(bound) * 1.00001f + delta);
}

// Eight lanes per band query that kMeshBand64 put aside (groupSearch), from the root with the query's own bound.
template <int EVAL>
__global__ void __launch_bounds__(32 * BAND_WARPS, 6) kMeshBandGroups(const __grid_constant__ MeshQueryArgs a, float delta)
{
  __shared__ BandMem mem[4 * BAND_WARPS];
  const EbgMeshView& m     = a.mesh;
  const uint32_t     count = *a.later_count;
  const uint32_t     nG    = gridDim.x * (4 * BAND_WARPS);
  const int          sub   = threadIdx.x & 7;
  const unsigned     base  = threadIdx.x & 24;
  BandMem&           w     = mem[threadIdx.x >> 3];

  for (uint32_t j0 = blockIdx.x * (4 * BAND_WARPS) + (threadIdx.x >> 5) * 4; j0 < count; j0 += nG) {
    const uint32_t j   = j0 + (base >> 3);
    const bool     on  = j < count;
    const uint32_t pos = a.band_list[a.later[on ? j : j0]];
    const uint32_t id  = a.order ? a.order[pos] : pos;
    const float    px = a.points[3 * size_t(id)], py = a.points[3 * size_t(id) + 1], pz = a.points[3 * size_t(id) + 2];
    const D3       P   = bandPoint(a, id, px, py, pz);
    const float    d32 = a.out_d[id]; // the FP32 pass's distance
    float        shift;
    const float  r     = bandRadius(P, px, py, pz, d32, delta, shift);
    float        bound = r * r;
    double       best  = DBL_MAX;
    int          bt    = -1, nc = 0;

    // up to eight waiting triangles, a lane each
    auto evaluate = [&]() {
      const int  n  = nc < 8 ? nc : 8;
      const bool ev = sub < n;
      double     d  = DBL_MAX;
      int        tt = 0x7fffffff;
      if (ev) {
        tt = int(w.cand[nc - 1 - sub]);
        d  = triEval64<EVAL>(m, uint32_t(tt), P);
      }
      // the least |d| of the group, ties to the lower leaf position
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const double od = __shfl_xor_sync(FULL, d, o);
        const int    ot = __shfl_xor_sync(FULL, tt, o);
        if (fabs(od) < fabs(d) || (fabs(od) == fabs(d) && ot < tt)) {
          d  = od;
          tt = ot;
        }
      }
      nc -= n;
      if (n > 0 && fabs(d) < DBL_MAX && (fabs(d) < fabs(best) || (fabs(d) == fabs(best) && tt < bt))) {
        best           = d;
        bt             = tt;
        const float rb = winnerRadius(d, shift);
        bound          = fminf(bound, rb * rb);
      }
      __syncwarp(); // read before more are appended
    };
    int  err  = 0;
    bool todo = on;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
      err |= groupSearch<false>(m, todo, px, py, pz, bound, 0.f, w.g, [&](bool, uint32_t t0, int cnt, int most) {
        for (int t = sub; t - sub < most; t += 8) {
          const bool     cand = t < cnt && bandCandidate(m, t0 + uint32_t(t), px, py, pz, bound, delta);
          const unsigned mk = (__ballot_sync(FULL, cand) >> base) & 0xffu;
          if (cand) {
            w.cand[nc + __popc(mk & ((1u << sub) - 1u))] = t0 + uint32_t(t);
          }
          nc += __popc(mk);
          __syncwarp();
          if (__any_sync(FULL, nc >= BAND_CAND - 8)) {
            evaluate();
          }
        }
      });
      while (__any_sync(FULL, nc > 0)) {
        evaluate();
      }
      const float rb = winnerRadius(best, shift);
      todo           = todo && !(bt >= 0 && rb <= r);
      if (!__any_sync(FULL, todo)) {
        break;
      }
      if (todo) {
        bound = bt >= 0 ? rb * rb : FLT_MAX;
      }
    }
    if (on && sub == 0) {
      if (err) {
        atomicOr(a.status, err);
      }
      bandStore(a, m, id, d32, best, bt);
    }
    __syncwarp();
  }
}

constexpr int BAND_PAIRS = 256; // (query, leaf) pairs waiting for their triangle tests
constexpr int BAND_QUEUE = 64;  // (query, triangle) candidates waiting for their FP64 test

struct BandPacketMem
{
  float4   query[32];               // FP32 points and squared bounds
  double   px[32], py[32], pz[32];  // FP64 points
  double   res[32];
  float4   corner[2];
  uint32_t pairTri[BAND_PAIRS];
  uint32_t candTri[BAND_QUEUE];
  uint32_t node[POINT_NODES];
  uint32_t leafRef[POINT_LEAVES], leafCount[POINT_LEAVES];
  uint16_t pairLane[BAND_PAIRS]; // triangle count and lane
  uint8_t  candLane[BAND_QUEUE];
};

// Packets of 32 consecutive band queries (neighbours: the list is in position order): one search of the
// tree for the packet's box, as the FP32 packet search does it (mesh_packet.cu).  A query's radius is at
// most the largest of the packet's, and -- where the FP32 pass left its winning triangles (a.tri32) -- at
// most the distance to a point of one of them; the tighter of the two bounds goes to the corners.
// The (query, leaf) pairs left are tested a lane each in FP32, and only triangles whose FP32 lower
// bound is within the radius are evaluated in FP64, 32 candidates at a time.  A packet too wide or
// with too many leaves in reach leaves its queries to kMeshBandGroups, as a query does whose radius did not
// hold its winner.
template <int EVAL>
__global__ void __launch_bounds__(32 * BAND_WARPS, 6) kMeshBand64(const __grid_constant__ MeshQueryArgs a, float delta,
                                                                  float split)
{
  __shared__ BandPacketMem mem[BAND_WARPS];
  const EbgMeshView& m     = a.mesh;
  const uint32_t     count = *a.band_count;
  const int          lane  = threadIdx.x & 31;
  const unsigned     lt    = (1u << lane) - 1u;
  const float        inf   = __int_as_float(0x7f800000);
  BandPacketMem&     w     = mem[threadIdx.x >> 5];
  const uint32_t     numPk = (count + 31) / 32;
  for (uint32_t pk = blockIdx.x * BAND_WARPS + (threadIdx.x >> 5); pk < numPk; pk += gridDim.x * BAND_WARPS) {
    const uint32_t j   = pk * 32 + lane;
    const bool     on  = j < count;
    const uint32_t jj  = on ? j : count - 1;
    const uint32_t pos = a.band_list[jj];
    const uint32_t id  = a.order ? a.order[pos] : pos;
    const float    px = a.points[3 * size_t(id)], py = a.points[3 * size_t(id) + 1], pz = a.points[3 * size_t(id) + 2];
    const D3       P   = bandPoint(a, id, px, py, pz);
    const float    d32 = a.out_d[id]; // the FP32 pass's distance
    float          shift;
    const float    r = bandRadius(P, px, py, pz, d32, delta, shift);
    float          bound = r * r;
    double         best  = DBL_MAX;
    int            bt    = -1, err = 0;

    Reach       box;
    const float lx = warpMin(px), ly = warpMin(py), lz = warpMin(pz), ux = warpMax(px), uy = warpMax(py), uz = warpMax(pz);
    box.cx = 0.5f * lx + 0.5f * ux, box.cy = 0.5f * ly + 0.5f * uy, box.cz = 0.5f * lz + 0.5f * uz;
    box.hx = fmaxf(ux - box.cx, box.cx - lx), box.hy = fmaxf(uy - box.cy, box.cy - ly), box.hz = fmaxf(uz - box.cz, box.cz - lz);
    const float rm = warpMax(r);
    bool        ok = fmaxf(box.hx, fmaxf(box.hy, box.hz)) <= split && fabsf(box.cx) + fabsf(box.cy) + fabsf(box.cz) < 1e12f;
    if (ok) {
      // the corners' bounds: the largest radius, or the distances to a mesh point if those are smaller
      __syncwarp(); // the packet before has read its memory
      if (lane < 8) {
        reinterpret_cast<float*>(w.corner)[lane] = rm * 1.00001f + delta;
      }
      const int own = a.tri32 ? a.tri32[id] : -1;
      if (__all_sync(FULL, own >= 0)) {
        const float4* h  = reinterpret_cast<const float4*>(m.hot + own);
        const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
        float         s, t, ax, ay, az;
        int           reg;
        triDist2<false>(h0, h1, h2, px, py, pz, s, t, reg);
        triPoint(h0, h1, h2, s, t, ax, ay, az);
        const float ex = box.cx - ax, ey = box.cy - ay, ez = box.cz - az, dc = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
        const int   from = (__ffs(int(__ballot_sync(FULL, dc == warpMin(dc)))) - 1) & 31;
        ax               = __shfl_sync(FULL, ax, from);
        ay               = __shfl_sync(FULL, ay, from);
        az               = __shfl_sync(FULL, az, from);
        // the FP32 distance of any query is at most |p - a| (1 + 1e-5) + delta
        const float gx = fabsf(box.cx - ax) + box.hx, gy = fabsf(box.cy - ay) + box.hy, gz = fabsf(box.cz - az) + box.hz;
        const float far = sqrtf(fmaf(gx, gx, fmaf(gy, gy, gz * gz)));
        const float sm  = warpMax(shift);
        if (far < 1.5f * rm) {
          setCorners(w.corner, box, ax, ay, az, 0.f);
          if (lane < 8) {
            float* A = reinterpret_cast<float*>(w.corner) + lane;
            *A       = *A * 1.00004f + 4.f * delta + 2.1f * sm;
          }
        }
      }
      w.query[lane] = make_float4(px, py, pz, on ? bound : -1.f);
      w.px[lane]    = P.x;
      w.py[lane]    = P.y;
      w.pz[lane]    = P.z;
      int sp = 0, nl = 0, np = 0, nc = 0, listed = 0;
      if (lane == 0) {
        w.node[0]      = m.root_ref;
        w.leafRef[0]   = m.root_ref;
        w.leafCount[0] = m.root_count;
      }
      (m.root_ref & EBG_LEAF_BIT ? nl : sp) = 1;
      __syncwarp();

      // up to 32 waiting candidates, a lane each; every query takes its least (|d|, triangle)
      auto evaluate = [&]() {
        const int n = nc < 32 ? nc : 32;
        nc -= n;
        if (lane < n) {
          const int q = w.candLane[nc + lane];
          w.res[lane] = triEval64<EVAL>(m, w.candTri[nc + lane], D3{w.px[q], w.py[q], w.pz[q]});
        }
        __syncwarp();
        for (int i = 0; i < n; i++) {
          if (int(w.candLane[nc + i]) == lane) {
            const double d = w.res[i];
            const int    t = int(w.candTri[nc + i]);
            if (fabs(d) < DBL_MAX && (fabs(d) < fabs(best) || (fabs(d) == fabs(best) && t < bt))) {
              best           = d;
              bt             = t;
              const float rb = winnerRadius(d, shift);
              bound          = fminf(bound, rb * rb);
            }
          }
        }
        w.query[lane].w = on ? bound : -1.f;
        __syncwarp();
      };
      // up to 32 waiting pairs, a lane each: their candidates join the queue
      auto testPairs = [&](int n) {
        np -= n;
        const bool     act = lane < n;
        const uint32_t v   = act ? w.pairLane[np + lane] : 0u;
        const uint32_t t0  = act ? w.pairTri[np + lane] : 0u;
        const int      cnt = int(v >> 5), q = int(v & 31u);
        const int      most = int(__reduce_max_sync(FULL, uint32_t(cnt)));
        for (int t = 0; t < most; t++) {
          const float4   p    = w.query[q];
          const bool     cand = t < cnt && bandCandidate(m, t0 + uint32_t(t), p.x, p.y, p.z, p.w, delta);
          const unsigned mk   = __ballot_sync(FULL, cand);
          if (cand) {
            const int i   = nc + __popc(mk & lt);
            w.candTri[i]  = t0 + uint32_t(t);
            w.candLane[i] = uint8_t(q);
          }
          nc += __popc(mk);
          __syncwarp();
          if (nc >= 32) {
            evaluate();
          }
        }
      };
      uint32_t iters = 0;
#pragma unroll 1
      while (sp > 0 || nl > 0) {
        if (++iters > MAX_ITERS) {
          err |= ST_ITERS;
          break;
        }
        if (nl >= 32 || sp == 0) {
          const int take = nl < 32 ? nl : 32;
          uint32_t  ref = 0, cw = 0;
          unsigned  mask = 0u;
          if (lane < take) {
            ref  = w.leafRef[nl - 1 - lane] & ~EBG_LEAF_BIT;
            cw   = w.leafCount[nl - 1 - lane];
            mask = lanesReach(reinterpret_cast<const float4*>(m.obb + (cw >> EBG_COUNT_BITS)), w.query, 0, 32);
          }
          nl -= take;
          listed += take;
          const uint32_t cnt5 = (cw & EBG_COUNT_MASK) << 5;
          while (__any_sync(FULL, mask != 0u)) {
            // the pairs of as many leaves as there is room for
            const int mine = __popc(mask);
            int       at   = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int v = __shfl_up_sync(FULL, at, o);
              at += lane >= o ? v : 0;
            }
            const bool fits = np + at <= BAND_PAIRS;
            const int  end  = np + int(__reduce_max_sync(FULL, fits ? uint32_t(at) : 0u));
            if (fits) {
              at += np - mine;
              while (mask != 0u) {
                w.pairTri[at]    = ref;
                w.pairLane[at++] = uint16_t(cnt5 | uint32_t(__ffs(int(mask)) - 1));
                mask &= mask - 1u;
              }
            }
            np = end;
            __syncwarp();
            while (np >= 32) {
              testPairs(32);
            }
          }
          if (listed > 512 && (sp > 0 || nl > 0)) {
            ok = false;
            break;
          }
          continue;
        }
        const int  take = sp <= POINT_WIDE ? (sp < 8 ? sp : 8) : 1;
        const int  g    = lane >> 2;
        uint32_t   child = 0, cw = 0;
        float      d2;
        const bool need = g < take && childReach(m, w.corner, box, w.node[g < take ? sp - 1 - g : 0], lane & 3, child, cw, d2);
        const bool leaf = (child & EBG_LEAF_BIT) != 0u;
        sp -= take;
        const unsigned ml = __ballot_sync(FULL, need && leaf), mn = __ballot_sync(FULL, need && !leaf);
        __syncwarp(); // the taken entries are read before they are overwritten
        if (need && leaf) {
          const int p    = nl + __popc(ml & lt);
          w.leafRef[p]   = child;
          w.leafCount[p] = cw;
        }
        if (need && !leaf) {
          w.node[sp + __popc(mn & lt)] = child;
        }
        nl += __popc(ml);
        sp += __popc(mn);
        __syncwarp();
        if (sp > POINT_NODES - 4) { // never for trees the builder accepts
          err |= ST_STACK;
          break;
        }
      }
      if (ok) {
        if (np > 0) {
          testPairs(np);
        }
        if (nc > 0) {
          evaluate();
        }
      }
    }
    if (err && lane == 0) {
      atomicOr(a.status, err);
    }
    ok = ok && bt >= 0 && winnerRadius(best, shift) <= r;
    if (on && ok) {
      bandStore(a, m, id, d32, best, bt);
    }
    const unsigned mk = __ballot_sync(FULL, on && !ok);
    if (mk != 0u) {
      uint32_t at = 0;
      if (lane == 0) {
        at = atomicAdd(a.later_count, uint32_t(__popc(mk)));
      }
      at = __shfl_sync(FULL, at, 0);
      if (on && !ok) {
        a.later[at + __popc(mk & lt)] = j;
      }
    }
    __syncwarp();
  }
}

// FlatMeshSDF (MeshT::DirectSignedDistance2, DCEL_MeshImplem.hpp:574-595): every face, the first
// in soup order with the smallest unsigned distance^2 wins, and its signed distance is the value.
// One query per thread; the block walks the triangles (leaf order) through shared-memory tiles of
// their vertices and DCEL normals and keeps the lexicographic minimum of (d^2, soup index).
constexpr int FLAT_TILE = 64;

__global__ void __launch_bounds__(128) kMeshFlat64(const EbgMeshView m, int64_t numTris, const double* __restrict__ pts,
                                                   int64_t n, double* __restrict__ out, int32_t* __restrict__ outTri,
                                                   int* __restrict__ status)
{
  __shared__ double  sv[FLAT_TILE][12];
  __shared__ int32_t sid[FLAT_TILE];
  for (int64_t base = int64_t(blockIdx.x) * blockDim.x; base < n; base += int64_t(gridDim.x) * blockDim.x) {
    const int64_t q     = base + threadIdx.x;
    const bool    valid = q < n;
    const D3      P     = valid ? D3{pts[3 * q], pts[3 * q + 1], pts[3 * q + 2]} : D3{0.0, 0.0, 0.0};
    const bool    finite = isfinite(P.x) && isfinite(P.y) && isfinite(P.z);
    if (valid && !finite) {
      atomicOr(status, ST_INPUT);
    }
    double        best  = CUDART_INF;
    int32_t       bsoup = INT32_MAX;
    int64_t       bpos  = -1;
    for (int64_t t0 = 0; t0 < numTris; t0 += FLAT_TILE) {
      __syncthreads();
      for (int k = threadIdx.x; k < FLAT_TILE * 12; k += blockDim.x) {
        const int64_t tt = t0 + k / 12;
        const int     c  = k % 12;
        sv[k / 12][c]    = tt < numTris ? (c < 9 ? m.tri64[30 * tt + c] : m.dcel_n[3 * tt + (c - 9)]) : 0.0;
      }
      for (int k = threadIdx.x; k < FLAT_TILE; k += blockDim.x) {
        sid[k] = t0 + k < numTris ? m.tri_id[t0 + k] : INT32_MAX;
      }
      __syncthreads();
      const int cnt = int(numTris - t0 < FLAT_TILE ? numTris - t0 : FLAT_TILE);
      for (int k = 0; k < cnt; k++) {
        const double d2 = dcelFaceUd2(sv[k], sv[k] + 9, P);
        if (d2 < best || (d2 == best && sid[k] < bsoup)) {
          best  = d2;
          bsoup = sid[k];
          bpos  = t0 + k;
        }
      }
    }
    if (valid) {
      // a non-finite point (reported through the status word) gets NaN
      out[q] = (finite && bpos >= 0) ? dcelFaceSd(m.tri64 + 30 * bpos, m.dcel_n + 3 * bpos, P) : CUDART_NAN;
      if (outTri) {
        outTri[q] = (finite && bpos >= 0) ? bsoup : -1;
      }
    }
  }
}

} // namespace

cudaError_t launchMeshFlat64(const EbgMeshView& m, int64_t numTris, const double* pts, int64_t n, double* out,
                             int32_t* outTri, int* status, int numSms, cudaStream_t s)
{
  int64_t blocks = (n + 127) / 128;
  blocks         = blocks < int64_t(numSms) * 16 ? blocks : int64_t(numSms) * 16;
  kMeshFlat64<<<unsigned(blocks < 1 ? 1 : blocks), 128, 0, s>>>(m, numTris, pts, n, out, outTri, status);
  return cudaGetLastError();
}

namespace {
__global__ void kDoubleToFloat(const double* __restrict__ in, float* __restrict__ out, int64_t count)
{
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x) {
    out[i] = float(in[i]);
  }
}
} // namespace

void launchDoubleToFloat(const double* in, float* out, int64_t count, cudaStream_t s)
{
  int64_t blocks = (count + 255) / 256;
  blocks         = blocks < 4096 ? blocks : 4096;
  kDoubleToFloat<<<unsigned(blocks < 1 ? 1 : blocks), 256, 0, s>>>(in, out, count);
}

cudaError_t launchMeshBand64(const MeshQueryArgs& a, float delta, float split, int numSms, cudaStream_t s)
{
  const unsigned blocks = unsigned(numSms * 6);
  if (a.eval == 1) {
    kMeshBand64<1><<<blocks, 32 * BAND_WARPS, 0, s>>>(a, delta, split);
    kMeshBandGroups<1><<<blocks, 32 * BAND_WARPS, 0, s>>>(a, delta);
  }
  else {
    kMeshBand64<0><<<blocks, 32 * BAND_WARPS, 0, s>>>(a, delta, split);
    kMeshBandGroups<0><<<blocks, 32 * BAND_WARPS, 0, s>>>(a, delta);
  }
  return cudaGetLastError();
}

} // namespace ebg
