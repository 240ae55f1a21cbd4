// Mesh signed distance of few points (sm_100a): one warp per query (mesh_point.cuh).  Compiled with
// -fmad=false like the other FP64 passes (band64.cuh).
//
// One launch does what the packet path needs an ordering, a traversal, a compaction and a band pass
// for, and takes no workspace.
#include <cfloat>

#include <math_constants.h>

#include "band64.cuh"
#include "mesh_kernels.h"
#include "mesh_point.cuh"

namespace ebg {

namespace {

constexpr int POINT_WARPS = 4;

// F64: FP64 points and results with evaluator EVAL (0 the Triangle test, 1 the DCEL face).  Else
// FP32 points and distances (no triangles): the FP32 search, and the FP64 one where |d| is within the band.
// Bound by the latency of its dependent loads (two per tree level and two per leaf batch), so the
// FP32 form keeps 32 queries in flight per SM at the cost of a few spills in its rare FP64 part.
// B200, 20,480 triangles, uniform points, packet path before -> now: 1 point 166 -> 15 us, 32 points
// 1,281 -> 15 us, 1,000 points 616 -> 27 us, 65,536 points 1.41 -> 0.21 ms; in FP64 1,000 points
// 1,695 -> 19 us, 65,536 points 3.62 -> 0.27 ms.
template <bool F64, int EVAL>
__global__ void __launch_bounds__(32 * POINT_WARPS, F64 ? 5 : 8) kMeshPoint(const MeshQueryArgs a, float delta, int band64)
{
  __shared__ PointMem mem[POINT_WARPS];
  const EbgMeshView&  m    = a.mesh;
  PointMem&           w    = mem[threadIdx.x >> 5];
  const int           lane = threadIdx.x & 31;
  const int64_t       nW   = int64_t(gridDim.x) * POINT_WARPS;
  for (int64_t id = int64_t(blockIdx.x) * POINT_WARPS + (threadIdx.x >> 5); id < a.n; id += nW) {
    D3    P;
    float px, py, pz;
    if (F64) {
      P  = {a.points64[3 * id], a.points64[3 * id + 1], a.points64[3 * id + 2]};
      px = float(P.x), py = float(P.y), pz = float(P.z);
    }
    else {
      px = __ldg(a.points + 3 * id), py = __ldg(a.points + 3 * id + 1), pz = __ldg(a.points + 3 * id + 2);
      P  = {double(px), double(py), double(pz)};
    }
    if (!(isfinite(px) && isfinite(py) && isfinite(pz))) {
      if (lane == 0) {
        atomicOr(a.status, ST_INPUT);
        if (F64) {
          a.out_d64[id] = double(FLT_MAX);
        }
        else {
          a.out_d[id] = FLT_MAX;
        }
        if (F64 && a.out_tri) {
          a.out_tri[id] = -1;
        }
      }
      continue;
    }
    const double ex = P.x - double(px), ey = P.y - double(py), ez = P.z - double(pz);
    const float  shift = F64 ? float(sqrt(ex * ex + ey * ey + ez * ez)) * 1.0001f : 0.f;
    double       best = DBL_MAX;
    int          bt   = -1, err;
    if (F64) {
      err = pointSearch64<EVAL, true, true>(m, P, px, py, pz, shift, delta, FLT_MAX, best, bt, w);
      if (lane == 0) {
        a.out_d64[id] = bt >= 0 ? best : double(FLT_MAX);
        if (a.out_tri) {
          a.out_tri[id] = bt >= 0 ? __ldg(m.tri_id + bt) : -1;
        }
      }
    }
    else {
      float bd2  = FLT_MAX;
      err        = pointNearest(m, px, py, pz, delta, w, bd2, bt);
      float dist = bt >= 0 ? signedFromWinner(m, uint32_t(bt), px, py, pz) : FLT_MAX;
      if (band64 && bt >= 0 && fabsf(dist) <= a.band) {
        const float r = (fabsf(dist) * 1.00001f + delta) * 1.000001f;
        int         b64;
        err |= pointSearch64<0, false, true>(m, P, px, py, pz, 0.f, delta, r * r, best, b64, w);
        dist = b64 >= 0 ? float(best) : dist;
      }
      if (lane == 0) {
        a.out_d[id] = dist;
      }
    }
    if (err && lane == 0) {
      atomicOr(a.status, err);
    }
  }
}

} // namespace

cudaError_t launchMeshPoint(const MeshQueryArgs& a, float delta, bool band64, int numSms, cudaStream_t s)
{
  const int64_t need = (a.n + POINT_WARPS - 1) / POINT_WARPS;
  const int64_t most = int64_t(numSms) * 32;
  const unsigned grid = unsigned(need < most ? need : most);
  if (a.out_d64 == nullptr) {
    kMeshPoint<false, 0><<<grid, 32 * POINT_WARPS, 0, s>>>(a, delta, band64 ? 1 : 0);
  }
  else if (a.eval == 1) {
    kMeshPoint<true, 1><<<grid, 32 * POINT_WARPS, 0, s>>>(a, delta, 1);
  }
  else {
    kMeshPoint<true, 0><<<grid, 32 * POINT_WARPS, 0, s>>>(a, delta, 1);
  }
  return cudaGetLastError();
}

} // namespace ebg
