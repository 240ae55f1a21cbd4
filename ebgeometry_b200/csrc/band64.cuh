// FP64 evaluation of mesh triangles for the near-surface passes (sm_100a), shared by the mesh band
// kernels (mesh_band64.cu), the search of few points (mesh_point.cu) and the CSG union's band kernel
// (scene_band64.cu).  Include it only from
// translation units compiled with -fmad=false: the point-triangle arithmetic keeps the reference's
// separate multiplies and adds in the reference's order.
//
//  - triSd64: a lane-by-lane restatement of the AVX W=4 double path of TriangleSoAT::signedDistance
//    (TriangleSoAImplem.hpp:1029-1180, sign-bit convention of :1076-1082);
//  - dcelFaceSd / dcelFaceUd2: one triangle as a DCEL face, the algorithm of MeshSDF and FlatMeshSDF;
//  - pointSearch64: the FP64 search of a mesh for one point.
#ifndef EBG_BAND64_CUH
#define EBG_BAND64_CUH

#include <cfloat>

#include "ebg_device.cuh"
#include "mesh_point.cuh"
#include "mesh_traverse.cuh"

namespace ebg {

namespace {

struct D3
{
  double x, y, z;
};
__device__ __forceinline__ D3 ld3(const double* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ D3 sub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross(D3 a, D3 b)
{
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ D3 scl(double s, D3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double sgnb(double x) { return signbit(x) ? -1.0 : 1.0; }

// tri: v0 v1 v2 n vn0 vn1 vn2 en0 en1 en2 (30 doubles)
__device__ double triSd64(const double* __restrict__ tri, D3 P)
{
  const D3 v0 = ld3(tri), v1 = ld3(tri + 3), v2 = ld3(tri + 6), n = ld3(tri + 9);
  const D3 v21 = sub(v1, v0), v32 = sub(v2, v1), v13 = sub(v0, v2);
  const D3 p1 = sub(P, v0), p2 = sub(P, v1), p3 = sub(P, v2);
  const double s0 = sgnb(dot(cross(v21, n), p1));
  const double s1 = sgnb(dot(cross(v32, n), p2));
  const double s2 = sgnb(dot(cross(v13, n), p3));
  if (fabs((s0 + s1) + s2) >= 2.0) {
    return dot(n, p1);
  }
  const double t1 = dot(p1, v21) / dot(v21, v21);
  const double t2 = dot(p2, v32) / dot(v32, v32);
  const double t3 = dot(p3, v13) / dot(v13, v13);
  const D3     y1 = sub(p1, scl(t1, v21)), y2 = sub(p2, scl(t2, v32)), y3 = sub(p3, scl(t3, v13));

  double bd2 = dot(p1, p1);
  double bs  = sgnb(dot(ld3(tri + 12), p1));
  const double p2d2 = dot(p2, p2), p3d2 = dot(p3, p3);
  if (p2d2 < bd2) {
    bd2 = p2d2;
    bs  = sgnb(dot(ld3(tri + 15), p2));
  }
  if (p3d2 < bd2) {
    bd2 = p3d2;
    bs  = sgnb(dot(ld3(tri + 18), p3));
  }
  const double y1d2 = dot(y1, y1), y2d2 = dot(y2, y2), y3d2 = dot(y3, y3);
  if (t1 > 0.0 && t1 < 1.0 && y1d2 < bd2) {
    bd2 = y1d2;
    bs  = sgnb(dot(ld3(tri + 21), y1));
  }
  if (t2 > 0.0 && t2 < 1.0 && y2d2 < bd2) {
    bd2 = y2d2;
    bs  = sgnb(dot(ld3(tri + 24), y2));
  }
  if (t3 > 0.0 && t3 < 1.0 && y3d2 < bd2) {
    bd2 = y3d2;
    bs  = sgnb(dot(ld3(tri + 27), y3));
  }
  return bs * sqrt(bd2);
}

// ---- one triangle as a DCEL face: the algorithm of MeshSDF and FlatMeshSDF ----------------------
// (FaceT::signedDistance / unsignedDistance2, DCEL_FaceImplem.hpp:388-458; EdgeT, DCEL_EdgeImplem.hpp:
// 283-358; VertexT, DCEL_VertexImplem.hpp:368-380; Polygon2D crossing number,
// Polygon2DImplem.hpp:80-118,164-193).  It differs from the Triangle test above in the last bits:
// the face value is n . (p - centroid) with the DCEL normal, and vertex/edge signs are
// (pseudonormal . delta > 0 ? +1 : -1).

__device__ __forceinline__ D3 add3(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ double len3(D3 a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }

__device__ __forceinline__ double dcelVertexSd(D3 x, D3 vn, D3 P)
{
  const D3 d = sub(P, x);
  return len3(d) * ((dot(vn, d) > 0.0) ? 1.0 : -1.0);
}

__device__ __forceinline__ D3 dcelCentroid(D3 x0, D3 x1, D3 x2)
{
  const double is = 1.0 / 3.0;
  return scl(is, add3(add3(x0, x1), x2));
}

// crossing number of P projected into the face plane, in the 2D projection that drops the axis of
// largest |n| (the first on ties)
__device__ __forceinline__ bool dcelInside(const D3 (&x)[3], D3 n, D3 c, D3 P)
{
  const double ax = fabs(n.x), ay = fabs(n.y), az = fabs(n.z);
  int          ig = 0;
  if (ay > ax) {
    ig = 1;
  }
  if (az > (ig == 0 ? ax : ay)) {
    ig = 2;
  }
  const D3     q  = sub(P, scl(dot(n, sub(P, c)), n));
  const double qx = ig == 0 ? q.y : q.x, qy = ig == 2 ? q.y : q.z;
  int          cn = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const D3     a = x[i], b = x[(i + 1) % 3];
    const double ax2 = ig == 0 ? a.y : a.x, ay2 = ig == 2 ? a.y : a.z;
    const double bx2 = ig == 0 ? b.y : b.x, by2 = ig == 2 ? b.y : b.z;
    const bool   up = (ay2 <= qy) && (by2 > qy), down = (ay2 > qy) && (by2 <= qy);
    if (up || down) {
      const double t = (qy - ay2) / (by2 - ay2);
      if (qx < ax2 + t * (bx2 - ax2)) {
        cn++;
      }
    }
  }
  return (cn & 1) != 0;
}

// tri: the 30-double record (v0 v1 v2 n vn0 vn1 vn2 en0 en1 en2); fn: the DCEL face normal
__device__ double dcelFaceSd(const double* __restrict__ tri, const double* __restrict__ fn, D3 P)
{
  const D3 x[3] = {ld3(tri), ld3(tri + 3), ld3(tri + 6)};
  const D3 n    = ld3(fn);
  const D3 c    = dcelCentroid(x[0], x[1], x[2]);
  if (dcelInside(x, n, c, P)) {
    return dot(n, sub(P, c));
  }
  double best = CUDART_INF;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const int    j    = (i + 1) % 3;
    const D3     x2x1 = sub(x[j], x[i]);
    const double t    = dot(sub(P, x[i]), x2x1) / dot(x2x1, x2x1);
    double       d;
    if (t <= 0.0) {
      d = dcelVertexSd(x[i], ld3(tri + 12 + 3 * i), P);
    }
    else if (t >= 1.0) {
      d = dcelVertexSd(x[j], ld3(tri + 12 + 3 * j), P);
    }
    else {
      const D3 delta = sub(P, add3(x[i], scl(t, x2x1)));
      d              = ((dot(ld3(tri + 21 + 3 * i), delta) > 0.0) ? 1.0 : -1.0) * len3(delta);
    }
    best = fabs(d) < fabs(best) ? d : best;
  }
  return best;
}

__device__ double dcelFaceUd2(const double* __restrict__ tri, const double* __restrict__ fn, D3 P)
{
  const D3 x[3] = {ld3(tri), ld3(tri + 3), ld3(tri + 6)};
  const D3 n    = ld3(fn);
  const D3 c    = dcelCentroid(x[0], x[1], x[2]);
  if (dcelInside(x, n, c, P)) {
    const double nd = dot(n, sub(P, c));
    return nd * nd;
  }
  double best = CUDART_INF;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const D3 x2x1 = sub(x[(i + 1) % 3], x[i]);
    double   t    = dot(sub(P, x[i]), x2x1) / dot(x2x1, x2x1);
    t             = t < 0.0 ? 0.0 : (t > 1.0 ? 1.0 : t);
    const D3     delta = sub(P, add3(x[i], scl(t, x2x1)));
    const double d2    = dot(delta, delta);
    best               = d2 < best ? d2 : best;
  }
  return best;
}

// Whether an FP32 lower bound `low` of a triangle's distance leaves room for it within `reach`; dd its FP32
// squared distance, from whose root `low` was made: too small a square has underflowed and says nothing.
// (Not "low <= ...": a point on the triangle has no direction and a NaN bound.)
__device__ __forceinline__ bool mayReach(float low, float dd, float reach) { return !(dd >= 1e-30f) || !(low > reach); }

// The radius about the FP32 point, `shift` from the FP64 one, that holds an FP64 winner of value d (never so
// small that its square loses precision).
__device__ __forceinline__ float winnerRadius(double d, float shift)
{
  return (float(fabs(d)) + shift) * 1.000001f + 1e-18f;
}

// The triangle of smallest |d| in FP64 within `limit` (squared) of the FP32 point (px, py, pz), which lies
// `shift` from P (strict <, MeshDistanceFunctionsImplem.hpp:492-502; ties to the lower leaf position): all
// lanes on one point (mesh_point.cuh), whose FP32 distances shrink the bound and select the triangles worth
// an FP64 test.  `best` DBL_MAX and `bt` -1 if there is none.
//
// FP32 distances can be too small by more than `delta`: those of needle-like triangles, or where squares
// underflow.  A winner within the bound that the search ended with shows that they were not; without
// one it runs again with bounds from FP64 values alone.  NEAREST: `limit` itself comes from such a
// distance, and the nearest triangle is wanted however far it is.
template <int EVAL, bool UPPER, bool NEAREST>
__device__ int pointSearch64(const EbgMeshView& m, D3 P, float px, float py, float pz, float shift, float delta,
                             float limit, double& best, int& bt, PointMem& w)
{
  const float inf   = __int_as_float(0x7f800000);
  float       slack = delta + 2.f * shift, bound = limit;
  int         err   = 0;
  best              = DBL_MAX;
  bt                = -1;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    err |= pointSearch<UPPER>(m, px, py, pz, bound, slack, w, [&](bool active, uint32_t tri) {
      float dd = inf, low = inf;
      if (active) {
        const float4* h  = reinterpret_cast<const float4*>(m.hot + tri);
        const float4  h0 = __ldg(h), h1 = __ldg(h + 1), h2 = __ldg(h + 2);
        float         s, t;
        int           r;
        dd  = triDist2<false>(h0, h1, h2, px, py, pz, s, t, r);
        low = triLower(h0, h1, h2, px, py, pz, s, t, dd);
      }
      const float near = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(dd)));
      const float rn   = (sqrtf(near) * 1.00001f + slack) * 1.000001f;
      bound            = fminf(bound, rn * rn);
      const bool cand  = active && mayReach(low, dd, sqrtf(bound) * 1.00001f + delta);
      if (!__any_sync(FULL, cand)) {
        return;
      }
      double d = DBL_MAX;
      if (cand) {
        d = EVAL == 0 ? triSd64(m.tri64 + 30 * size_t(tri), P)
                      : dcelFaceSd(m.tri64 + 30 * size_t(tri), m.dcel_n + 3 * size_t(tri), P);
      }
      // the warp's least (|d|, triangle): non-negative doubles order like their words
      const uint32_t hi = cand ? uint32_t(__double2hiint(fabs(d))) : 0xffffffffu;
      const uint32_t mh = __reduce_min_sync(FULL, hi);
      const uint32_t lo = hi == mh ? uint32_t(__double2loint(d)) : 0xffffffffu;
      const uint32_t ml = __reduce_min_sync(FULL, lo);
      const uint32_t ti = cand && hi == mh && lo == ml ? tri : 0xffffffffu;
      const uint32_t mt = __reduce_min_sync(FULL, ti);
      const unsigned who = __ballot_sync(FULL, ti == mt && cand);
      if (mt == 0xffffffffu || who == 0u) {
        return; // only NaN values
      }
      const double dm = __shfl_sync(FULL, d, __ffs(int(who)) - 1);
      if (fabs(dm) < fabs(best) || (fabs(dm) == fabs(best) && int(mt) < bt)) {
        best           = dm;
        bt             = int(mt);
        const float rb = winnerRadius(dm, shift);
        bound          = fminf(bound, rb * rb);
      }
    });
    const float rb = winnerRadius(best, shift);
    if ((bt >= 0 && rb * rb <= bound) || (!NEAREST && bound == limit)) {
      break;
    }
    slack = inf; // shrinks nothing
    bound = NEAREST ? (bt >= 0 ? rb * rb : FLT_MAX) : limit;
  }
  return err;
}

} // namespace

} // namespace ebg

#endif
