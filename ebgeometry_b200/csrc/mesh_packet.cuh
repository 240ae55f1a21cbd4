// The tests of a packet's box against the tree, shared by the FP32 packet search (mesh_packet.cu, which
// explains them) and the FP64 pass (mesh_band64.cu).
#ifndef EBG_MESH_PACKET_CUH
#define EBG_MESH_PACKET_CUH

#include "ebg_device.cuh"
#include "mesh_traverse.cuh"

namespace ebg {

__device__ __forceinline__ float warpMin(float x)
{
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float warpMax(float x)
{
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

// The point of the triangle with weights s, t, moved into the triangle where rounding left it outside.
__device__ __forceinline__ void triPoint(const float4 h0, const float4 h1, const float4 h2, float s, float t, float& x,
                                         float& y, float& z)
{
  s             = fmaxf(s, 0.f);
  t             = fmaxf(t, 0.f);
  const float k = __fdividef(1.f, fmaxf(1.f, s + t));
  s *= k;
  t *= k;
  x = h0.x + fmaf(s, h1.x, t * h2.x);
  y = h0.y + fmaf(s, h1.y, t * h2.y);
  z = h0.z + fmaf(s, h1.z, t * h2.z);
}

// Whether some corner of the packet's box (half-extents hx, hy, hz about c) reaches the entry whose
// nearest point to c lies at c - (wx, wy, wz); A0, A1 the corners' bounds, signs (+++, ---, ++-, --+) and
// (+-+, -+-, +--, -++).  An entry that contains c (no direction, NaN) is kept.
__device__ __forceinline__ bool cornersReach(const float4 A0, const float4 A1, float hx, float hy, float hz, float wx,
                                             float wy, float wz, float& d2)
{
  d2              = fmaf(wx, wx, fmaf(wy, wy, wz * wz));
  const float inv = rsqrtf(d2), d = d2 * inv;
  const float tx = wx * hx * inv, ty = wy * hy * inv, tz = wz * hz * inv;
  const float p = tx + ty, q = tx - ty;
  const float k0 = p + tz, k1 = p - tz, k2 = q + tz, k3 = q - tz;
  const float m0 = fmaxf(fmaxf(A0.x - k0, A0.y + k0), fmaxf(A0.z - k1, A0.w + k1));
  const float m1 = fmaxf(fmaxf(A1.x - k2, A1.y + k2), fmaxf(A1.z - k3, A1.w + k3));
  return !(fmaxf(m0, m1) < d);
}

__device__ __forceinline__ bool cornersReachObb(const float4 A0, const float4 A1, float hx, float hy, float hz,
                                                const float4* __restrict__ ob, float cx, float cy, float cz, float& d2)
{
  const float4 o0 = __ldg(ob), o1 = __ldg(ob + 1), o2 = __ldg(ob + 2), o3 = __ldg(ob + 3);
  const float  a = fmaf(o0.x, cx, fmaf(o0.y, cy, fmaf(o0.z, cz, -o0.w)));
  const float  b = fmaf(o1.x, cx, fmaf(o1.y, cy, fmaf(o1.z, cz, -o1.w)));
  const float  e = fmaf(o2.x, cx, fmaf(o2.y, cy, fmaf(o2.z, cz, -o2.w)));
  const float  wa = copysignf(fmaxf(fabsf(a) - o3.x, 0.f), a);
  const float  wb = copysignf(fmaxf(fabsf(b) - o3.y, 0.f), b);
  const float  we = copysignf(fmaxf(fabsf(e) - o3.z, 0.f), e);
  return cornersReach(A0, A1, hx, hy, hz, fmaf(wa, o0.x, fmaf(wb, o1.x, we * o2.x)),
                      fmaf(wa, o0.y, fmaf(wb, o1.y, we * o2.y)), fmaf(wa, o0.z, fmaf(wb, o1.z, we * o2.z)), d2);
}

// The packet's (or group's) box and the mesh point that bounds its distances.
struct Reach
{
  float cx, cy, cz, hx, hy, hz;
};

// The corners' bounds |corner - a| by the lanes 0..7 in cornersReach's order (bit i of each mask: the
// sign of corner i on that axis, 1 = plus).
__device__ __forceinline__ void setCorners(float4* corner, const Reach& r, float ax, float ay, float az, float delta)
{
  const int   lane = threadIdx.x & 31;
  const bool  sx = (0x55u >> (lane & 7)) & 1u, sy = (0xa5u >> (lane & 7)) & 1u, sz = (0x99u >> (lane & 7)) & 1u;
  const float ex = (sx ? r.cx + r.hx : r.cx - r.hx) - ax, ey = (sy ? r.cy + r.hy : r.cy - r.hy) - ay,
              ez = (sz ? r.cz + r.hz : r.cz - r.hz) - az;
  const float A  = sqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez))) * 1.000004f + delta;
  __syncwarp(); // the box before has been read
  if (lane < 8) {
    reinterpret_cast<float*>(corner)[lane] = A;
  }
  __syncwarp();
}

// Whether the packet reaches the child of slot k of node `node`; child and cw are its words, d2 the squared
// distance from the box's centre to it.
__device__ __forceinline__ bool childReach(const EbgMeshView& m, const float4* corner, const Reach& r, uint32_t node, int k,
                                           uint32_t& child, uint32_t& cw, float& d2)
{
  const float4  A0 = corner[0], A1 = corner[1];
  const float4* sl = reinterpret_cast<const float4*>(m.children + 4 * size_t(node) + k);
  const float4  lo = __ldg(sl), hi = __ldg(sl + 1);
  child = __float_as_uint(lo.w);
  cw    = __float_as_uint(hi.w);
  if ((child | cw) == 0u) { // an empty slot
    return false;
  }
  if (!cornersReach(A0, A1, r.hx, r.hy, r.hz, r.cx - fminf(fmaxf(r.cx, lo.x), hi.x),
                    r.cy - fminf(fmaxf(r.cy, lo.y), hi.y), r.cz - fminf(fmaxf(r.cz, lo.z), hi.z), d2)) {
    return false;
  }
  const bool leaf = (child & EBG_LEAF_BIT) != 0u;
  if (!leaf && !(cw & EBG_NODE_HAS_OBB)) {
    return true;
  }
  return cornersReachObb(A0, A1, r.hx, r.hy, r.hz,
                         reinterpret_cast<const float4*>(leaf ? m.obb + (cw >> EBG_COUNT_BITS) : m.node_obb + child), r.cx,
                         r.cy, r.cz, d2);
}

// The lanes (bits) whose bound reaches this lane's leaf box: lanes [b, e), points and bounds in q.
__device__ __forceinline__ unsigned lanesReach(const float4* __restrict__ ob, const float4* q, int b, int e)
{
  const float4 o0 = __ldg(ob), o1 = __ldg(ob + 1), o2 = __ldg(ob + 2), o3 = __ldg(ob + 3);
  unsigned     mask = 0u;
#pragma unroll 1
  for (int j = b & ~3; j < e; j += 4) {
    unsigned four = 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float4 p = q[j + i];
      if (obbDist2(o0, o1, o2, o3, p.x, p.y, p.z) <= p.w) {
        four |= 1u << i;
      }
    }
    mask |= four << j;
  }
  return mask;
}

} // namespace ebg

#endif
