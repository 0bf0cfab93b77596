// Up to which distance a lower bound of the distance to a triangle also holds
// for the reference's f32 arithmetic.  No CUDA needed: the tests compile this
// header for the host.
//
// A search skips a triangle when a bound lb <= D, D the distance from its query
// p to the triangle, exceeds the best distance so far.  That is exact if the
// distance r that closest_point_proper gives is never below lb.  r falls short
// of D by more than rounding only where rounding lets the face region through
// although the foot f of the perpendicular lies outside the triangle, by g.
// The f32 point lies in the triangle's plane up to rounding, so r is then at
// least h = sqrt(D^2 - g^2).
//
// With L and s the longest and shortest edge, W twice the area, a = L^2 / W,
// Q = s / a and u = 2^-24: the dot products d1 .. d6 err by at most 5u |edge|
// |p - vertex|, vc = d1 d4 - d3 d2 by 24u |ab| |ac| |ap| |bp| and va, vb alike.
//
//  1. If va, vb and vc all come out non-negative, the point lies in the triangle
//     and r >= D.  Otherwise one of them is negative and its edge's test failed
//     by d1 .. d6: with the vertex tests, which failed too, this leaves f within
//     58u a^2 (1 + D / L) |vp| of a vertex v.  For a <= 64 and D <= 8 L that is at most
//     0.13 |vp|, so |vp| <= 1.15 D, and an edge line is crossed unnoticed by at
//     most g = 28u D (1.15 D / Q + a) + 19u a D.
//  2. At any distance, going through the regions one by one: g <= 28u (D + L)^2 / Q.
//
// Up to D = 1.01 * 1024 Q either way (1 below 8 L, 2 above) D - h <= 40u D; r's own
// rounding takes at most 25u |triangle| + 5u D, and the slack of the bounds, 2^-17 =
// 128u of |triangle| + |p| (largest coordinates; D is at most sqrt(3) times their
// sum), covers both.  Farther away, up to 370 reaches, g < 0.65 D, and r still
// exceeds every best distance within the reach.  Callers keep D inside that.
//
// The reach is therefore 1024 Q, and 0 for triangles thinner than a <= 64 and
// where products of four lengths could leave the normal range (an area below
// 2^-51; L times the reach above 2^52).  Coordinates must be below 2^28.
// Triangles without an area never enter the face region: they have no limit.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define M2S_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define M2S_HOST_DEVICE inline
#endif

namespace m2s {

constexpr float kReach = 1024.0f;
constexpr float kReachThin = 64.0f;
constexpr float kReachScale = 268435456.0f;  // 2^28: of the coordinates
constexpr float kReachSpan = 256.0f;         // reaches that a pillbox's box may span

// The reach of triangle a, b, c (three floats each), which has an area.
M2S_HOST_DEVICE float tri_reach(const float* a, const float* b, const float* c) {
  const float ux = b[0] - a[0], uy = b[1] - a[1], uz = b[2] - a[2];
  const float vx = c[0] - a[0], vy = c[1] - a[1], vz = c[2] - a[2];
  const float ex = c[0] - b[0], ey = c[1] - b[1], ez = c[2] - b[2];
  const float nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
  const float w2 = nx * nx + ny * ny + nz * nz;
  const float e0 = ux * ux + uy * uy + uz * uz, e1 = vx * vx + vy * vy + vz * vz, e2 = ex * ex + ey * ey + ez * ez;
  const float l2 = fmaxf(e0, fmaxf(e1, e2)), s2 = fminf(e0, fminf(e1, e2)), w = sqrtf(w2);
  if (!(w2 > 7.8886090522101181e-31f && l2 <= kReachThin * w)) return 0.0f;  // 2^-100; also where anything is NaN
  return fminf(kReach * w * sqrtf(s2) / l2, 4503599627370496.0f / sqrtf(l2));  // 2^52
}

}  // namespace m2s
