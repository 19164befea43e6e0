// sun_fit.cuh -- the fitted sun rays of k_first_order_fit.cu: their table and
// its evaluation at one point.
#pragma once

#include "atmo_device.cuh"

namespace sfsim {

constexpr int kFitRows = 8192;   // values of sqrt(q / q_top)
constexpr int kFitDeg = 5;       // degree of the segments' polynomials
constexpr int kFitNodes = kFitDeg + 1;

// Geometry of a height: q, cq = top^2 - r^2, the range [dmin, dmin + range] of exit distances.
struct FitRange {
  float cq, dmin, range;
};
__device__ __forceinline__ FitRange fit_range(const AtmoParams& P, float q) {
  FitRange f;
  f.cq = fmaxf(P.f_Hh2 - q, 0.0f);
  f.dmin = f.cq / (P.f_top + sqrtf(fmaf(P.f_R, P.f_R, q)));
  f.range = sqrtf(q) + P.f_Hh - f.dmin;
  return f;
}

__device__ __forceinline__ float reciprocal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The sun ray of a lit point at q = |p|^2 - R^2 with b = p.l: its length times
// the mean densities (Rayleigh, Mie) by the fits of `segs` segments in `table`.
// The same steps as in k_first_order_fit, which says why they are these; the
// coefficients are interpolated between the table's rows for this point alone.
__device__ __forceinline__ float2 sun_fit_depths(const AtmoParams& P, const float4* table, int segs, float q, float b) {
  const float qc = fminf(fmaxf(q, 0.0f), P.f_Hh2), rho = sqrtf(qc);
  const FitRange f = fit_range(P, qc);
  const float x = fminf(sqrtf(qc / P.f_Hh2), 1.0f) * (float)(kFitRows - 1);
  const int row = min((int)x, kFitRows - 2);
  const float w = x - (float)row;
  const float root = Bulk<float>::sqrt(fmaf(b, b, f.cq)), size = fabsf(b), far = size + root;
  const bool up = b >= 0.0f;
  const float num = up ? f.cq : fmaf(-b, b, qc) * (far + (rho + P.f_Hh));
  const float part = num * reciprocal(up ? far : (root + P.f_Hh) * (rho + size));
  const float scale = 1.0f / f.range, zmax = __uint_as_float(__float_as_uint((float)segs) - 1u);
  const float z = __saturatef(fmaf(part, scale, up ? -f.dmin * scale : 0.0f)) * zmax;
  const int i = min((int)z, segs - 1);
  const float t = up ? (z - (float)i) - 0.5f : 0.5f - (z - (float)i);
  const float4* k = table + ((size_t)row * segs + (up ? i : segs - 1 - i)) * (kFitNodes / 2);
  float2 p = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int c = kFitNodes / 2 - 1; c >= 0; c--) {
    const float4 A = __ldg(k + c), B = __ldg(k + c + segs * (kFitNodes / 2));
    p.x = fmaf(fmaf(p.x, t, fmaf(B.z - A.z, w, A.z)), t, fmaf(B.x - A.x, w, A.x));
    p.y = fmaf(fmaf(p.y, t, fmaf(B.w - A.w, w, A.w)), t, fmaf(B.y - A.y, w, A.y));
  }
  const float dist = up ? part : far;
  return make_float2(dist * Bulk<float>::exp2(p.x), dist * Bulk<float>::exp2(p.y));
}

}  // namespace sfsim
