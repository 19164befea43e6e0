// k_setup.cu -- node maps, transmittance and surface-base tables, per-row ray
// samples and per-height sphere directions of the atmosphere LUT build.
#include <type_traits>

#include "atmo_device.cuh"
#include "kernels.h"

namespace sfsim {

// ---------------------------------------------------------------------------
// Re-interpolation maps.  Every table that the reference writes is
// make-lookup-table of an interpolated function, so each node's value is the
// table interpolated at forward(backward(node)) (interpolate.clj:68-110,
// atmosphere_lut.clj:94-101).  These kernels store that coordinate per node.
// ---------------------------------------------------------------------------

// Per view row (i, j), once: the row's geometry (RowInfo), and its height and
// elevation coordinates, which every node of the row shares (row_map: only the
// accumulations and the outputs read them, so they are no part of the chain to
// the first order).
__device__ void row_info(const AtmoParams* params, const BuildDims& d, RowInfo* info, long long row, int b) {
  const long long nrows = d.rows();
  const AtmoParams& P = params[b];
  const int j = (int)(row % d.n1), i = (int)(row / d.n1);
  double r, sv, cv;
  int above;
  view_geometry(P, d, i, j, &r, &sv, &cv, &above);
  const d3 x = mk3(r, 0, 0), v = mk3(sv, cv, 0);
  const d3 e = above ? atmosphere_intersection(P, x, v) : surface_intersection(P, x, v);
  const d3 D = sub3(e, x);
  RowInfo ri;
  ri.r = r;
  ri.sv = sv;
  ri.cv = cv;
  ri.D[0] = D.x;
  ri.D[1] = D.y;
  ri.D[2] = D.z;
  ri.L = mag3(D);
  ri.Ls = ri.L / d.S;
  {
    const double c0 = dmul(dsub(r, P.R), dadd(r, P.R)), xD = dmul(r, D.x), DD = dot3(D, D);
    ri.qmin = DD > 0.0 ? c0 - xD * xD / DD : c0;
    ri.t = DD > 0.0 ? xD / DD : 0.0;
  }
  ri.f_r = (float)r;
  ri.f_sv = (float)sv;
  ri.f_cv = (float)cv;
  ri.f_D[0] = (float)D.x;
  ri.f_D[1] = (float)D.y;
  ri.f_D[2] = (float)D.z;
  ri.f_Ls = (float)ri.Ls;
  ri.above = above;
  info[b * nrows + row] = ri;
}

template <class Real>
__device__ void row_map(const AtmoParams* params, const BuildDims& d, Remap2<Real>* rowmap, long long row, int b) {
  const AtmoParams& P = params[b];
  double r, sv, cv;
  int above;
  view_geometry(P, d, (int)(row / d.n1), (int)(row % d.n1), &r, &sv, &cv, &above);
  const d3 x = mk3(r, 0, 0), v = mk3(sv, cv, 0);
  Remap2<Real> m;
  split_coord<Real>(height_to_index(P, d.n0, mag3(x)), d.n0, &m.u[0], &m.s[0]);
  split_coord<Real>(elevation_to_index(P, d.n1, x, v, above), d.n1, &m.u[1], &m.s[1]);
  rowmap[b * d.rows() + row] = m;
}

// The height and elevation coordinates of a node are its row's (row_map);
// its light direction l = index-to-sun-direction(v, sin(k), a) has
// x.l = r sin(k) with x = (r, 0, 0), so its sun-elevation coordinate is the
// (i, k) one of point_row, which also holds sin(k).  Left per node are the
// sun-angle coordinate and l itself.
template <class Real>
__global__ void k_remap4(BuildDims d, const RowInfo* info, const PointRow<Real>* prow,
                         const double* __restrict__ hdvs, Coord<Real>* angle, CellGeom<Real>* geom) {
  const long long n4 = d.n4();
  const long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (node >= n4) return;
  int a = (int)(node % d.n3);
  int k = (int)((node / d.n3) % d.n2);
  const long long row = node / ((long long)d.n3 * d.n2);
  const int i = (int)(row / d.n1);
  const RowInfo& ri = info[b * d.rows() + row];
  const PointRow<Real>& pk = prow[((long long)b * d.n0 + i) * d.n2 + k];
  const double sv = ri.sv, cv = ri.cv;
  const d3 v = mk3(sv, cv, 0);
  const d3 l = node_light(sv, cv, pk.ss, pk.cs, hdvs[a]);
  Coord<Real> m;
  split_coord<Real>(sun_angle_to_index(d.n3, v, l), d.n3, &m.u, &m.s);
  angle[b * n4 + node] = m;
  geom[b * n4 + node] = cell_geom<Real>(sv, cv, l);
}

template <class Real>
__device__ void remap_T(const AtmoParams* params, const BuildDims& d, Remap2<Real>* out, long long node, int b) {
  const long long n = d.nT();
  const AtmoParams& P = params[b];
  int j = (int)(node % d.nT1), i = (int)(node / d.nT1);
  double r = index_to_radius(P, d.nT0, (double)i), sv, cv;
  int above;
  index_to_elevation(P, d.nT1, r, (double)j, &sv, &cv, &above);
  d3 x = mk3(r, 0, 0), v = mk3(sv, cv, 0);
  Remap2<Real> m;
  split_coord<Real>(height_to_index(P, d.nT0, mag3(x)), d.nT0, &m.u[0], &m.s[0]);
  split_coord<Real>(elevation_to_index(P, d.nT1, x, v, above), d.nT1, &m.u[1], &m.s[1]);
  out[b * n + node] = m;
}

__host__ __device__ inline void surface_node(const AtmoParams& P, const BuildDims& d, int i, int k, d3* x, d3* l) {
  double r = index_to_radius(P, d.nE0, (double)i);
  double s = index_to_sin_sun_elevation(d.nE1, (double)k);
  double c = sqrt(dmax(0.0, 1 - sqr(s)));
  *x = mk3(r, 0, 0);
  *l = mk3(s, c, 0);
}

template <class Real>
__device__ void remap_E(const AtmoParams* params, const BuildDims& d, Remap2<Real>* out, long long node, int b) {
  const long long n = d.nE();
  const AtmoParams& P = params[b];
  int k = (int)(node % d.nE1), i = (int)(node / d.nE1);
  d3 x, l;
  surface_node(P, d, i, k, &x, &l);
  Remap2<Real> m;
  split_coord<Real>(height_to_index(P, d.nE0, mag3(x)), d.nE0, &m.u[0], &m.s[0]);
  split_coord<Real>(sun_elevation_to_index(d.nE1, x, l), d.nE1, &m.u[1], &m.s[1]);
  out[b * n + node] = m;
}

// ---------------------------------------------------------------------------
// Transmittance table (atmosphere_lut.clj:74, atmosphere.clj:114-128)
// ---------------------------------------------------------------------------

template <class Real>
__device__ void transmittance_node(const AtmoParams* params, const BuildDims& d, Vec4<Real>* T, long long node, int b) {
  const long long n = d.nT();
  const AtmoParams& P = params[b];
  int j = (int)(node % d.nT1), i = (int)(node / d.nT1);
  double r = index_to_radius(P, d.nT0, (double)i), sv, cv;
  int above;
  index_to_elevation(P, d.nT1, r, (double)j, &sv, &cv, &above);
  d3 x = mk3(r, 0, 0), v = mk3(sv, cv, 0);
  d3 e = above ? atmosphere_intersection(P, x, v) : surface_intersection(P, x, v);
  Real tau[3];
  segment_depth<Real>(P, x, sub3(e, x), d.S, tau);
  Vec4<Real> o;
  o.x = exp_neg(tau[0]);
  o.y = exp_neg(tau[1]);
  o.z = exp_neg(tau[2]);
  o.w = 0;
  T[b * n + node] = o;
}

// ---------------------------------------------------------------------------
// Surface radiance of direct sun light E0 (atmosphere.clj:131-137)
// ---------------------------------------------------------------------------

template <class Real>
__device__ void surface_base_node(const AtmoParams* params, const BuildDims& d, Vec4<Real>* E0, long long node, int b) {
  const long long n = d.nE();
  const AtmoParams& P = params[b];
  int k = (int)(node % d.nE1), i = (int)(node / d.nE1);
  d3 x, l;
  surface_node(P, d, i, k, &x, &l);
  d3 normal = mul3(x, 1.0 / mag3(x));
  double cosine = dmax(0.0, dot3(normal, l));
  Vec4<Real> o;
  o.x = o.y = o.z = o.w = 0;
  if (cosine > 0.0) {
    d3 e = atmosphere_intersection(P, x, l);
    Real tau[3];
    segment_depth<Real>(P, x, sub3(e, x), d.S, tau);
    o.x = exp_neg(tau[0]) * (Real)(P.intensity[0] * cosine);
    o.y = exp_neg(tau[1]) * (Real)(P.intensity[1] * cosine);
    o.z = exp_neg(tau[2]) * (Real)(P.intensity[2] * cosine);
  }
  E0[b * n + node] = o;
}

// ---------------------------------------------------------------------------
// View rows: for every (height i, elevation j) of the 4-D space the ray from
// x to its extremity (atmosphere.clj:192-200) and its S midpoint samples.
// One thread per (row, sample).
// ---------------------------------------------------------------------------

// Sample s of a row, everything but the optical depth from the row's node.
// The sample's coordinates are generic (between nodes), so the FP64 forms
// are reduced where that moves them by rounding only: the point (r + su D.x,
// su D.y, su D.z) without adding x's zero components, the atmosphere's
// horizon distance P.Hh in the height coordinate, and rs = p.v in the
// elevation coordinate (elevation-to-index forms |p| ((p.v) / |p|)).
template <class Real>
__device__ inline RowSample<Real> view_sample(const AtmoParams& P, const BuildDims& d, const RowInfo& ri, int s) {
  // sample point as integral-ray forms it (ray.clj:22-24)
  const double su = (0.5 + s) * d.inv_S;
  const d3 p = mk3(dadd(ri.r, dmul(ri.D[0], su)), dmul(ri.D[1], su), dmul(ri.D[2], su));
  const double pr = mag3(p);
  const double h = pr - P.R;
  RowSample<Real> o;
  if (std::is_same<Real, float>::value) {
    // the densities exp(-h/H) as the FP32 integrands form them
    o.er = (Real)Bulk<float>::exp2((float)h * P.f_kr);
    o.em = (Real)Bulk<float>::exp2((float)h * P.f_km);
    o.inv_r = (Real)__frcp_rn((float)pr);
  } else {
    o.er = (Real)exp(-(h / P.ray_scale));
    o.em = (Real)exp(-(h / P.mie_scale));
    o.inv_r = (Real)(1.0 / pr);
  }
  o.q = (Real)(h * (pr + P.R));
  o.us = (Real)su;
  // height-to-index and elevation-to-index (atmosphere.clj:239-253, 273-288)
  const double rho = horizon_distance(P, pr);
  split_coord<Real>(dmul((double)(d.n0 - 1), rho / P.Hh), d.n0, &o.u0, &o.s0);
  const double rs = dadd(dmul(p.x, ri.sv), dmul(p.y, ri.cv));
  const double Delta = dsub(sqr(rs), sqr(rho));
  double idx;
  if (ri.above)
    idx = dsub(0.5, limit_quot(dsub(rs, sqrt(dmax(0.0, dadd(Delta, P.Hh2)))), dadd(dadd(rho, rho), dmul(2.0, P.Hh)),
                               -0.5, 0.0));
  else
    idx = dadd(0.5, limit_quot(dadd(rs, sqrt(dmax(0.0, Delta))), dadd(rho, rho), -0.5, 0.0));
  split_coord<Real>(dmul((double)(d.n1 - 1), idx), d.n1, &o.u1, &o.s1);
  o.pad = 0;
  return o;
}

// T(x, p_s) by the nested midpoint sums over x -> p_s = x + su D (S samples).
// The segment's height form comes from the row's (qmin and t are the same
// for every su up to rounding; u* scales as t / su), and its sample step in
// distance is su L / S.
template <class Real>
__device__ inline void view_depth(const AtmoParams& P, const BuildDims& d, const RowInfo& ri, int s, Real tau[3]) {
  if (!(ri.L > 0.0)) {
    tau[0] = tau[1] = tau[2] = 0;
    return;
  }
  const double du = d.inv_S, su = (0.5 + s) * du;
  const double c0 = dmul(dsub(ri.r, P.R), dadd(ri.r, P.R));
  const double DD = su * su * (ri.D[0] * ri.D[0] + ri.D[1] * ri.D[1] + ri.D[2] * ri.D[2]);
  QForm f;
  f.C = DD;
  if (DD > 0.0 && fabs(ri.qmin) < c0) {
    f.A = ri.qmin;
    f.B = 0.0;
    f.w0 = 0.5 * du + ri.t / su;
  } else {
    f.A = c0;
    f.B = 2.0 * (su * (ri.r * ri.D[0]));
    f.w0 = 0.5 * du;
  }
  Real sr, sm;
  optical_sums_w<Real, 5>((Real)f.A, (Real)f.B, (Real)f.C, (Real)f.w0, (Real)du, d.S, Bulk<Real>::hpoly(P),
                          Bulk<Real>::alpha(P), Bulk<Real>::beta(P), Bulk<Real>::kr(P), Bulk<Real>::km(P), sr, sm);
  const Real a = (Real)(su * ri.Ls);
#pragma unroll
  for (int ch = 0; ch < 3; ch++) tau[ch] = a * (Bulk<Real>::ray_ext(P, ch) * sr + Bulk<Real>::mie_ext(P, ch) * sm);
}

template <class Real>
__global__ void k_view_rows(const AtmoParams* params, BuildDims d, const RowInfo* info, RowSample<Real>* samples) {
  const long long nrows = d.rows();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (t >= nrows * d.S) return;
  const AtmoParams& P = params[b];
  const int s = (int)(t % d.S);
  const long long row = t / d.S;
  const RowInfo& ri = info[b * nrows + row];
  RowSample<Real> o = view_sample<Real>(P, d, ri, s);
  view_depth<Real>(P, d, ri, s, o.tau);
  samples[(b * nrows + row) * d.S + s] = o;
}

// The same samples with the optical depth from the row's node x to each
// p_s by one prefix scan over the row (SFSIM_ATMO_SCAN_RAYS), instead of S
// samples between x and every p_s.  With cells [n du, (n + 1) du] of the
// row parameter u (du = 1/S) and rho_n the density at the midpoint u_n of
// cell n (the sample points themselves),
//   tau(x, p_s) = L du (sum_{n<s} rho_n + rho((s + 1/4) du) / 2):
// the midpoint rule on the whole cells before p_s and on the half cell up
// to it.  The densities are the integrand of the nested sums: the row's
// height form q(u) (segment_q_form) in Real.  One warp per row; lane l takes
// samples l, l + 32, ...; each 32 samples are one shuffle scan, carried on
// to the next 32.
template <class Real>
__global__ void k_view_rows_scan(const AtmoParams* params, BuildDims d, const RowInfo* info,
                                 RowSample<Real>* samples) {
  const long long nrows = d.rows();
  const int lane = threadIdx.x & 31;
  const long long row = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int b = blockIdx.y;
  if (row >= nrows) return;  // whole warps
  const AtmoParams& P = params[b];
  const RowInfo& ri = info[b * nrows + row];
  const double du = 1.0 / d.S;
  const double c0 = dmul(dsub(ri.r, P.R), dadd(ri.r, P.R));
  const d3 D = mk3(ri.D[0], ri.D[1], ri.D[2]);
  const QForm f = segment_q_form(c0, dmul(ri.r, D.x), dot3(D, D), du);
  const Real A = (Real)f.A, B = (Real)f.B, C = (Real)f.C, w0 = (Real)f.w0, dur = (Real)du;
  const Real* hp = Bulk<Real>::hpoly(P);
  const Real al = Bulk<Real>::alpha(P), be = Bulk<Real>::beta(P), kr = Bulk<Real>::kr(P), km = Bulk<Real>::km(P);
  const Real Ls = (Real)(ri.L * du);
  Real carry_r = 0, carry_m = 0;
  for (int s0 = 0; s0 < d.S; s0 += 32) {
    const int s = s0 + lane;
    Real rr = 0, rm = 0, qr = 0, qm = 0;
    if (s < d.S) {
      // w of the sample's midpoint (as optical_sums_w forms it) and of the
      // half cell's midpoint (s + 1/4) du
      const Real wm = fma(Real(s), dur, w0);
      const Real wq = fma(Real(s) - Real(0.25), dur, w0);
      const Real hm = height_from_q<Real, 5>(fma(wm, fma(wm, C, B), A), hp, al, be);
      const Real hq = height_from_q<Real, 5>(fma(wq, fma(wq, C, B), A), hp, al, be);
      rr = Bulk<Real>::exp2(hm * kr);
      rm = Bulk<Real>::exp2(hm * km);
      qr = Bulk<Real>::exp2(hq * kr);
      qm = Bulk<Real>::exp2(hq * km);
    }
    // inclusive scan over the 32 lanes
    Real ir = rr, im = rm;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
      const Real ur = __shfl_up_sync(0xffffffffu, ir, k), um = __shfl_up_sync(0xffffffffu, im, k);
      if (lane >= k) {
        ir += ur;
        im += um;
      }
    }
    Real er = __shfl_up_sync(0xffffffffu, ir, 1), em = __shfl_up_sync(0xffffffffu, im, 1);
    if (lane == 0) er = em = 0;
    if (s < d.S) {
      RowSample<Real> o = view_sample<Real>(P, d, ri, s);
      const Real sr = carry_r + er + Real(0.5) * qr, sm = carry_m + em + Real(0.5) * qm;
#pragma unroll
      for (int ch = 0; ch < 3; ch++) o.tau[ch] = Ls * (Bulk<Real>::ray_ext(P, ch) * sr + Bulk<Real>::mie_ext(P, ch) * sm);
      samples[(b * nrows + row) * d.S + s] = o;
    }
    carry_r += __shfl_sync(0xffffffffu, ir, 31);
    carry_m += __shfl_sync(0xffffffffu, im, 31);
  }
}

// ---------------------------------------------------------------------------
// Rings of the quadratures
// ---------------------------------------------------------------------------

// First direction of ring k of `rings` between polar angles 0 and `range`: the
// directions follow one another by ring and their polar cosine falls from ring
// to ring.
__device__ inline int ring_start(const DirLocal* dirs, int count, int rings, double range, int k) {
  if (k == 0) return 0;
  if (k >= rings) return count;
  const double edge = cos(range * k / rings);  // between rings k - 1 and k
  int lo = 0, hi = count;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (dirs[mid].x < edge)
      hi = mid;
    else
      lo = mid + 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// Sphere rings of point scatter per height row (atmosphere.clj:203-222,
// sphere.clj:62-105): where the ring's directions end, whether that end is on
// the ground, the elevation coordinate of the dS lookup and, for ground ends,
// T(x, g) * brightness / pi.  x = (r, 0, 0), so the ring's directions have
// the same first component and with it the same end; the ring's first
// direction stands for all.  A warp takes a ring, its lanes the samples of the
// ground's optical depth.
// ---------------------------------------------------------------------------

template <class Real>
__device__ void sphere_ring(const AtmoParams* params, const BuildDims& d, const DirLocal* dirs, SphereRing<Real>* out,
                            int i, int k, int b, int lane) {
  const AtmoParams& P = params[b];
  const double r = index_to_radius(P, d.n0, (double)i);
  const d3 x = mk3(r, 0, 0);
  const d3 n = axis_normal(P, x);
  const d3 o1 = orthogonal(n);
  const d3 o2 = cross3(n, o1);
  const int w = ring_start(dirs, d.P, d.T, M_PI, k);
  const d3 omega = to_world(n, o1, o2, dirs[w]);
  const d3 g = ray_extremity(P, x, omega);
  const int surface = surface_point(P, g);
  SphereRing<Real> o;
  o.x0 = (Real)omega.x;
  o.weight = (Real)dirs[w].w;
  o.surface = surface;
  o.w0 = w;
  o.n = ring_start(dirs, d.P, d.T, M_PI, k + 1) - w;
  split_coord<Real>(elevation_to_index(P, d.n1, x, omega, !surface), d.n1, &o.u1, &o.s1);
  o.tR = o.ground[0] = o.ground[1] = o.ground[2] = 0;
  if (surface) {
    Real tau[3];
    segment_depth_warp<Real>(P, x, sub3(g, x), d.S, lane, tau);
    for (int c = 0; c < 3; c++) o.ground[c] = exp_neg(tau[c]) * (Real)(P.brightness[c] / M_PI);
    const double tR = mag3(sub3(g, x)) / P.R;
    o.tR = ordinary_radii(P) ? (Real)tR : Real(0);
  }
  if (lane == 0) out[((long long)b * d.n0 + i) * d.T + k] = o;
}

// Per direction: its components across the axis (the same at every height),
// and in FP64 builds the ground point's height coordinate, which is on the
// ground up to its rounding.
template <class Real>
__device__ void sphere_direction(const AtmoParams* params, const BuildDims& d, const DirLocal* dirs, Real* dirs4,
                                 Real* offsets, int i, int t, int b) {
  const AtmoParams& P = params[b];
  const d3 x = mk3(index_to_radius(P, d.n0, (double)i), 0, 0);
  const d3 n = axis_normal(P, x);
  const d3 o1 = orthogonal(n);
  const d3 omega = to_world(n, o1, cross3(n, o1), dirs[t]);
  if (i == 0 && b == 0) {
    dirs4[4 * t] = dirs4[4 * t + 1] = (Real)omega.y;
    dirs4[4 * t + 2] = dirs4[4 * t + 3] = (Real)omega.z;
  }
  if (std::is_same<Real, double>::value) {
    const d3 g = ray_extremity(P, x, omega);
    int u = 0;
    Real s = 0;
    if (surface_point(P, g)) split_coord<Real>(height_to_index(P, d.nE0, mag3(g)), d.nE0, &u, &s);
    offsets[((long long)b * d.n0 + i) * d.P + t] = s;
  }
}

// The same per direction, for the work census (one thread per height and direction).
template <class Real>
__global__ void k_sphere_setup(const AtmoParams* params, BuildDims d, const DirLocal* dirs,
                               SphereDir<Real>* out) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (t >= (long long)d.n0 * d.P) return;
  const AtmoParams& P = params[b];
  const int w = (int)(t % d.P), i = (int)(t / d.P);
  double r = index_to_radius(P, d.n0, (double)i);
  d3 x = mk3(r, 0, 0);
  d3 n = mul3(x, 1.0 / mag3(x));
  d3 o1 = orthogonal(n);
  d3 o2 = cross3(n, o1);
  d3 omega = to_world(n, o1, o2, dirs[w]);
  d3 g = ray_extremity(P, x, omega);
  int surface = surface_point(P, g);
  SphereDir<Real> o;
  o.w[0] = (Real)omega.x;
  o.w[1] = (Real)omega.y;
  o.w[2] = (Real)omega.z;
  o.weight = (Real)dirs[w].w;
  o.surface = surface;
  split_coord<Real>(elevation_to_index(P, d.n1, x, omega, !surface), d.n1, &o.u1, &o.s1);
  if (surface) {
    Real tau[3];
    segment_depth<Real>(P, x, sub3(g, x), d.S, tau);
    double gr = mag3(g);
    for (int c = 0; c < 3; c++) o.ground[c] = exp_neg(tau[c]) * (Real)(P.brightness[c] / M_PI);
    o.tR = (Real)(mag3(sub3(g, x)) / P.R);
    split_coord<Real>(height_to_index(P, d.nE0, gr), d.nE0, &o.uE0, &o.sE0);
  } else {
    for (int c = 0; c < 3; c++) o.ground[c] = 0;
    o.tR = 0;
    o.uE0 = 0;
    o.sE0 = 0;
  }
  out[((long long)b * d.n0 + i) * d.P + w] = o;
}

// Point-scatter constants per (height i, sun elevation k): the coordinates
// of ray-scatter-forward (atmosphere.clj:203-222) at x = (r_i, 0, 0) with the
// sun at elevation k, and beta_c(x) (atmosphere.clj:42-47, 140-151), in FP64
// once here instead of in every thread of the point-scatter blocks.
template <class Real>
__device__ void point_row(const AtmoParams* params, const BuildDims& d, PointRow<Real>* out, int t, int b) {
  const AtmoParams& P = params[b];
  const int i = t / d.n2, k = t % d.n2;
  const double r = index_to_radius(P, d.n0, (double)i);
  const double ss = index_to_sin_sun_elevation(d.n2, (double)k);
  PointRow<Real> o;
  o.ss = ss;
  o.cs = sqrt(dmax(0.0, dsub(1.0, sqr(ss))));
  o.lz = (Real)sqrt(dmax(0.0, dsub(dsub(1.0, sqr(o.cs)), sqr(ss))));
  const double gA = r * ss / P.R;
  o.gA = ordinary_radii(P) ? (Real)gA : Real(0);
  split_coord<Real>(height_to_index(P, d.n0, r), d.n0, &o.u0, &o.s0);
  split_coord<Real>(sun_elevation_to_index(d.n2, mk3(r, 0, 0), mk3(ss, 0, 0)), d.n2, &o.u2, &o.s2);
  const double h = r - P.R;
  const double er = exp(-(h / P.ray_scale)), em = exp(-(h / P.mie_scale));
  for (int c = 0; c < 3; c++) {
    o.bR[c] = (Real)(P.ray_base[c] * er);
    o.bM[c] = (Real)(P.mie_base[c] * em);
  }
  out[(long long)b * d.n0 * d.n2 + t] = o;
}

// The world frame of the directions at x = (r, 0, 0), whatever r.
struct Frame {
  d3 n, o1, o2;
  __device__ Frame() : n(mk3(1, 0, 0)), o1(orthogonal(n)), o2(cross3(n, o1)) {}
  __device__ d3 world(const DirLocal& q) const { return to_world(n, o1, o2, q); }
};

// Surface radiance's tables that do not depend on the light's direction
// (k_surface.cu), in this order: nodes,
// elevation coordinates per (height, ring), and once for all atmospheres the
// rings and the directions.
template <class Real>
__device__ void surface_row(const AtmoParams* params, const BuildDims& d, const DirLocal* dirs,
                            const SetupBuffers<Real>& o, long long t, int b) {
  const AtmoParams& P = params[b];
  if (t < d.nE()) {
    const double r = index_to_radius(P, d.nE0, (double)(t / d.nE1));
    const double ss = index_to_sin_sun_elevation(d.nE1, (double)(t % d.nE1));
    const d3 x = mk3(r, 0, 0), l = mk3(ss, sqrt(dmax(0.0, 1 - sqr(ss))), 0);
    SurfRow<Real> row;
    split_coord<Real>(height_to_index(P, d.n0, mag3(x)), d.n0, &row.u0, &row.s0);
    split_coord<Real>(sun_elevation_to_index(d.n2, x, l), d.n2, &row.u2, &row.s2);
    row.lx = (Real)l.x;
    row.ly = (Real)l.y;
    o.erow[(long long)b * d.nE() + t] = row;
    return;
  }
  t -= d.nE();
  if (t < (long long)d.nE0 * d.Th) {
    const int i = (int)(t / d.Th), k = (int)(t - (long long)i * d.Th);
    const d3 x = mk3(index_to_radius(P, d.nE0, (double)i), 0, 0);
    Coord<Real> c;
    split_coord<Real>(elevation_to_index(P, d.n1, x, Frame().world(dirs[ring_start(dirs, d.Ph, d.Th, M_PI / 2, k)]), 1), d.n1, &c.u,
                      &c.s);
    o.half_rows[(long long)b * d.nE0 * d.Th + t] = c;
    return;
  }
  t -= (long long)d.nE0 * d.Th;
  if (b > 0) return;
  if (t <= d.Th) {
    HalfRing<Real> ring{};
    ring.w0 = ring_start(dirs, d.Ph, d.Th, M_PI / 2, (int)t);
    if (t < d.Th) {
      const double x0 = Frame().world(dirs[ring.w0]).x;
      ring.x0 = (Real)x0;
      ring.weight = (Real)(dirs[ring.w0].w * x0);
    }
    o.half_rings[t] = ring;
    return;
  }
  t -= d.Th + 1;
  if (t < d.Ph) o.half_y[t] = (Real)Frame().world(dirs[t]).y;
}

__host__ __device__ inline long long surface_row_items(const BuildDims& d) {
  // a build without iterations may ask for no directions (ray steps below 4)
  return d.nE() + (d.Th > 0 ? (long long)d.nE0 * d.Th + d.Th + 1 + d.Ph : 0);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

static inline dim3 grid1(long long n, int block, int B) { return dim3((unsigned)((n + block - 1) / block), B); }

// The set-up tables that need nothing but the parameters and the quadrature
// directions, in one launch: they are FP64 chains of 10 to 25 us each (small
// tables), and nine launches one after another held the iterations of a small
// build back by 150 of its 260 us, 162 with this launch (8x16x8x4 tables,
// FP32; 127 with what came later).  Blocks of one warp, so that what work
// there is spreads over the SMs' FP64 units.  Where the work is large (16
// atmospheres of 16x128x16x8) they take as long as they did apart, 1.9 ms with
// the maps and view rows, bound by FP64.
struct SetupParts {
  int blocks[kSetupParts];  // blocks of each part, 0 where it is not asked for
};

template <class Real>
__global__ void __launch_bounds__(32)
    k_setup_tables(const AtmoParams* params, BuildDims d, const DirLocal* dirs, const DirLocal* half_dirs,
                   SetupBuffers<Real> o, Vec4<Real>* T, Vec4<Real>* E0, SetupParts parts) {
  const int b = blockIdx.y, lane = threadIdx.x;
  int block = blockIdx.x, part = 0;
  while (block >= parts.blocks[part]) block -= parts.blocks[part++];
  const long long t = block * 32LL + lane;
  switch (part) {
    case kPartRings: {  // a warp a ring
      const int i = block / d.T;
      sphere_ring<Real>(params, d, dirs, o.rings, i, block - i * d.T, b, lane);
      break;
    }
    case kPartTransmittance:
      if (t < d.nT()) transmittance_node<Real>(params, d, T, t, b);
      break;
    case kPartBase:
      if (t < d.nE()) surface_base_node<Real>(params, d, E0, t, b);
      break;
    case kPartRows:
      if (t < d.rows()) row_info(params, d, o.rowinfo, t, b);
      break;
    case kPartRowMap:
      if (t < d.rows()) row_map<Real>(params, d, o.rowmap, t, b);
      break;
    case kPartPoints:
      if (t < d.n0 * d.n2) point_row<Real>(params, d, o.prow, (int)t, b);
      break;
    case kPartHeadings:
      // v.l of heading a as index_to_sun_direction forms it, for every atmosphere
      if (b == 0 && t < d.n3) o.hdvs[t] = dsub(dmul(2.0, (double)t / (d.n3 - 1)), 1.0);
      break;
    case kPartSurface:
      surface_row<Real>(params, d, half_dirs, o, t, b);
      break;
    case kPartDirections:
      if (t < (long long)(sizeof(Real) == 8 ? d.n0 : 1) * d.P)
        sphere_direction<Real>(params, d, dirs, o.dirs4, o.offsets, (int)(t / d.P), (int)(t % d.P), b);
      break;
    case kPartMapT:
      if (t < d.nT()) remap_T<Real>(params, d, o.remapT, t, b);
      break;
    case kPartMapE:
      if (t < d.nE()) remap_E<Real>(params, d, o.remapE, t, b);
      break;
  }
}

// The parts in `which` (bits 1 << kPart...).
template <class Real>
void launch_setup_tables(const AtmoParams* params, const BuildDims& d, const DirLocal* dirs, const DirLocal* half_dirs,
                         const SetupBuffers<Real>& o, Vec4<Real>* T, Vec4<Real>* E0, unsigned which, cudaStream_t st) {
  const long long items[kSetupParts] = {
      32LL * d.n0 * d.T, d.nT(), d.nE(), d.rows(), (long long)d.n0 * d.n2, d.n3, surface_row_items(d),
      (long long)(sizeof(Real) == 8 ? d.n0 : 1) * d.P, d.nT(), d.nE(), d.rows()};
  SetupParts parts;
  int blocks = 0;
  for (int p = 0; p < kSetupParts; p++) {
    // a build without iterations may ask for no sphere directions (sphere steps below 2): no rings
    parts.blocks[p] = which >> p & 1u ? (int)((items[p] + 31) / 32) : 0;
    blocks += parts.blocks[p];
  }
  if (blocks > 0)
    k_setup_tables<Real><<<dim3((unsigned)blocks, d.B), 32, 0, st>>>(params, d, dirs, half_dirs, o, T, E0, parts);
}

template <class Real>
void launch_node_maps(const AtmoParams* params, const BuildDims& d, const SetupBuffers<Real>& o, cudaStream_t st) {
  const int blk = 128;
  k_remap4<Real><<<grid1(d.n4(), blk, d.B), blk, 0, st>>>(d, o.rowinfo, o.prow, o.hdvs, o.angle, o.geom);
}

template <class Real>
void launch_view_rows(const AtmoParams* params, const BuildDims& d, const SetupBuffers<Real>& o, cudaStream_t st) {
  // one warp a block: a small build's samples spread over the SMs' FP64 units
  const int blk = 32;
  if (d.scan_rays)
    k_view_rows_scan<Real><<<grid1(d.rows(), blk / 32, d.B), blk, 0, st>>>(params, d, o.rowinfo, o.rows);
  else
    k_view_rows<Real><<<grid1(d.rows() * d.S, blk, d.B), blk, 0, st>>>(params, d, o.rowinfo, o.rows);
}

template <class Real>
void launch_sphere_dirs(const AtmoParams* params, const BuildDims& d, const DirLocal* dirs, SphereDir<Real>* out,
                        cudaStream_t st) {
  const int blk = 128;
  if (d.P > 0) k_sphere_setup<Real><<<grid1((long long)d.n0 * d.P, blk, d.B), blk, 0, st>>>(params, d, dirs, out);
}

#define SFSIM_INSTANTIATE(Real)                                                                                  \
  template void launch_setup_tables<Real>(const AtmoParams*, const BuildDims&, const DirLocal*, const DirLocal*, \
                                          const SetupBuffers<Real>&, Vec4<Real>*, Vec4<Real>*, unsigned,         \
                                          cudaStream_t);                                                         \
  template void launch_node_maps<Real>(const AtmoParams*, const BuildDims&, const SetupBuffers<Real>&,           \
                                       cudaStream_t);                                                            \
  template void launch_view_rows<Real>(const AtmoParams*, const BuildDims&, const SetupBuffers<Real>&,           \
                                       cudaStream_t);                                                            \
  template void launch_sphere_dirs<Real>(const AtmoParams*, const BuildDims&, const DirLocal*, SphereDir<Real>*, \
                                         cudaStream_t);

SFSIM_INSTANTIATE(float)
SFSIM_INSTANTIATE(double)

}  // namespace sfsim
