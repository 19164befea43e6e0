// k_point_scatter.cu -- point scatter J of the multiple-scattering iterations
// (atmosphere.clj:203-222), for the nodes of one (height i, sun elevation k)
// pair at a time.
//
// The sphere quadrature (sphere.clj:62-93) is a set of rings about x, which
// lies on the first axis.  All directions of a ring share everything but
// their azimuth: where they end, the ground's transmittance, and the height,
// elevation and sun-elevation coordinates of the dS lookup (x.l = r sin(k) for
// every node of the pair).  So dS collapses to one row along the sun-angle
// axis per ring, and a direction's lookup is linear in that row at its own
// omega.l.  The ground term is a linear lookup in the lowest row of the
// surface-radiance table (a ray that ends on the ground ends at height 0).
//
// One thread holds one elevation j and kHP pairs of headings; the two FP32
// lanes of every packed operation are two headings.  It walks the
// directions ring by ring, forms the direction's two phase weights (they
// depend on j and the direction only) once, and adds the interpolated rows of
// all its headings.  The first and last headings ask for v.l = -1 and 1, which
// clamps the light to the plane of x and v for every view
// (index-to-sun-direction, atmosphere.clj:375-384): their l is the same for
// all j, so the block interpolates their rows once per direction into shared
// memory and every thread adds them from there.
//
// What bounds it: the FMA pipe (packed operations take it for two cycles) and
// the shared-memory wavefronts together, about 70 and 60 % of a launch.  A
// heading and direction gathers 24 bytes of its ring's row (two channels'
// values and steps in one load, the third's in another) and 24 more of the
// ground's.  Production tables (32x255x32x8, 336 directions, 5 iterations):
// 98M wavefronts and 0.58 ms a launch, 3.18 ms for the build's five, 0.13 of
// them for the phases' distances |omega -+ v|, |omega -+ l| (PhaseCS::at), 0.10
// for the compensation of the sums; with 4-byte loads it was 160M and 3.49 ms.
// With a row per direction instead of per ring (gathered to HBM by a kernel of
// its own), the phases exchanged by shuffles and every heading walked, it was
// 7.08 ms.  The 16 atmospheres of a sweep (16x128x16x8) went from 11.8 to 5.0
// ms, the reference's tables (32x127x32x8, 71 directions) from 0.96 to 0.44.
#include <algorithm>
#include <type_traits>

#include "atmo_device.cuh"
#include "kernels.h"

namespace sfsim {

// A record of a row: the values of two channels and their steps to the next
// texel, value and step of the third.  With the Mie strength (first
// iteration) its two channels follow the first four, and its third the other
// two.  All of it is read in 8- and 16-byte loads, which take half the
// wavefronts of 4-byte ones where the lanes of each pair (2n, 2n + 1) read the
// same record, as neighbouring elevations mostly do, and no more where they do
// not.
template <bool FIRST>
__host__ __device__ constexpr int row_stride() {
  return FIRST ? 12 : 8;
}
constexpr int kGroundStride = 6;  // the same for the surface-radiance row

// Records of a ring row: a copy of texel 0, then the n3 texels, so that a
// coordinate that rounding pushed just below 0 reads texel 0; the last
// texel's step is 0.
__host__ __device__ constexpr int row_records(int n3) { return n3 + 1; }

// Shared-memory layout, in this order, each part 16-byte aligned.
struct PointLayout {
  unsigned dirs;    // [P][4] x1, x1, x2, x2
  unsigned edge;    // [P][8] HeadingPair of the first and last heading
  unsigned rings;   // [T] SphereRing
  unsigned rows;    // [T][n3 + 1][row_stride]
  unsigned etab;    // [nE1][kGroundStride]
  unsigned bytes;
};
template <class Real>
__host__ __device__ inline PointLayout point_layout(const BuildDims& d, bool first) {
  auto up = [](size_t x) { return (x + 15) & ~size_t(15); };
  PointLayout l;
  size_t o = 0;
  l.dirs = 0;
  o = up(o + sizeof(Real) * 4 * d.P);
  l.edge = (unsigned)o;
  o = up(o + sizeof(Real) * 8 * d.P);
  l.rings = (unsigned)o;
  o = up(o + sizeof(SphereRing<Real>) * d.T);
  l.rows = (unsigned)o;
  o = up(o + sizeof(Real) * d.T * row_records(d.n3) * (first ? row_stride<true>() : row_stride<false>()));
  l.etab = (unsigned)o;
  o = up(o + sizeof(Real) * kGroundStride * d.nE1);
  l.bytes = (unsigned)o;
  return l;
}

// Where a record keeps channel c's value (c < 3: dS, c >= 3: the Mie
// strength), and its step.
template <bool FIRST>
__device__ __forceinline__ constexpr int value_at(int c) {
  return c < 2 ? c : c == 2 ? (FIRST ? 8 : 4) : c < 5 ? c + 1 : 10;
}
template <bool FIRST>
__device__ __forceinline__ constexpr int step_at(int c) {
  return value_at<FIRST>(c) + (c == 2 || c == 5 ? 1 : 2);
}

// Radiances of a pair of headings a and b: the first two channels of each,
// and the third of both.
template <class Real>
struct HeadingPair {
  V2<Real> a, b, z;
};

constexpr int kPointThreads = 128;
constexpr int kPointSlices = 8;  // at most
// Directions summed plainly at most, between steps of the compensated totals:
// production 3.27 / 3.18 / 3.14 ms (of 3.08 with plain totals) with 8 / 16 / 32;
// the sums' spread is the same with 8 and 16 (4.9e-8 of a sum of 1172
// directions; plain totals 7.6e-8, 32 5.6e-8).
constexpr int kPointRun = 16;

// Blocks per SM the registers are limited for.  Three heading pairs measured
// 3.11 / 2.96 / 3.04 / 3.25 ms of a production build (5 launches) at 2 / 3 /
// 4 / 5 blocks.
template <class Real, int HP>
constexpr int point_min_blocks() {
  return sizeof(Real) == 8 ? 2 : HP == 3 ? 3 : HP == 2 ? 4 : 5;
}

template <class Real, int HP, bool FIRST>
__global__ void __launch_bounds__(kPointThreads, point_min_blocks<Real, HP>())
    k_point_scatter(const AtmoParams* params, BuildDims d, PointLayout lay, const RowInfo* rowinfo,
                    const SphereRing<Real>* rings, const Real* dirs4, const Real* offsets,
                    const PointRow<Real>* prow, const CellGeom<Real>* geom, const Vec4<Real>* dS, const Vec4<Real>* Mt, const Vec4<Real>* dE,
                    Vec4<Real>* J, int groups, int chunks, int slices) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using R2 = V2<Real>;
  constexpr int KS = row_stride<FIRST>();
  const int tid = threadIdx.x, nt = blockDim.x;
  const int b = blockIdx.y;
  const int ik = blockIdx.x / chunks, chunk = blockIdx.x - ik * chunks;
  const int i = ik / d.n2, k = ik - i * d.n2;
  const AtmoParams& P = params[b];
  const PointRow<Real> pk = prow[((long long)b * d.n0 + i) * d.n2 + k];
  Real* sdirs = reinterpret_cast<Real*>(smem_raw + lay.dirs);
  Real* sedge = reinterpret_cast<Real*>(smem_raw + lay.edge);
  SphereRing<Real>* sring = reinterpret_cast<SphereRing<Real>*>(smem_raw + lay.rings);
  Real* srows = reinterpret_cast<Real*>(smem_raw + lay.rows);
  Real* setab = reinterpret_cast<Real*>(smem_raw + lay.etab);
  constexpr int ES = kGroundStride;
  const int nrec = row_records(d.n3);
  const long long base4 = (long long)b * d.n4();

  // ring records, directions, the rows' texels and the dE row
  {
    const SphereRing<Real>* src = rings + ((long long)b * d.n0 + i) * d.T;
    for (int t = tid; t < (int)(sizeof(SphereRing<Real>) / 16) * d.T; t += nt)
      reinterpret_cast<int4*>(sring)[t] = reinterpret_cast<const int4*>(src)[t];
    for (int t = tid; t < (int)(sizeof(Real) * 4 / 16) * d.P; t += nt)
      reinterpret_cast<int4*>(sdirs)[t] = reinterpret_cast<const int4*>(dirs4)[t];
    for (int t = tid; t < d.T * d.n3; t += nt) {
      const int r = t / d.n3, a = t - r * d.n3;
      const int u1 = src[r].u1;
      const Real s1 = src[r].s1;
      Real v[3], vm[3];
      gather_row_texel(dS + base4, d, pk.u0, pk.s0, u1, s1, pk.u2, pk.s2, a, v);
      if (FIRST) gather_row_texel(Mt + base4, d, pk.u0, pk.s0, u1, s1, pk.u2, pk.s2, a, vm);
      Real* o = srows + (r * nrec + a + 1) * KS;
#pragma unroll
      for (int c = 0; c < (FIRST ? 6 : 3); c++) {
        const Real x = c < 3 ? v[c % 3] : vm[c % 3];
        o[value_at<FIRST>(c)] = x;
        if (a == 0) {
          o[value_at<FIRST>(c) - KS] = x;
          o[step_at<FIRST>(c) - KS] = Real(0);
        }
      }
    }
    const Vec4<Real>* e = dE + b * d.nE();
    for (int t = tid; t < d.nE1; t += nt) {
      Real A[3], B[3];
      ld3(e, t, A);
      ld3(e, upper_index(t, d.nE1), B);
#pragma unroll
      for (int c = 0; c < 3; c++) {
        setab[t * ES + value_at<false>(c)] = A[c];
        setab[t * ES + step_at<false>(c)] = B[c] - A[c];
      }
    }
  }
  __syncthreads();
  for (int t = tid; t < d.T * d.n3; t += nt) {
    const int r = t / d.n3, a = t - r * d.n3;
    Real* o = srows + (r * nrec + a + 1) * KS;
#pragma unroll
    for (int c = 0; c < (FIRST ? 6 : 3); c++)
      o[step_at<FIRST>(c)] = a < d.n3 - 1 ? o[KS + value_at<FIRST>(c)] - o[value_at<FIRST>(c)] : Real(0);
  }
  __syncthreads();

  const PhaseCS<Real> phR(Bulk<Real>::phase_ray(P)), phM(Bulk<Real>::phase_mie(P));
  // Rayleigh's phase as the reference has it, g = 0, is k (1 + mu^2)
  const bool flat = phR.b == Real(0);
  const Real flatR = phR(Real(0));
  const Real scale3 = Real(0.5) * Real(d.n3 - 1);
  const Real scaleE = Bulk<Real>::sun_scale_E(d);
  const unsigned kstride = KS * sizeof(Real), estride = ES * sizeof(Real);
  const unsigned ebase = lookup_base<Real>(lay.etab, estride);
  const Real log2e = Real(1.4426950408889634);
  const Real zA = fma(Real(-3) * log2e, pk.gA, Real(-0.6 * 1.4426950408889634 + Bulk<Real>::kExp2Shift));
  const Real lx = (Real)pk.ss;
  // the light reaching x from direction (x0, x1, x2) of a ring, for the two
  // light directions (lx, ly, lz) of a pair: dS along the ring's row and, for
  // rings that end on the ground, the ground's radiance
  auto incoming = [&](auto ground, const SphereRing<Real>& rc, unsigned rbase, R2 c0, R2 x1, R2 x2, R2 ly, R2 lz,
                      Real off, HeadingPair<Real>& X) {
    const R2 mu = fma2(x1, ly, fma2(x2, lz, c0));  // omega . l
    // the sun-angle coordinate; |mu| <= 1 up to rounding, so its floor lies in
    // [-1, n3 - 1], whose records give the clamped interpolation
    unsigned oa, ob;
    const R2 s = lookup(fma2(dup(scale3), mu, dup(scale3)), rbase, rbase, kstride, oa, ob);
    const Real* ra = reinterpret_cast<const Real*>(smem_raw + oa);
    const Real* rb = reinterpret_cast<const Real*>(smem_raw + ob);
    R2 v, step, third;
    ld_pairs(ra, v, step);
    X.a = fma2(step, dup(s.x), v);
    ld_pairs(rb, v, step);
    X.b = fma2(step, dup(s.y), v);
    if (FIRST) {
      // |omega -+ l|^2 for the phase of the light
      const Real dx = fma(phM.s, lx, rc.x0);
      const R2 dy = fma2(dup(phM.s), ly, x1), dz = fma2(dup(phM.s), lz, x2);
      const R2 ph = phM.at(mu, fma2(dy, dy, fma2(dz, dz, dup(dx * dx))));
      R2 thirdm;
      ld_pairs(ra + 4, v, step);
      X.a = fma2(fma2(step, dup(s.x), v), dup(ph.x), X.a);
      ld_pairs(rb + 4, v, step);
      X.b = fma2(fma2(step, dup(s.y), v), dup(ph.y), X.b);
      ld_pairs(ra + 8, third, thirdm);
      X.z.x = fma(fma(thirdm.y, s.x, thirdm.x), ph.x, fma(third.y, s.x, third.x));
      ld_pairs(rb + 8, third, thirdm);
      X.z.y = fma(fma(thirdm.y, s.y, thirdm.x), ph.y, fma(third.y, s.y, third.x));
    } else {
      third = *reinterpret_cast<const R2*>(ra + 4);
      X.z.x = fma(third.y, s.x, third.x);
      third = *reinterpret_cast<const R2*>(rb + 4);
      X.z.y = fma(third.y, s.y, third.x);
    }
    if (decltype(ground)::value) {
      // the ground point's sin of the sun elevation, g.l / |g| = gA + tR (omega . l)
      // and its coordinate (1 - exp(-3 sin - 0.6)) / (1 - exp(-3.6)) (nE1 - 1),
      // at least 0; the sine is at most 1, as the point is on the ground
      // (sphere_ring and point_row see to it where the radii are no ordinary numbers)
      const R2 z = fma2(dup(Real(-3) * log2e * rc.tR), mu, dup(zA));
      const R2 ex = mk2(Bulk<Real>::exp2(z.x), Bulk<Real>::exp2(z.y));
      R2 ie = fma2(dup(-scaleE), ex, dup(scaleE));
      ie = mk2(fmax(ie.x, Real(0)), fmax(ie.y, Real(0)));
      const R2 se = lookup(ie, ebase, ebase, estride, oa, ob);
      const R2* ea = reinterpret_cast<const R2*>(smem_raw + oa);
      const R2* eb = reinterpret_cast<const R2*>(smem_raw + ob);
      const R2 g = mk2(rc.ground[0], rc.ground[1]);
      X.a = fma2(g, fma2(ea[1], dup(se.x), ea[0]), X.a);
      X.b = fma2(g, fma2(eb[1], dup(se.y), eb[0]), X.b);
      const R2 ta = ea[2], tb = eb[2];
      X.z = fma2(dup(rc.ground[2]), mk2(fma(ta.y, se.x, ta.x), fma(tb.y, se.y, tb.x)), X.z);
      if constexpr (std::is_same<Real, double>::value) {
        // the FP64 build's ground point is off height 0 by its rounding, as
        // the reference's is: the next height's row has that weight
        if (off != 0.0) {
          const Vec4<double>* e0 = dE + b * d.nE();
          const Vec4<double>* e1 = e0 + d.nE1;
          const int ia = (int)ie.x, ib = (int)ie.y;
          double A[3], B[3], C[3], D[3];
          auto above = [&](int u, double s, double (&o)[3]) {  // row 1 less row 0
            const int v = upper_index(u, d.nE1);
            ld3(e1, u, A), ld3(e1, v, B), ld3(e0, u, C), ld3(e0, v, D);
#pragma unroll
            for (int c = 0; c < 3; c++) o[c] = (A[c] - C[c]) * (1.0 - s) + (B[c] - D[c]) * s;
          };
          double ya[3], yb[3];
          above(ia, se.x, ya);
          above(ib, se.y, yb);
          const R2 go = mk2(rc.ground[0] * off, rc.ground[1] * off);
          X.a = fma2(go, mk2(ya[0], ya[1]), X.a);
          X.b = fma2(go, mk2(yb[0], yb[1]), X.b);
          X.z = fma2(dup(rc.ground[2] * off), mk2(ya[2], yb[2]), X.z);
        }
      }
    }
  };
  // the height coordinate of direction w's ground point (FP64 builds; 0 but for rounding)
  auto offset = [&](int w) -> Real {
    if constexpr (std::is_same<Real, double>::value)
      return offsets[((long long)b * d.n0 + i) * d.P + w];
    else
      return 0;
  };
  auto ring_base = [&](int r) { return lookup_base<Real>(lay.rows + (unsigned)(r * nrec + 1) * kstride, kstride); };

  // the first and last headings' rows at every direction
  {
    const R2 ly = mk2((Real)-pk.cs, (Real)pk.cs), lz = dup(pk.lz);
    for (int r = 0; r < d.T; r++) {
      const SphereRing<Real>& rc = sring[r];
      const unsigned rbase = ring_base(r);
      for (int m = tid; m < rc.n; m += nt) {
        const Real* x = sdirs + 4 * (rc.w0 + m);
        HeadingPair<Real> X;
        if (rc.surface)
          incoming(std::true_type{}, rc, rbase, dup(rc.x0 * lx), dup(x[0]), dup(x[2]), ly, lz, offset(rc.w0 + m), X);
        else
          incoming(std::false_type{}, rc, rbase, dup(rc.x0 * lx), dup(x[0]), dup(x[2]), ly, lz, offset(rc.w0 + m), X);
        R2* o = reinterpret_cast<R2*>(sedge + 8 * (rc.w0 + m));
        o[0] = X.a, o[1] = X.b, o[2] = X.z;
      }
    }
  }
  __syncthreads();

  // this thread's elevation and headings; a thread past the last item repeats it and stores nothing
  const int items = d.n1 * groups;
  // the directions of every ring go to `slices` threads an item in turn (then all items are in one block)
  const int slice = slices > 1 ? tid / items : 0;
  const int item_raw = slices > 1 ? tid - slice * items : chunk * nt + tid;
  const bool valid = item_raw < items && slice < slices;
  const int item = valid ? item_raw : items - 1;
  const int grp = item / d.n1, j = item - grp * d.n1;
  const int a0 = 1 + grp * 2 * HP;  // its headings a0 .. a0 + 2 HP - 1, those below n3 - 1
  const long long node0 = base4 + idx4(d, i, j, k, 0);
  Real sv, cv;
  {
    const RowR<Real> rw = row_r<Real>(rowinfo[(long long)b * d.rows() + (long long)i * d.n1 + j]);
    sv = rw.sv, cv = rw.cv;
  }
  R2 ly[HP], lz[HP];
#pragma unroll
  for (int h = 0; h < HP; h++) {
    const CellGeom<Real> ga = geom[node0 + min(a0 + 2 * h, d.n3 - 1)];
    const CellGeom<Real> gb = geom[node0 + min(a0 + 2 * h + 1, d.n3 - 1)];
    ly[h] = mk2(ga.ly, gb.ly);
    lz[h] = mk2(ga.lz, gb.lz);
  }
  // Compensated sums over the directions (pair HP: the first and last
  // heading): runs of up to kPointRun directions are summed plainly, and each
  // run starts from what the total lost when it took the last one.
  HeadingPair<Real> tot[HP + 1], run[HP + 1];
  const HeadingPair<Real> none{dup(Real(0)), dup(Real(0)), dup(Real(0))};
#pragma unroll
  for (int h = 0; h <= HP; h++) tot[h] = run[h] = none;
  auto flush = [&]() {
    auto take = [](R2& t, R2& x) {
      const R2 n = add2(t, x);
      x = sub2(x, sub2(n, t));
      t = n;
    };
#pragma unroll
    for (int h = 0; h <= HP; h++) {
      take(tot[h].a, run[h].a);
      take(tot[h].b, run[h].b);
      take(tot[h].z, run[h].z);
    }
  };

  const int shift = __ffs(slices) - 1;
  int pending = 0;  // directions in the run
  for (int r = 0; r < d.T; r++) {
    const SphereRing<Real>& rc = sring[r];
    const unsigned rbase = ring_base(r);
    const R2 c0 = dup(rc.x0 * lx);
    const Real mv0 = sv * rc.x0, dv = fma(phM.s, sv, rc.x0), dv2 = dv * dv, cvs = phM.s * cv;
    const int n = rc.n;
    const Real* x = sdirs + 4 * (rc.w0 + slice);
    const Real* e = sedge + 8 * (rc.w0 + slice);
    // beta_c(x) (atmosphere.clj:42-47, 140-151) times the ring's weight
    Real bR[3], bM[3];
#pragma unroll
    for (int c = 0; c < 3; c++) bR[c] = rc.weight * pk.bR[c], bM[c] = rc.weight * pk.bM[c];
    auto add = [](HeadingPair<Real>& t, R2 w, Real wz, const HeadingPair<Real>& X) {
      t.a = fma2(w, X.a, t.a);
      t.b = fma2(w, X.b, t.b);
      t.z = fma2(dup(wz), X.z, t.z);
    };
    auto walk = [&](auto ground) {
      for (int m0 = slice; m0 < n; m0 += kPointRun * slices) {
        const int len = min(kPointRun, (n - m0 + slices - 1 + slice) >> shift);  // the slices' longest
        if (pending + len > kPointRun) {
          flush();
          pending = 0;
        }
        pending += len;
        const int m1 = min(n, m0 + kPointRun * slices);
        for (int m = m0; m < m1; m += slices, x += 4 * slices, e += 8 * slices) {
          R2 x1, x2;
          ld_pairs(x, x1, x2);
          const Real mv = fma(cv, x1.x, mv0);
          Real fR = flatR * fma(mv, mv, Real(1));
          if (!flat) fR = phR(mv);
          const Real dy = x1.x + cvs;  // |omega -+ v|^2 for the phase of the view
          const Real fM = phM.at(mv, fma(dy, dy, fma(x2.x, x2.x, dv2)));
          const R2 w = fma2(mk2(bM[0], bM[1]), dup(fM), mul2(mk2(bR[0], bR[1]), dup(fR)));
          const Real wz = fma(bM[2], fM, bR[2] * fR);
#pragma unroll
          for (int h = 0; h < HP; h++) {
            HeadingPair<Real> X;
            incoming(ground, rc, rbase, c0, x1, x2, ly[h], lz[h], offset(rc.w0 + m), X);
            add(run[h], w, wz, X);
          }
          HeadingPair<Real> X;
          ld_pairs(e, X.a, X.b);
          X.z = *reinterpret_cast<const R2*>(e + 4);
          add(run[HP], w, wz, X);
        }
      }
    };
    if (rc.surface)
      walk(std::true_type{});
    else
      walk(std::false_type{});
  }
  flush();
  if (slices > 1) {
    // the slices' sums, in order
    HeadingPair<Real>* sums = reinterpret_cast<HeadingPair<Real>*>(smem_raw);
    __syncthreads();
    if (valid && slice > 0) {
#pragma unroll
      for (int h = 0; h <= HP; h++) {
        HeadingPair<Real>* o = sums + 2 * ((slice - 1) * (HP + 1) + h) * items + item;
        o[0] = tot[h];
        o[items] = run[h];
      }
    }
    __syncthreads();
    if (slice == 0) {
      auto plus = [](HeadingPair<Real>& x, const HeadingPair<Real>& y) {
        x.a = add2(x.a, y.a);
        x.b = add2(x.b, y.b);
        x.z = add2(x.z, y.z);
      };
      for (int q = 0; q < (slices - 1); q++) {
        const HeadingPair<Real>* o = sums + 2 * q * (HP + 1) * items + item;
#pragma unroll
        for (int h = 0; h <= HP; h++) plus(run[h], o[2 * h * items]);
        flush();
#pragma unroll
        for (int h = 0; h <= HP; h++) plus(run[h], o[(2 * h + 1) * items]);
      }
      flush();
    }
  }
  if (!valid || slice > 0) return;
  auto put = [&](int at, R2 xy, Real z) {
    Vec4<Real> o;
    o.x = xy.x;
    o.y = xy.y;
    o.z = z;
    o.w = 0;
    J[node0 + at] = o;
  };
#pragma unroll
  for (int h = 0; h < HP; h++) {
    const int a = a0 + 2 * h;
    if (a < d.n3 - 1) put(a, tot[h].a, tot[h].z.x);
    if (a + 1 < d.n3 - 1) put(a + 1, tot[h].b, tot[h].z.y);
  }
  if (grp == 0) {
    put(0, tot[HP].a, tot[HP].z.x);
    put(d.n3 - 1, tot[HP].b, tot[HP].z.y);
  }
}

// 40 bytes a direction (FP32; 76 in FP64), two rows of n3 + 2 RGB texels
// each, and the surface-radiance table, with room for 16 directions more.
// The tables above are smaller (a row per ring, not per direction), so a
// configuration within this limit always fits.
template <class Real>
size_t point_scatter_capacity(const BuildDims& d) {
  const size_t n = (size_t)d.P + 16;
  return ((n * (9 * sizeof(Real) + sizeof(int)) + 15) & ~size_t(15)) +
         sizeof(Real) * 3 * (n * (d.n3 + 2) * 2 + d.nE());
}
template size_t point_scatter_capacity<float>(const BuildDims&);
template size_t point_scatter_capacity<double>(const BuildDims&);

template <class Real>
int launch_point_scatter(const AtmoParams* params, const BuildDims& d, const RowInfo* rowinfo,
                         const SphereRing<Real>* rings, const Real* dirs4, const Real* offsets,
                         const PointRow<Real>* prow, const CellGeom<Real>* geom, const Vec4<Real>* dS, const Vec4<Real>* mie, const Vec4<Real>* dE,
                         Vec4<Real>* J, cudaStream_t st) {
  const bool first = mie != nullptr;
  PointLayout lay = point_layout<Real>(d, first);
  const int inner = d.n3 - 2;
  int hp = sizeof(Real) == 8 ? 1 : inner > 4 ? 3 : inner > 2 ? 2 : 1;
  const int groups = inner > 0 ? (inner + 2 * hp - 1) / (2 * hp) : 1;
  const int items = d.n1 * groups;
  const int chunks = (items + kPointThreads - 1) / kPointThreads;
  int block = ((items + chunks - 1) / chunks + 31) / 32 * 32;
  // Few elevations leave a warp's lanes unused, and in a small build most of
  // the warps that an SM holds: then several threads share an item's
  // directions.  16 elevations, 4 headings, 8 heights and sun elevations, two
  // iterations: FP32 46 us with 1 thread an item, 31 with 4, 27 with 8; FP64
  // 885, 305 and 219.  What counts is one atmosphere's size: the slices order
  // the sums, and an atmosphere of a batch has the bits of its own build.
  const bool few = (long long)d.n0 * d.n2 * chunks * (block / 32) < 1824;  // 12 warps an SM
  int slices = 1;
  while (chunks == 1 && 2 * slices * items <= kPointThreads && slices < kPointSlices && (few || slices * items < 32))
    slices *= 2;
  if (slices > 1) {
    block = (slices * items + 31) / 32 * 32;
    lay.bytes = std::max<unsigned>(lay.bytes, sizeof(HeadingPair<Real>) * 2 * (hp + 1) * items * (slices - 1));
  }
  const dim3 grid((unsigned)(d.n0 * d.n2 * chunks), d.B);
  auto go = [&](auto kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.bytes) != cudaSuccess)
      return -1;
    kernel<<<grid, block, lay.bytes, st>>>(params, d, lay, rowinfo, rings, dirs4, offsets, prow, geom, dS, mie,
                                           dE, J, groups, chunks, slices);
    return 0;
  };
  if constexpr (std::is_same<Real, float>::value) {
    if (hp == 3) return first ? go(k_point_scatter<Real, 3, true>) : go(k_point_scatter<Real, 3, false>);
    if (hp == 2) return first ? go(k_point_scatter<Real, 2, true>) : go(k_point_scatter<Real, 2, false>);
  }
  return first ? go(k_point_scatter<Real, 1, true>) : go(k_point_scatter<Real, 1, false>);
}

template int launch_point_scatter<float>(const AtmoParams*, const BuildDims&, const RowInfo*, const SphereRing<float>*,
                                         const float*, const float*, const PointRow<float>*, const CellGeom<float>*,
                                         const Vec4<float>*, const Vec4<float>*, const Vec4<float>*, Vec4<float>*,
                                         cudaStream_t);
template int launch_point_scatter<double>(const AtmoParams*, const BuildDims&, const RowInfo*,
                                          const SphereRing<double>*, const double*, const double*, const PointRow<double>*,
                                          const CellGeom<double>*, const Vec4<double>*, const Vec4<double>*,
                                          const Vec4<double>*, Vec4<double>*, cudaStream_t);

}  // namespace sfsim
