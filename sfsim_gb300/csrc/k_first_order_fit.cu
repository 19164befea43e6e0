// k_first_order_fit.cu -- the FP32 first order with fitted sun rays:
// first-order Rayleigh ray scatter and Mie strength (atmosphere_lut.clj:68-78
// with atmosphere.clj:154-200) of builds large enough that a table of the sun
// rays' optical depths pays (k_first_order.cu integrates them otherwise).
//
// The S-sample midpoint sums of a sun ray depend only on where it starts: q =
// |p_s|^2 - R^2 and its exit distance d from the atmosphere.  For one q, d runs
// from the zenith's dmin to the distance dmax of the ray that grazes the
// ground, and the log2 of the two mean densities along the ray (sum / S) is a
// smooth function of d, through the horizontal as well.  k_sun_fit evaluates
// the sums for kFitRows values of sqrt(q / q_top), at six Chebyshev nodes in
// each of `segs` equal segments of [dmin, dmax], and stores the quintics
// through them.  A ray sample of a view row interpolates the coefficients of
// its two neighbouring rows once, for all the cells of the row; a cell then
// evaluates one quintic for both components and multiplies 2^F by d.
//
// Accuracy (numpy model of this scheme, FP32 storage and evaluation, against
// the sums in FP64; Earth, the reference's 35 km atmosphere, the sweep's
// extremes, 25 random atmospheres, 13 to 512 steps): transmittance within
// 8e-7, optical depth within 3e-6 relative.  Measured first-order tables
// against FP64 builds, 2-norm: 1.1e-7 (Rayleigh) and 1.1e-7 to 1.8e-7 (Mie);
// bilinear tables of 6.3M nodes 0.9e-7 to 3.1e-7, integrating every sun ray
// 0.9e-7 to 1.1e-7 and 1.1e-7 to 1.7e-7.  Largest relative error, at nodes a
// millionth as bright as the brightest: 1.5e-5 to 5.4e-5, against 1.0e-5 to
// 3.2e-5 and 1.1e-5 to 3.3e-5.  The number of segments follows
// the width of the density peak at a grazing ray's perigee, sqrt(2 R h) for
// the smaller scale height h, and the steps must resolve that peak
// (sun_fit_segments).
//
// Mapping: one block per view row, one lane per cell (sun elevation k, sun
// heading a), all lanes of a warp at the same sample, so what depends on the
// sample is a broadcast from shared memory and no sum crosses lanes.  Rows
// with few cells split their samples over several groups of warps.
//
// What bounds it: latency and instruction issue (54% issued; two samples at
// a time keep two dependent chains per lane in flight).  Production tables (2.67e8
// pairs, 71% lit): 0.81 ms with the fits, 2.49 ms with bilinear tables of 6.3M
// nodes (80 MB, their gathers bound by L1; 0.25 ms to fill, here 0.03); the
// reference's tables 0.37 against 1.49 ms, 16 atmospheres of a sweep 2.2
// against 9.3.  (With descending rays placed by d itself: 0.73 ms, and three
// times the error at the darkest nodes; one sample at a time 1.0 ms; three
// blocks per SM at 128 samples a batch within 1%.)
#include "atmo_device.cuh"
#include "kernels.h"
#include "sun_fit.cuh"

namespace sfsim {

size_t sun_fit_bytes(int segs) { return sizeof(float2) * kFitNodes * (size_t)segs * kFitRows; }

// Coefficients of the polynomial in t in [-1/2, 1/2] (segments, from the
// segment's middle) through values at the Chebyshev nodes: the inverse of
// their Vandermonde matrix.
struct FitBasis {
  double inv[kFitNodes][kFitNodes];  // [power][node]
  float node[kFitNodes];             // t + 1/2
};

// One block: kFitPerBlock heights, one thread per (height, segment, node).
constexpr int kFitPerBlock = 4;
__global__ void k_sun_fit(const AtmoParams* params, int first, int S, int segs, FitBasis basis, float2* out) {
  extern __shared__ float2 F[];  // [height][segment][node]
  const int b = blockIdx.y;
  const AtmoParams& P = params[atmosphere_of(params, first, b)];
  const int per = segs * kFitNodes;
  for (int t = threadIdx.x; t < kFitPerBlock * per; t += blockDim.x) {
    const int h = t / per, e = t - h * per, g = e / kFitNodes, n = e - g * kFitNodes;
    const int row = blockIdx.x * kFitPerBlock + h;
    const float x = (float)row / (float)(kFitRows - 1);
    const float q = x * x * P.f_Hh2;
    const FitRange f = fit_range(P, q);
    const float d = fmaf((g + basis.node[n]) / (float)segs, f.range, f.dmin);
    const float bp = d > 0.0f ? (f.cq - d * d) / (2.0f * d) : 0.0f;
    constexpr int NP = Bulk<float>::kSunNP;
    float hc[NP];
#pragma unroll
    for (int c = 0; c < NP; c++) hc[c] = Bulk<float>::hpr(P)[c];
    float sr, smie;
    sun_sums<float, NP>(q, bp, d / (float)S, S, hc, Bulk<float>::alpha(P), Bulk<float>::beta(P),
                        Bulk<float>::hratio(P), sr, smie);
    // 2^-126 keeps the logarithm finite where the density underflows
    const float inv_s = 1.0f / (float)S;
    F[t] = make_float2(log2f(fmaxf(sr * inv_s, 1.17549435e-38f)), log2f(fmaxf(smie * inv_s, 1.17549435e-38f)));
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kFitPerBlock * per; t += blockDim.x) {
    const int m = t % kFitNodes;
    const float2* v = F + (t - m);
    double r = 0, e = 0;
#pragma unroll
    for (int n = 0; n < kFitNodes; n++) {
      r += basis.inv[m][n] * (double)v[n].x;
      e += basis.inv[m][n] * (double)v[n].y;
    }
    out[((size_t)b * kFitRows + (size_t)blockIdx.x * kFitPerBlock) * per + t] = make_float2((float)r, (float)e);
  }
}

static_assert(sizeof(float2) * kFitNodes == 48, "a segment is 48 bytes, three 16-byte words");
static FitBasis fit_basis() {
  FitBasis f;
  double t[kFitNodes], a[kFitNodes][2 * kFitNodes];
  const double pi = 3.14159265358979323846;
  for (int n = 0; n < kFitNodes; n++) {
    t[n] = -cos(pi * (n + 0.5) / kFitNodes);
    f.node[n] = (float)(0.5 * (t[n] + 1.0));
    t[n] = (double)f.node[n] - 0.5;
  }
  // Gauss-Jordan on the Vandermonde matrix
  for (int n = 0; n < kFitNodes; n++) {
    double p = 1.0;
    for (int m = 0; m < kFitNodes; m++, p *= t[n]) a[n][m] = p;
    for (int m = 0; m < kFitNodes; m++) a[n][kFitNodes + m] = n == m ? 1.0 : 0.0;
  }
  for (int c = 0; c < kFitNodes; c++) {
    int piv = c;
    for (int r = c + 1; r < kFitNodes; r++)
      if (fabs(a[r][c]) > fabs(a[piv][c])) piv = r;
    for (int m = 0; m < 2 * kFitNodes; m++) {
      const double s = a[c][m];
      a[c][m] = a[piv][m];
      a[piv][m] = s;
    }
    const double d = a[c][c];
    for (int m = 0; m < 2 * kFitNodes; m++) a[c][m] /= d;
    for (int r = 0; r < kFitNodes; r++) {
      if (r == c) continue;
      const double s = a[r][c];
      for (int m = 0; m < 2 * kFitNodes; m++) a[r][m] -= s * a[c][m];
    }
  }
  for (int m = 0; m < kFitNodes; m++)
    for (int n = 0; n < kFitNodes; n++) f.inv[m][n] = a[m][kFitNodes + n];
  return f;
}

void launch_sun_fit(const AtmoParams* params, const BuildDims& d, unsigned char* table, cudaStream_t st, int first) {
  static const FitBasis basis = fit_basis();
  const int per = kFitPerBlock * d.sun_segs * kFitNodes;
  const int block = per < 512 ? (per + 31) / 32 * 32 : 512;
  k_sun_fit<<<dim3(kFitRows / kFitPerBlock, d.B), block, sizeof(float2) * per, st>>>(params, first, d.S, d.sun_segs,
                                                                                    basis, reinterpret_cast<float2*>(table));
}

// What the cells share of two consecutive ray samples, side by side.  The sun
// is above a sample's horizon for p_s.l >= lit, below it for p_s.l <= dark;
// between the two FP32 cannot decide (p_s.l carries about 1 m of rounding).
struct alignas(16) FitPair {
  float2 us, cq;      // (s + 1/2) / S; cq = top^2 - r^2
  float2 dark, lit;
  float2 q, rho;      // rho = sqrt(q)
  float2 scale, off;  // 1 / range and -dmin / range of the exit distances
  float2 er, em;      // exp(-h/H)
  float2 tau[3];      // -log2(e) tau(x, p_s)
  float2 frac;        // sqrt(q / q_top) in the table: fraction and row
  int2 row;
  int2 pad;
};

// Samples whose coefficients are in shared memory at a time: 24.6 KB at 8 segments.
constexpr int kFitBatch = 64 * 8;  // segments x samples
constexpr int kFitThreads = 256;

static int fit_batch(const BuildDims& d) {
  const int n = d.sun_segs < kFitBatch / 2 ? (kFitBatch / d.sun_segs) & ~1 : 2;  // whole pairs
  return d.S < n ? (d.S + 1) & ~1 : n;
}

// Cells a pass covers and the groups of warps that share their samples.
static void fit_shape(int ncell, int* cells, int* groups) {
  *cells = ncell < kFitThreads ? (ncell + 31) / 32 * 32 : kFitThreads;
  *groups = kFitThreads / *cells;
}

size_t first_order_fit_smem(const BuildDims& d) {
  int cells, groups;
  fit_shape(d.n2 * d.n3, &cells, &groups);
  const int batch = fit_batch(d);
  const size_t coef = sizeof(float2) * kFitNodes * (size_t)d.sun_segs * batch;
  const size_t sums = sizeof(float) * 12 * (size_t)cells * groups;
  return (sizeof(CellGeom<float>) + sizeof(double2)) * (size_t)d.n2 * d.n3 + sizeof(FitPair) * (batch / 2) + (coef > sums ? coef : sums);
}

__global__ void __launch_bounds__(kFitThreads, 4)
    k_first_order_fit(const AtmoParams* params, BuildDims d, int first, int cells, int groups, int batch, const RowInfo* rowinfo,
                      const RowSample<float>* rows, const PointRow<float>* prow, const double* hdvs,
                      const float4* table, Vec4<float>* rayleigh, Vec4<float>* mie) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int b = atmosphere_of(params, first, blockIdx.y), tid = threadIdx.x, nt = blockDim.x;
  const long long row = blockIdx.x, nrows = d.rows();
  const AtmoParams& P = params[b];
  const int ncell = d.n2 * d.n3;
  const unsigned segs = d.sun_segs;
  const RowInfo& ri = rowinfo[b * nrows + row];
  CellGeom<float>* cg = reinterpret_cast<CellGeom<float>*>(smem_raw);
  double2* cl = reinterpret_cast<double2*>(cg + ncell);  // second and third component of the lights
  FitPair* smp = reinterpret_cast<FitPair*>(cl + ncell);
  float4* coef = reinterpret_cast<float4*>(smp + batch / 2);  // two coefficient pairs a word
  const RowSample<float>* rs = rows + (b * nrows + row) * d.S;
  const PointRow<float>* pr = prow + ((long long)b * d.n0 + row / d.n1) * d.n2;
  for (int c = tid; c < ncell; c += nt) {
    const int k = c / d.n3, a = c - k * d.n3;
    const d3 l = node_light(ri.sv, ri.cv, pr[k].ss, pr[k].cs, hdvs[a]);
    cg[c] = cell_geom<float>(ri.sv, ri.cv, l);
    cl[c] = make_double2(l.y, l.z);
  }
  // the sun's horizon test at sample s in FP64, on p_s as integral-ray forms
  // it (atmosphere.clj:95-102, 154-160; ray.clj:22-24)
  auto sun_above = [&](int cell, int s) {
    const double su = (0.5 + s) * (1.0 / d.S);
    const double2 l = cl[cell];
    return (bool)is_above_horizon(P, add3(mk3(ri.r, 0, 0), mul3(mk3(ri.D[0], ri.D[1], ri.D[2]), su)),
                                  mk3(pr[cell / d.n3].ss, l.x, l.y));
  };
  const float log2e = 1.4426950408889634f;
  float rext[3], mext[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    rext[c] = -log2e * P.f_ray_ext[c];
    mext[c] = -log2e * P.f_mie_ext[c];
  }
  const float zmax = __uint_as_float(__float_as_uint((float)segs) - 1u);  // just below the last segment's end
  const int words = segs * (kFitNodes / 2);                               // of one sample's coefficients
  const unsigned coef0 = (unsigned)(reinterpret_cast<unsigned char*>(coef) - smem_raw);
  const float2 Hh2 = make_float2(P.f_Hh, P.f_Hh);
  const float4* tab = table + (size_t)blockIdx.y * kFitRows * words;
  const long long node0 = (b * nrows + row) * ncell;
  const int group = tid / cells, lane = tid - group * cells;

  for (int c0 = 0; c0 < ncell; c0 += cells) {
    const int cell = c0 + lane;
    const bool active = group < groups && cell < ncell;
    float b0 = 0, Dl = 0;
    // (Rayleigh, Mie) per channel, and what the totals lost
    float2 tot[3] = {make_float2(0, 0), make_float2(0, 0), make_float2(0, 0)}, lost[3] = {tot[0], tot[0], tot[0]};
    __syncthreads();  // the cells' directions are there; the last pass is done with the sums
    if (active) {
      const CellGeom<float> g = cg[cell];
      b0 = ri.f_r * g.lx;
      Dl = fmaf(ri.f_D[0], g.lx, fmaf(ri.f_D[1], g.ly, ri.f_D[2] * g.lz));
    }
    for (int s0 = 0; s0 < d.S; s0 += batch) {
      const int ns = min(batch, d.S - s0), n = (ns + 1) & ~1;
      __syncthreads();
      for (int u = tid; u < n; u += nt) {
        const RowSample<float> v = rs[s0 + min(u, ns - 1)];
        const float q = fminf(fmaxf(v.q, 0.0f), P.f_Hh2);
        const FitRange f = fit_range(P, q);
        const float x = fminf(sqrtf(q / P.f_Hh2), 1.0f) * (float)(kFitRows - 1);
        float* o = reinterpret_cast<float*>(smp + (u >> 1)) + (u & 1);
        auto put = [&](const float2& field, float value) { o[reinterpret_cast<const float*>(&field) - reinterpret_cast<const float*>(smp)] = value; };
        put(smp->us, v.us);
        put(smp->cq, f.cq);
        // |(p.l)^2 - q| < 1e8 m^2 and p.l < 4 m around the horizon p.l = -sqrt(q);
        // a sample that only fills the last pair is dark
        put(smp->dark, u < ns ? -sqrtf(q + 1.0e8f) : 3.0e38f);
        put(smp->lit, u >= ns ? 3.0e38f : q < 1.0e8f ? 4.0f : -sqrtf(q - 1.0e8f));
        const float scale = 1.0f / f.range;
        put(smp->scale, scale);
        put(smp->off, -f.dmin * scale);
        put(smp->q, q);
        put(smp->rho, sqrtf(q));
        put(smp->er, v.er);
        put(smp->em, v.em);
#pragma unroll
        for (int c = 0; c < 3; c++) put(smp->tau[c], -log2e * v.tau[c]);
        const int r = min((int)x, kFitRows - 2);
        put(smp->frac, x - (float)r);
        reinterpret_cast<int*>(&smp[u >> 1].row)[u & 1] = r;
      }
      __syncthreads();
      for (int t = tid; t < n * words; t += nt) {
        const int u = t / words, e = t - u * words;
        const FitPair& f = smp[u >> 1];
        const float4* p = tab + (size_t)(u & 1 ? f.row.y : f.row.x) * words + e;
        const float4 A = __ldg(p), B = __ldg(p + words);
        const float w = u & 1 ? f.frac.y : f.frac.x;
        coef[t] = make_float4(fmaf(B.x - A.x, w, A.x), fmaf(B.y - A.y, w, A.y), fmaf(B.z - A.z, w, A.z),
                              fmaf(B.w - A.w, w, A.w));
      }
      __syncthreads();
      if (active) {
        // 8 pairs' sums at a time (x: even, y: odd samples), then the totals; the
        // next sums start from what the totals lost (1 % of the stage; with plain
        // totals 4096 steps spread a sum by 1.5e-7, so by 0.7e-7, its roundings)
        for (int v0 = group; v0 < n / 2; v0 += 8 * groups) {
          float2 accR[3], accM[3];
#pragma unroll
          for (int c = 0; c < 3; c++) accR[c] = make_float2(lost[c].x, 0), accM[c] = make_float2(lost[c].y, 0);
          const int v1 = min(v0 + 8 * groups, n / 2);
#pragma unroll 1
          for (int v = v0; v < v1; v += groups) {
            const FitPair* f = smp + v;
            float2 us, cq, dark, lit;
            ld_pairs(&f->us.x, us, cq);
            ld_pairs(&f->dark.x, dark, lit);
            const float2 bp = fma2(us, make_float2(Dl, Dl), make_float2(b0, b0));  // p_s.l
            bool la = bp.x >= lit.x, lb = bp.y >= lit.y;
            if (bp.x > dark.x && bp.x < lit.x)
              la = sun_above(cell, s0 + 2 * v);
            if (bp.y > dark.y && bp.y < lit.y)
              lb = sun_above(cell, s0 + 2 * v + 1);
            if (!la && !lb) continue;
            float2 scale, off, er, em;
            ld_pairs(&f->scale.x, scale, off);
            ld_pairs(&f->er.x, er, em);
            er = make_float2(la ? er.x : 0.0f, lb ? er.y : 0.0f);
            em = make_float2(la ? em.x : 0.0f, lb ? em.y : 0.0f);
            float2 q, rho;
            ld_pairs(&f->q.x, q, rho);
            // The exit distance d, cancellation-free, and its position in
            // [dmin, dmax]: from dmin for a climbing ray, and for a descending
            // one from dmax by dmax - d = m (1 / (Hh + root) + 1 / (rho + |b|)),
            // m = q - b^2 the perigee's, so that near the ground, where the
            // depth varies over meters of it, the position keeps the perigee's
            // precision and not that of d (0.1 m in FP32).
            const float2 m = fma2(make_float2(-bp.x, -bp.y), bp, q), disc = fma2(bp, bp, cq);
            const float2 root = make_float2(Bulk<float>::sqrt(disc.x), Bulk<float>::sqrt(disc.y));
            const float2 size = make_float2(fabsf(bp.x), fabsf(bp.y));
            const float2 far = add2(size, root), rim = add2(rho, Hh2);
            const float2 num = mul2(m, add2(far, rim)), den = mul2(add2(root, Hh2), add2(rho, size));
            const bool ua = bp.x >= 0.0f, ub = bp.y >= 0.0f;
            const float2 part = make_float2((ua ? cq.x : num.x) * reciprocal(ua ? far.x : den.x),
                                            (ub ? cq.y : num.y) * reciprocal(ub ? far.y : den.y));
            const float2 dist = make_float2(ua ? part.x : far.x, ub ? part.y : far.y);
            // segment and position in it, from its middle (a NaN gives a valid one)
            const float2 z = fma2(make_float2(__saturatef(fmaf(part.x, scale.x, ua ? off.x : 0.0f)),
                                              __saturatef(fmaf(part.y, scale.y, ub ? off.y : 0.0f))),
                                  make_float2(zmax, zmax), make_float2(-0.5f, -0.5f));
            const float2 zr = add2(z, make_float2(kFloorMagic, kFloorMagic));
            const float2 t = sub2(z, add2(zr, make_float2(-kFloorMagic, -kFloorMagic)));
            const unsigned at = (unsigned)(2 * v) * (unsigned)(words * 16) + coef0;
            auto fit = [&](unsigned offset, float x) {  // (Rayleigh, Mie) at position x of a segment
              const float4* k = reinterpret_cast<const float4*>(smem_raw + offset);
              const float4 k2 = k[2], k1 = k[1], k0 = k[0];
              const float2 tt = make_float2(x, x);
              float2 p = make_float2(k2.z, k2.w);
              p = fma2(p, tt, make_float2(k2.x, k2.y));
              p = fma2(p, tt, make_float2(k1.z, k1.w));
              p = fma2(p, tt, make_float2(k1.x, k1.y));
              p = fma2(p, tt, make_float2(k0.z, k0.w));
              return fma2(p, tt, make_float2(k0.x, k0.y));
            };
            const unsigned ia = __float_as_uint(zr.x) - kFloorBits, ib = __float_as_uint(zr.y) - kFloorBits;
            const float2 pa = fit((ua ? ia : segs - 1 - ia) * 48u + at, ua ? t.x : -t.x);
            const float2 pb = fit((ub ? ib : segs - 1 - ib) * 48u + (at + (unsigned)(words * 16)), ub ? t.y : -t.y);
            const float2 odr = mul2(dist, make_float2(Bulk<float>::exp2(pa.x), Bulk<float>::exp2(pb.x)));
            const float2 odm = mul2(dist, make_float2(Bulk<float>::exp2(pa.y), Bulk<float>::exp2(pb.y)));
#pragma unroll
            for (int c = 0; c < 3; c++) {
              const float2 e = fma2(make_float2(mext[c], mext[c]), odm, fma2(make_float2(rext[c], rext[c]), odr, f->tau[c]));
              const float2 T = make_float2(Bulk<float>::exp2(e.x), Bulk<float>::exp2(e.y));
              accR[c] = fma2(T, er, accR[c]);
              accM[c] = fma2(T, em, accM[c]);
            }
          }
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const float2 x = make_float2(accR[c].x + accR[c].y, accM[c].x + accM[c].y), n = add2(tot[c], x);
            lost[c] = sub2(x, sub2(n, tot[c]));
            tot[c] = n;
          }
        }
      }
    }
    // the groups' sums, each with what it lost
    float2* sums = reinterpret_cast<float2*>(coef);
    if (groups > 1) {
      __syncthreads();
      if (group < groups) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
          sums[((2 * c) * groups + group) * cells + lane] = tot[c];
          sums[((2 * c + 1) * groups + group) * cells + lane] = lost[c];
        }
      }
      __syncthreads();
      if (group == 0) {
#pragma unroll
        for (int c = 0; c < 3; c++)
          for (int g = 1; g < groups; g++) {
            const float2 x = sums[((2 * c) * groups + g) * cells + lane], n = add2(tot[c], x), v = sub2(n, tot[c]);
            lost[c] = add2(lost[c], add2(add2(sub2(tot[c], sub2(n, v)), sub2(x, v)),
                                         sums[((2 * c + 1) * groups + g) * cells + lane]));
            tot[c] = n;
          }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) tot[c] = add2(tot[c], lost[c]);
    if (group == 0 && active) {
      const float w = ri.f_Ls;
      const float phR = w * PhaseCS<float>(P.f_phR)(cg[cell].mu);
      Vec4<float> o1, o2;
      o1.x = phR * P.f_srcR[0] * tot[0].x;
      o1.y = phR * P.f_srcR[1] * tot[1].x;
      o1.z = phR * P.f_srcR[2] * tot[2].x;
      o1.w = 0;
      o2.x = w * P.f_srcM[0] * tot[0].y;
      o2.y = w * P.f_srcM[1] * tot[1].y;
      o2.z = w * P.f_srcM[2] * tot[2].y;
      o2.w = 0;
      rayleigh[node0 + cell] = o1;
      mie[node0 + cell] = o2;
    }
  }
}

int launch_first_order_fit(const AtmoParams* params, const BuildDims& d, const RowInfo* rowinfo,
                           const RowSample<float>* rows, const PointRow<float>* prow, const double* hdvs,
                           const unsigned char* table, Vec4<float>* rayleigh, Vec4<float>* mie, cudaStream_t st, int first) {
  int cells, groups;
  fit_shape(d.n2 * d.n3, &cells, &groups);
  const size_t smem = first_order_fit_smem(d);
  if (cudaFuncSetAttribute(k_first_order_fit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return -1;
  k_first_order_fit<<<dim3((unsigned)d.rows(), d.B), cells * groups, smem, st>>>(
      params, d, first, cells, groups, fit_batch(d), rowinfo, rows, prow, hdvs,
      reinterpret_cast<const float4*>(table), rayleigh, mie);
  return 0;
}

}  // namespace sfsim
