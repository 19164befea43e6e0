// k_ray_scatter.cu -- ray scatter dS of the multiple-scattering iterations
// (atmosphere.clj:192-200) with J from the point-scatter table.
//
// One block per view row (i, j).  For a ray sample p_s the J lookup's height
// and elevation coordinates depend on the row only, so J collapses to a plane
// [sun heading][sun elevation] per sample.  Every thread builds one cell of
// the planes of the next CH samples into one of two buffers and gathers from
// the other, with one barrier per CH samples.
//
// Building: the J values of the sample's four (height, elevation) corners
// stay in registers, each in the slot of its height's and elevation's parity,
// so that a step to a neighbouring (height, elevation) cell loads only the
// new corners and moves none.  T(x, p_s) (k_view_rows) goes into the plane.
//
// Gathering: a thread follows one heading column along the ray, linear in
// the sun elevation of p_s.  A node's sun-angle coordinate is that of (v, l)
// at every sample, and for an inner heading whose v.l some light of the
// node's sun elevation reaches it is the heading itself
// (index-to-sun-direction solves for it), so one column is enough.  The
// headings that no light reaches are clamped to the two lights in the plane
// of x and v, the same two for all of them, and the first and last heading
// always are: these two nodes per sun elevation are gathered from their two
// columns by a thread each, and the clamped headings copy them.
//
// Plane layout: texel (sun elevation r, heading a) at a * st + r, three values
// a texel, st = 4 * odd > n2: a warp of 32 sun elevations of one heading
// reads 32 different banks, and the builder's stores (for 8 headings, 4 sun
// elevations x 8 headings a warp) do too.
//
// What bounds it: the L1 data pipe, 85 % busy with 236M wavefronts a launch of
// the production tables (32x255x32x8, 128 samples): of 226 a row and sample 60
// are the gathers, 48 the constants, 48 the loads of J, 32 the stores.  0.89 ms a
// launch, 4.43 ms of a build, 4.60 with the offsets of every sample (90 %, 261M);
// with a bilinear gather per node (four texels, every heading) 5.70.  The
// reference's tables (32x127x32x8, 100 samples) 2.20 -> 1.83 -> 1.75 ms; 16
// atmospheres of 16x128x16x8 7.6 -> 6.9.  Separate builder and gatherer warps
// took 6.1 to 7.8 ms, corners prefetched into registers 5.6, two columns and
// cells a thread 4.6 to 5.2 (231M wavefronts, but fewer warps).
#include <type_traits>

#include "atmo_device.cuh"
#include "kernels.h"

namespace sfsim {

// Samples whose constants are formed at a time.
constexpr int kRayBatch = 128;
// Threads of a block at most: one per column, and one per cell.  Blocks of 320
// go three to an SM, of 512 two, of 1024 one, 64 registers a thread all the
// same in FP32.  Rows of more columns take passes (WIDE), 512 at a time.
constexpr int kRayThreads = 320, kRayThreadsMore = 512, kRayThreadsMost = 1024;
constexpr int kRayThreadsWide = 512;

__host__ __device__ constexpr int ray_column(int n2) { return 4 * (((n2 + 4) / 4) | 1); }

// Shared memory, in this order: the gatherers' constants of a batch, (us, us',
// 1/r, 1/r') per sample pair; the builders', 8 values a sample (the four
// slots' weights, T, then the mask of the slots to load) and the
// slots' offsets; the columns' sums of the first and last headings; two
// buffers of CH planes.
struct RayLayout {
  unsigned gather, build, corners, edge, planes, plane_bytes, bytes;
  int ch;  // planes per buffer
};
template <class Real>
__host__ inline RayLayout ray_layout(const BuildDims& d, int ch, int groups) {
  auto up = [](size_t x) { return (x + 15) & ~size_t(15); };
  RayLayout l;
  size_t o = 0;
  l.gather = 0;
  o = up(o + sizeof(Real) * 2 * kRayBatch);
  l.build = (unsigned)o;
  o = up(o + sizeof(Real) * 8 * kRayBatch);
  l.corners = (unsigned)o;
  o = up(o + sizeof(int4) * kRayBatch);
  l.edge = (unsigned)o;
  o = up(o + sizeof(Real) * 12 * d.n2);
  l.planes = (unsigned)o;
  l.plane_bytes = (unsigned)(sizeof(Real) * 3 * ray_column(d.n2) * d.n3);
  o += 2 * (size_t)ch * groups * l.plane_bytes;
  l.bytes = (unsigned)o;
  l.ch = ch;
  return l;
}

// Sixteen planes, one sample's constants and (to 16 KB) a staged row: an
// upper bound of the layout above at four planes, kept as the limit of the
// accepted table shapes.
template <class Real>
size_t ray_scatter_capacity(const BuildDims& d) {
  const size_t texels = d.n2 % 32 == 0 ? (size_t)(d.n2 + 4) * d.n3 : (size_t)d.n2 * d.n3;
  const size_t row = (size_t)d.S * sizeof(RowSample<Real>);
  return ((16 * (7 * sizeof(Real) + 4 * sizeof(int)) + 15) & ~size_t(15)) + sizeof(Real) * 48 * texels +
         (row <= 16384 ? row : 0);
}
template size_t ray_scatter_capacity<float>(const BuildDims&);
template size_t ray_scatter_capacity<double>(const BuildDims&);

// (1 - exp2(z)) / (1 - exp(-3.6)) in [0, 1] (sun-elevation-to-index,
// atmosphere.clj:322-326); a NaN gives 0, so the result is always a valid
// coordinate.
__device__ __forceinline__ float sun_fraction(float z, float k) {
  return __saturatef(fmaf(-k, Bulk<float>::exp2(z), k));
}
__device__ __forceinline__ double sun_fraction(double z, double k) {
  return fmin(fmax(fma(-k, Bulk<double>::exp2(z), k), 0.0), 1.0);
}

// A mask kept among the values of its sample.
__device__ __forceinline__ float mask_value(float, int m) { return __int_as_float(m); }
__device__ __forceinline__ double mask_value(double, int m) { return __longlong_as_double(m); }
__device__ __forceinline__ int mask_of(float v) { return __float_as_int(v); }
__device__ __forceinline__ int mask_of(double v) { return (int)__double_as_longlong(v); }

// WIDE: more columns than kRayThreadsMost; they go in passes (the planes are
// built again for each) and the threads walk the cells without keeping corners.
// 32x127 rows, 100 samples, five iterations, by the sun elevations and headings:
//                                64x4  36x7  85x3  40x8  64x8  48x16  200x4 ms
//   one thread a column or cell  2.16  2.20  2.45  2.53  4.25  5.81   -
//   WIDE                         3.86  3.97  4.09  4.23  10.2  15.9   23.6
//   gathers per node (4 texels)  2.49  2.42  2.23  6.02  9.29  25.7   41.2
// Two or three headings have as many columns as the nodes have columns to read,
// so a column each gains nothing there: 128x2 2.32 and 2.24.  FP64, two
// iterations of 8x32 rows: 64x4 1.65 / 2.06 / 1.89, 64x8 2.88 / 4.90 / 4.75.
constexpr int kRayBlocks = 3;  // blocks per SM: 4.60 ms of a production build, two 5.04
constexpr int kRayUnroll = 2;  // samples whose new corners are on their way together
// SPLIT: several groups of threads share the ray's samples.
template <class Real, int THREADS, int BLOCKS, bool WIDE, bool SPLIT>
__global__ void __launch_bounds__(THREADS, BLOCKS)
    k_ray_scatter(BuildDims d, RayLayout lay, const RowInfo* rowinfo, const RowSample<Real>* rows,
                  const CellGeom<Real>* geom, const Coord<Real>* angle, const Vec4<Real>* J, Vec4<Real>* dS,
                  int ngroups) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using R2 = V2<Real>;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int groups = SPLIT ? ngroups : 1;
  const int per = SPLIT ? nt / groups : nt, group = SPLIT ? tid / per : 0, gt = SPLIT ? tid - group * per : tid;
  const int b = blockIdx.y;
  const long long row = blockIdx.x, nrows = d.rows();
  const int ncell = d.n2 * d.n3, CH = lay.ch;
  const long long node0 = (b * nrows + row) * ncell;
  Real* cg = reinterpret_cast<Real*>(smem_raw + lay.gather);
  Real* cb = reinterpret_cast<Real*>(smem_raw + lay.build);
  int4* cp = reinterpret_cast<int4*>(smem_raw + lay.corners);
  Real* edge = reinterpret_cast<Real*>(smem_raw + lay.edge);
  const RowSample<Real>* rs = rows + (b * nrows + row) * d.S;
  const RowR<Real> rw = row_r<Real>(rowinfo[b * nrows + row]);
  const int st = ray_column(d.n2);
  const unsigned plane_bytes = lay.plane_bytes;
  // the texel past the last sun elevation, read with weight 0 at the top
  for (int t = tid; t < 2 * CH * groups * d.n3; t += nt) {
    Real* p = reinterpret_cast<Real*>(smem_raw + lay.planes) + 3 * (t * st + d.n2);
    p[0] = p[1] = p[2] = Real(0);
  }

  const Vec4<Real>* Jb = J + (long long)b * d.n4();
  // J of the thread's cell in the slots 2 (height & 1) + (elevation & 1)
  Vec4<Real> v[4];
#pragma unroll
  for (int q = 0; q < 4; q++) v[q].x = v[q].y = v[q].z = v[q].w = Real(0);
  int g0 = 0;  // the group's first sample of the batch
  // the cell in the plane of batch sample u: new corners by the sample's mask, then their mix
  auto form = [&](int u, const Vec4<Real>* Jc, Real* o) {
    const Real* k = cb + 8 * u;
    R2 w01, w23, T01, T2m;
    ld_pairs(k, w01, w23);
    ld_pairs(k + 4, T01, T2m);
    const int mask = WIDE || (SPLIT && u == g0) ? 15 : mask_of(T2m.y);
    if (mask) {  // about half of the samples stay in the cell of the one before
      const int4 q = cp[u];
      if (mask & 1) v[0] = Jc[q.x];
      if (mask & 2) v[1] = Jc[q.y];
      if (mask & 4) v[2] = Jc[q.z];
      if (mask & 8) v[3] = Jc[q.w];
    }
    o[0] = fma(w01.x, v[0].x, fma(w01.y, v[1].x, fma(w23.x, v[2].x, w23.y * v[3].x))) * T01.x;
    o[1] = fma(w01.x, v[0].y, fma(w01.y, v[1].y, fma(w23.x, v[2].y, w23.y * v[3].y))) * T01.y;
    o[2] = fma(w01.x, v[0].z, fma(w01.y, v[1].z, fma(w23.x, v[2].z, w23.y * v[3].z))) * T2m.x;
  };
  const int pitch = (int)(plane_bytes / sizeof(Real));
  const int own = 3 * ((gt % d.n3) * st + gt / d.n3);
  // planes of batch samples u0 .. u1 - 1
  auto build = [&](int u0, int u1, int buf) {
    Real* plane = reinterpret_cast<Real*>(smem_raw + lay.planes + (unsigned)((2 * group + buf) * CH) * plane_bytes);
    if constexpr (WIDE) {
      for (int cell = tid; cell < ncell; cell += nt) {
        Real* o = plane + 3 * ((cell % d.n3) * st + cell / d.n3);
        for (int u = u0; u < u1; u++, o += pitch) form(u, Jb + cell, o);
      }
    } else if (gt < ncell) {
      Real* o = plane + own;
#pragma unroll kRayUnroll
      for (int u = u0; u < u1; u++, o += pitch) form(u, Jb + gt, o);
    }
  };

  const int inner = d.n3 - 2, ncol = d.n2 * (d.n3 + 2);
  const Real log2e = Real(1.4426950408889634);
  const Real kfrac = Real(1.0 / 0.97267627755270747);  // 1 / (1 - exp(-3.6))
  const R2 zc = dup(Real(-0.6 * 1.4426950408889634 + Bulk<Real>::kExp2Shift)), last = dup(Real(d.n2 - 1));

  for (int c0 = 0; c0 < ncol; c0 += per) {
    // column c0 + gt; the inner headings' columns, then the two
    // columns of the first and of the last heading, each for every sun elevation
    R2 acc[3] = {dup(Real(0)), dup(Real(0)), dup(Real(0))};  // even and odd samples
    R2 Dl = dup(Real(0)), b0 = dup(Real(0));
    unsigned col = 0;
    int cell = -1, slot = -1;  // the node to store, or the edge sum's slot
    Real wedge = 0;
    if (c0 + gt < ncol) {
      const int h = (c0 + gt) / d.n2, k = (c0 + gt) - h * d.n2;
      const int e = h - inner;
      const int a = e < 0 ? h + 1 : e < 2 ? 0 : d.n3 - 1;
      const CellGeom<Real> g = geom[node0 + k * d.n3 + a];
      int column = a;
      if (e < 0) {
        const CellGeom<Real> g0 = geom[node0 + k * d.n3], g1 = geom[node0 + k * d.n3 + d.n3 - 1];
        const bool clamped = (g.ly == g0.ly && g.lz == g0.lz) || (g.ly == g1.ly && g.lz == g1.lz);
        cell = clamped ? -1 : k * d.n3 + a;
      } else {
        const Coord<Real> m = angle[node0 + k * d.n3 + a];
        column = (e & 1) ? upper_index(m.u, d.n3) : m.u;
        wedge = (e & 1) ? m.s : Real(1) - m.s;
        slot = e * d.n2 + k;
      }
      // z = -log2(e) (3 p_s.l / |p_s| + 0.6), p_s.l = x.l + us D.l
      b0 = dup(Real(-3) * log2e * (rw.r * g.lx));
      Dl = dup(Real(-3) * log2e * fma(rw.D[0], g.lx, fma(rw.D[1], g.ly, rw.D[2] * g.lz)));
      col = (unsigned)(sizeof(Real) * 3 * column * st);
    }
    for (int s0 = 0; s0 < d.S; s0 += kRayBatch) {
      const int ns = min(kRayBatch, d.S - s0), n = (ns + 1) & ~1;
      __syncthreads();
      for (int u = tid; u < n; u += nt) {
        const RowSample<Real> q = rs[s0 + min(u, ns - 1)];
        Real* g = cg + 4 * (u >> 1) + (u & 1);
        g[0] = q.us;
        g[2] = q.inv_r;
        // the slots' offsets: the lower corner where the parities agree, else the upper one
        auto slots = [&](const RowSample<Real>& p) {
          const int v0 = upper_index(p.u0, d.n0), v1 = upper_index(p.u1, d.n1);
          const int he = p.u0 & 1 ? v0 : p.u0, ho = p.u0 & 1 ? p.u0 : v0;
          const int ee = p.u1 & 1 ? v1 : p.u1, eo = p.u1 & 1 ? p.u1 : v1;
          return make_int4((he * d.n1 + ee) * ncell, (he * d.n1 + eo) * ncell, (ho * d.n1 + ee) * ncell,
                           (ho * d.n1 + eo) * ncell);
        };
        const int4 o = slots(q);
        int mask = 15;
        if (u > 0) {
          const int4 p = slots(rs[s0 + min(u - 1, ns - 1)]);
          mask = (o.x != p.x) | (o.y != p.y) << 1 | (o.z != p.z) << 2 | (o.w != p.w) << 3;
        }
        cp[u] = o;
        const Real h1 = q.u0 & 1 ? Real(1) - q.s0 : q.s0, h0 = q.u0 & 1 ? q.s0 : Real(1) - q.s0;
        const Real e1 = q.u1 & 1 ? Real(1) - q.s1 : q.s1, e0 = q.u1 & 1 ? q.s1 : Real(1) - q.s1;
        Real* k = cb + 8 * u;
        k[0] = h0 * e0;
        k[1] = h0 * e1;
        k[2] = h1 * e0;
        k[3] = h1 * e1;
#pragma unroll
        for (int c = 0; c < 3; c++) k[4 + c] = u < ns ? exp_neg(q.tau[c]) : Real(0);
        k[7] = mask_value(Real(0), mask);
      }
      __syncthreads();
      // every group's part of the batch, in pairs; all groups meet every barrier
      const int part = !SPLIT ? n : 2 * ((n / 2 + groups - 1) / groups);
      g0 = SPLIT ? min(group * part, n) : 0;
      const int g1 = SPLIT ? min(g0 + part, n) : n;
      build(g0, min(g0 + CH, g1), 0);
      __syncthreads();
      for (int off = 0, buf = 0; off < part; off += CH, buf ^= 1) {
        const int u0 = g0 + off, u1 = min(u0 + CH, g1);
        {
          unsigned pa = lookup_base<Real>(lay.planes + (unsigned)((2 * group + buf) * CH) * plane_bytes + col,
                                             3 * sizeof(Real));
          const Real* k = cg + 2 * u0;
          auto pair = [&]() {
            R2 us, ir;
            ld_pairs(k, us, ir);
            const R2 z = fma2(fma2(us, Dl, b0), ir, zc);
            const R2 e = mul2(mk2(sun_fraction(z.x, kfrac), sun_fraction(z.y, kfrac)), last);
            unsigned oa, ob;
            const R2 f = lookup(e, pa, pa + plane_bytes, 3 * (unsigned)sizeof(Real), oa, ob);
            const Real* qa = reinterpret_cast<const Real*>(smem_raw + oa);
            const Real* qb = reinterpret_cast<const Real*>(smem_raw + ob);
#pragma unroll
            for (int c = 0; c < 3; c++) {
              const R2 lo = mk2(qa[c], qb[c]), hi = mk2(qa[c + 3], qb[c + 3]);
              acc[c] = add2(acc[c], fma2(sub2(hi, lo), f, lo));
            }
            pa += 2 * plane_bytes;
            k += 4;
          };
          if (u1 - u0 == 8) {
#pragma unroll
            for (int h = 0; h < 4; h++) pair();
          } else {
#pragma unroll 1
            for (int u = u0; u < u1; u += 2) pair();
          }
        }
        if (u1 < g1) build(u1, min(u1 + CH, g1), buf ^ 1);
        __syncthreads();
      }
    }
    if constexpr (SPLIT) {
      // the groups' sums, in order (the planes are no longer read)
      Real* sums = reinterpret_cast<Real*>(smem_raw + lay.planes);
      if (group > 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) sums[((group - 1) * 3 + c) * per + gt] = acc[c].x + acc[c].y;
      }
      __syncthreads();
      if (group == 0) {
        for (int g = 0; g < groups - 1; g++) {
#pragma unroll
          for (int c = 0; c < 3; c++) acc[c].x += sums[(g * 3 + c) * per + gt];
        }
      } else {
        cell = slot = -1;
      }
    }
    if (cell >= 0) {
      Vec4<Real> o;
      o.x = rw.Ls * (acc[0].x + acc[0].y);
      o.y = rw.Ls * (acc[1].x + acc[1].y);
      o.z = rw.Ls * (acc[2].x + acc[2].y);
      o.w = 0;
      dS[node0 + cell] = o;
    }
    if (slot >= 0) {
#pragma unroll
      for (int c = 0; c < 3; c++) edge[3 * slot + c] = wedge * (acc[c].x + acc[c].y);
    }
  }
  __syncthreads();
  // the first and last headings, and the inner ones clamped to their lights
  for (int t = tid; t < ncell; t += nt) {
    const int k = t / d.n3, a = t - k * d.n3;
    int side = a == 0 ? 0 : a == d.n3 - 1 ? 1 : -1;
    if (side < 0) {
      const CellGeom<Real> g = geom[node0 + t];
      const CellGeom<Real> g0 = geom[node0 + k * d.n3], g1 = geom[node0 + k * d.n3 + d.n3 - 1];
      side = g.ly == g0.ly && g.lz == g0.lz ? 0 : g.ly == g1.ly && g.lz == g1.lz ? 1 : -1;
    }
    if (side >= 0) {
      const Real *e0 = edge + 3 * (2 * side * d.n2 + k), *e1 = e0 + 3 * d.n2;
      Vec4<Real> o;
      o.x = rw.Ls * (e0[0] + e1[0]);
      o.y = rw.Ls * (e0[1] + e1[1]);
      o.z = rw.Ls * (e0[2] + e1[2]);
      o.w = 0;
      dS[node0 + t] = o;
    }
  }
}

template <class Real>
int launch_ray_scatter(const BuildDims& d, const RowInfo* rowinfo, const RowSample<Real>* rows,
                       const CellGeom<Real>* geom, const Coord<Real>* angle, const Vec4<Real>* J, Vec4<Real>* dS,
                       cudaStream_t st) {
  const int ncol = d.n2 * (d.n3 + 2);
  constexpr bool one = sizeof(Real) == 8;  // block per SM: FP64's registers
  const bool wide = ncol > kRayThreadsMost;
  // Few columns and few rows leave the SMs with a warp or two each, one after
  // another along the ray: then up to four groups of a block share its samples.
  // 128 rows of 48 columns, 64 samples, two iterations, 1 / 2 / 4 groups: FP32 37 /
  // 28 / 24 us; a build 144 / 137 / 131, in FP64 1650 / 1557 / 1531.  The rows
  // are one atmosphere's: the groups order the sums, and an atmosphere of a
  // batch has the bits of its own build.
  int groups = 1;
  const int per = wide ? kRayThreadsWide : (ncol + 31) / 32 * 32;
  while (!wide && groups < 4 && 2 * groups * per <= kRayThreads &&
         d.rows() * (2 * groups * per / 32) <= 4864)  // 32 warps an SM
    groups *= 2;
  const int block = per * groups;
  // the most planes per buffer that let two blocks share an SM (blocks that have one for themselves: that
  // fit), else that fit
  RayLayout lay = ray_layout<Real>(d, 8, groups);
  const unsigned room = (per > kRayThreadsMore ? 220 : 100) * 1024;
  for (int ch = 8; ch >= 2 && lay.bytes > room; ch /= 2) lay = ray_layout<Real>(d, ch, groups);
  const dim3 grid((unsigned)d.rows(), d.B);
  auto go = [&](auto kernel) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.bytes) != cudaSuccess)
      return -1;
    kernel<<<grid, block, lay.bytes, st>>>(d, lay, rowinfo, rows, geom, angle, J, dS, groups);
    return 0;
  };
  if (wide) return go(k_ray_scatter<Real, kRayThreadsWide, 1, true, false>);
  if (groups > 1) return go(k_ray_scatter<Real, kRayThreads, one ? 1 : kRayBlocks, false, true>);
  if (per <= kRayThreads) return go(k_ray_scatter<Real, kRayThreads, one ? 1 : kRayBlocks, false, false>);
  if (per <= kRayThreadsMore) return go(k_ray_scatter<Real, kRayThreadsMore, one ? 1 : 2, false, false>);
  return go(k_ray_scatter<Real, kRayThreadsMost, 1, false, false>);
}

template int launch_ray_scatter<float>(const BuildDims&, const RowInfo*, const RowSample<float>*,
                                       const CellGeom<float>*, const Coord<float>*, const Vec4<float>*, Vec4<float>*,
                                       cudaStream_t);
template int launch_ray_scatter<double>(const BuildDims&, const RowInfo*, const RowSample<double>*,
                                        const CellGeom<double>*, const Coord<double>*, const Vec4<double>*, Vec4<double>*,
                                        cudaStream_t);

}  // namespace sfsim
