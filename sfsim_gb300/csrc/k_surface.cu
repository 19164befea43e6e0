// k_surface.cu -- surface radiance dE of the multiple-scattering iterations
// (atmosphere.clj:225-230): at every node (height iE, sun elevation kE) the
// integral over the upper half sphere of dS(x, w, l, above) (w.n); the
// reference passes the ray steps as the sphere steps (atmosphere_lut.clj:89).
//
// The quadrature (sphere.clj:62-93) is a set of rings about the normal, which
// is the first axis.  A ring's directions share the height, elevation and
// sun-elevation coordinates of the lookup and differ in the sun angle w.l
// alone, and the lookup is linear in the ring's row of texels along that
// axis.  So the sum over a ring's directions is a sum over its row's texels
// with weights that hold all that depends on the directions: they are the
// same at every height and in every iteration and are summed once per build
// for each light, ring and texel (k_half_weights; in the first iteration the
// Mie strength takes those with the phase).
//
// What bounds it: the latency of a block's few dependent loads.  A node of
// 16x64 nodes with 128 ray steps (2607 directions in 32 rings, 8 headings)
// takes 256 texels of 8 corners, 32 KB through L1, where gathering every
// direction's 16 corners took 650 KB.  Measured for a build, gathered / by
// rings: 16 such atmospheres with 4 iterations 2739 / 304 us (63 a launch),
// one with 5 iterations 309 / 64, 63 sun elevations and 100 ray steps 177 /
// 54; the weights add 32 us of set-up to the 16 (5 to one), beside others.
#include <cstddef>

#include "atmo_device.cuh"
#include "kernels.h"

namespace sfsim {

// Weights of the lights [k0, k0 + kn), a warp per (light, ring).  A texel's
// part in the clamped linear interpolation at a direction is 1 less the
// distance of the direction's coordinate, if that is positive.  The lanes
// form the directions' coordinates and phases once, then each lane sums a
// slice of the directions for one texel.  A thread per texel that formed them
// itself walked the whole ring in one chain: an FP64 build of 32 lights, 16
// rings and 4 headings took 4.22 ms with it, 3.00 so.
constexpr int kWeightChunk = 128;  // directions formed at a time

template <class Real>
__global__ void __launch_bounds__(32)
    k_half_weights(const AtmoParams* params, BuildDims d, SetupBuffers<Real> o, int k0) {
  __shared__ Real coord[kWeightChunk], phase[kWeightChunk];
  const int lane = threadIdx.x, b = blockIdx.y;
  const int kk = blockIdx.x / d.Th, r = blockIdx.x - kk * d.Th;
  const SurfRow<Real> er = o.erow[(long long)b * d.nE() + k0 + kk];
  const HalfRing<Real> ring = o.half_rings[r];
  const int end = o.half_rings[r + 1].w0;
  const PhaseCS<Real> phase_mie(Bulk<Real>::phase_mie(params[b]));
  const Real scale3 = Real(0.5) * Real(d.n3 - 1), hi = Real(d.n3 - 1);
  const Real base = ring.x0 * er.lx;
  HalfWeight<Real>* out =
      o.half_weights + (((long long)b * d.half_slab + kk) * d.Th + r) * d.n3;
  const int width = d.n3 > 16 ? 32 : d.n3 > 8 ? 16 : d.n3 > 4 ? 8 : d.n3 > 2 ? 4 : 2;  // texels at a time
  const int slice = lane / width, slices = 32 / width;
  for (int a0 = 0; a0 < d.n3; a0 += width) {
    const Real a = Real(a0 + lane % width);
    Real ray = 0, cray = 0, mie = 0, cmie = 0;
    for (int w0 = ring.w0; w0 < end; w0 += kWeightChunk) {
      const int n = min(kWeightChunk, end - w0);
      __syncwarp();
      for (int w = lane; w < n; w += 32) {
        const Real mu = fma(o.half_y[w0 + w], er.ly, base);  // omega . l, l.z = 0
        coord[w] = fmin(fmax(scale3 * (Real(1) + mu), Real(0)), hi);
        phase[w] = phase_mie(mu);
      }
      __syncwarp();
      for (int w = slice; w < n; w += slices) {
        const Real part = Real(1) - fabs(coord[w] - a);
        if (part > Real(0)) {
          kahan_add(ray, cray, part);
          kahan_add(mie, cmie, part * phase[w]);
        }
      }
    }
    for (int s = 16; s >= width; s >>= 1) {
      ray += __shfl_xor_sync(0xffffffffu, ray, s);
      mie += __shfl_xor_sync(0xffffffffu, mie, s);
    }
    const int at = a0 + lane;
    if (slice == 0 && at < d.n3) out[at] = HalfWeight<Real>{ray * ring.weight, mie * ring.weight};
  }
}

constexpr int kSurfaceThreads = 128;

template <class Real, bool FIRST>
__global__ void __launch_bounds__(kSurfaceThreads)
    k_surface_radiance(BuildDims d, SetupBuffers<Real> o, const Vec4<Real>* dS, const Vec4<Real>* Mt, Vec4<Real>* dE,
                       int k0, int kn) {
  __shared__ Real red[3][kSurfaceThreads / 32];
  const int b = blockIdx.y;
  const int i = blockIdx.x / kn, kk = blockIdx.x - i * kn;
  const long long node = (long long)b * d.nE() + (long long)i * d.nE1 + k0 + kk;
  const SurfRow<Real> er = o.erow[node];
  const Vec4<Real>* tS = dS + (long long)b * d.n4();
  const Vec4<Real>* tM = FIRST ? Mt + (long long)b * d.n4() : nullptr;
  const Coord<Real>* row = o.half_rows + ((long long)b * d.nE0 + i) * d.Th;
  const HalfWeight<Real>* weights = o.half_weights + ((long long)b * d.half_slab + kk) * d.Th * d.n3;
  Real acc[3] = {0, 0, 0}, cmp[3] = {0, 0, 0};
  const int items = d.Th * d.n3;
  for (int t = threadIdx.x; t < items; t += kSurfaceThreads) {
    const HalfWeight<Real> w = weights[t];
    if (w.ray == Real(0)) continue;  // no direction reads this texel
    const int r = t / d.n3, a = t - r * d.n3;
    const Coord<Real> c = row[r];
    Real v[3], vm[3];
    gather_row_texel(tS, d, er.u0, er.s0, c.u, c.s, er.u2, er.s2, a, v);
    if (FIRST) gather_row_texel(tM, d, er.u0, er.s0, c.u, c.s, er.u2, er.s2, a, vm);
#pragma unroll
    for (int ch = 0; ch < 3; ch++) {
      Real x = v[ch] * w.ray;
      if (FIRST) x = fma(vm[ch], w.mie, x);
      kahan_add(acc[ch], cmp[ch], x);
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int ch = 0; ch < 3; ch++) {
    for (int s = 16; s > 0; s >>= 1) acc[ch] += __shfl_xor_sync(0xffffffffu, acc[ch], s);
    if (lane == 0) red[ch][warp] = acc[ch];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Vec4<Real> out;
    out.x = (red[0][0] + red[0][1]) + (red[0][2] + red[0][3]);
    out.y = (red[1][0] + red[1][1]) + (red[1][2] + red[1][3]);
    out.z = (red[2][0] + red[2][1]) + (red[2][2] + red[2][3]);
    out.w = 0;
    dE[node] = out;
  }
}

static inline dim3 grid1(long long n, int block, int B) { return dim3((unsigned)((n + block - 1) / block), B); }

template <class Real>
static void launch_half_weights(const AtmoParams* params, const BuildDims& d, const SetupBuffers<Real>& o, int k0,
                                int kn, cudaStream_t st) {
  k_half_weights<Real><<<dim3((unsigned)(kn * d.Th), d.B), 32, 0, st>>>(params, d, o, k0);
}

// The weights of all lights, where they are kept; the number of kernels launched.
template <class Real>
int launch_surface_weights(const AtmoParams* params, const BuildDims& d, const SetupBuffers<Real>& o,
                           cudaStream_t st) {
  if (d.Th == 0 || d.half_slab < d.nE1) return 0;
  launch_half_weights(params, d, o, 0, d.nE1, st);
  return 1;
}

// Where the weights of all lights are not kept (half_slab), those of half_slab
// lights at a time are summed before the nodes that read them.
template <class Real>
int launch_surface_radiance(const AtmoParams* params, const BuildDims& d, const SetupBuffers<Real>& o,
                            const Vec4<Real>* dS, const Vec4<Real>* mie, Vec4<Real>* dE, cudaStream_t st) {
  int launches = 0;
  for (int k0 = 0; k0 < d.nE1; k0 += d.half_slab) {
    const int kn = min(d.half_slab, d.nE1 - k0);
    if (d.half_slab < d.nE1 && d.Th > 0) {
      launch_half_weights(params, d, o, k0, kn, st);
      launches++;
    }
    const dim3 grid((unsigned)(d.nE0 * kn), d.B);
    if (mie)
      k_surface_radiance<Real, true><<<grid, kSurfaceThreads, 0, st>>>(d, o, dS, mie, dE, k0, kn);
    else
      k_surface_radiance<Real, false><<<grid, kSurfaceThreads, 0, st>>>(d, o, dS, mie, dE, k0, kn);
    launches++;
  }
  return launches;
}

#define SFSIM_INSTANTIATE(Real)                                                                                   \
  template int launch_surface_weights<Real>(const AtmoParams*, const BuildDims&, const SetupBuffers<Real>&,       \
                                            cudaStream_t);                                                        \
  template int launch_surface_radiance<Real>(const AtmoParams*, const BuildDims&, const SetupBuffers<Real>&,      \
                                             const Vec4<Real>*, const Vec4<Real>*, Vec4<Real>*, cudaStream_t);

SFSIM_INSTANTIATE(float)
SFSIM_INSTANTIATE(double)

}  // namespace sfsim
