// k_scatter.cu -- the re-interpolating accumulation of E and S in the
// multiple-scattering iterations (atmosphere_lut.clj:86-97) and the outputs.
#include <cstddef>

#include "atmo_device.cuh"
#include "kernels.h"

namespace sfsim {

// ---------------------------------------------------------------------------
// Re-interpolating accumulation and outputs
// ---------------------------------------------------------------------------

// A 4-D node's re-interpolation coordinates (forward of backward of the
// node): height and elevation of its view row, sun elevation of its (height,
// sun elevation) pair, its own sun angle.
template <class Real>
__device__ __forceinline__ void node_coords(const BuildDims& d, const Remap2<Real>* rowmap,
                                            const PointRow<Real>* prow, const Coord<Real>* angle, int b,
                                            long long node, int u[4], Real s[4]) {
  const unsigned rk = (unsigned)node / d.n3, row = rk / d.n2;  // a table has at most 2^31 nodes
  const Remap2<Real> rm = rowmap[b * d.rows() + row];
  const PointRow<Real>& pk = prow[((long long)b * d.n0 + row / d.n1) * d.n2 + (rk - row * d.n2)];
  const Coord<Real> c = angle[b * d.n4() + node];
  u[0] = rm.u[0], u[1] = rm.u[1], u[2] = pk.u2, u[3] = c.u;
  s[0] = rm.s[0], s[1] = rm.s[1], s[2] = pk.s2, s[3] = c.s;
}

template <class Real>
__global__ void k_accumulate4(BuildDims d, const Remap2<Real>* rowmap, const PointRow<Real>* prow,
                              const Coord<Real>* angle, const Vec4<Real>* A, const Vec4<Real>* Bt, Vec4<Real>* out) {
  const long long n4 = d.n4();
  const long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (node >= n4) return;
  int u[4];
  Real s[4];
  node_coords(d, rowmap, prow, angle, b, node, u, s);
  Real va[3], vb[3] = {0, 0, 0};
  interp4<Real, true>(A + b * n4, d, u, s, va);
  if (Bt) interp4<Real, true>(Bt + b * n4, d, u, s, vb);
  Vec4<Real> o;
  o.x = va[0] + vb[0];
  o.y = va[1] + vb[1];
  o.z = va[2] + vb[2];
  o.w = 0;
  out[b * n4 + node] = o;
}

template <class Real>
__global__ void k_accumulate2(int n0, int n1, const Remap2<Real>* remap, const Vec4<Real>* A, const Vec4<Real>* Bt,
                              Vec4<Real>* out) {
  const long long n = (long long)n0 * n1;
  const long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (node >= n) return;
  const Remap2<Real> m = remap[b * n + node];
  Real va[3] = {0, 0, 0}, vb[3] = {0, 0, 0};
  if (A) interp2(A + b * n, n0, n1, m.u, m.s, va);
  if (Bt) interp2(Bt + b * n, n0, n1, m.u, m.s, vb);
  Vec4<Real> o;
  o.x = va[0] + vb[0];
  o.y = va[1] + vb[1];
  o.z = va[2] + vb[2];
  o.w = 0;
  out[b * n + node] = o;
}

// convert-4d-to-2d (image.clj:299-312) + pack-matrices (matrix.clj:130-134)
template <class Real>
__global__ void k_output4(BuildDims d, const Remap2<Real>* rowmap, const PointRow<Real>* prow,
                          const Coord<Real>* angle, const Vec4<Real>* tab, float* out) {
  const long long n4 = d.n4();
  const long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (node >= n4) return;
  int u[4];
  Real s[4];
  node_coords(d, rowmap, prow, angle, b, node, u, s);
  Real v[3];
  interp4<Real, true>(tab + b * n4, d, u, s, v);
  const unsigned rk = (unsigned)node / d.n3, row = rk / d.n2;
  const int a = (int)((unsigned)node - rk * d.n3), k = (int)(rk - row * d.n2);
  const int i = (int)(row / d.n1), j = (int)(row - i * d.n1);
  const long long dst = ((long long)i * d.n2 + k) * ((long long)d.n1 * d.n3) + (long long)j * d.n3 + a;
  float* o = out + 3 * (b * n4 + dst);
  o[0] = (float)v[0];
  o[1] = (float)v[1];
  o[2] = (float)v[2];
}

template <class Real>
__global__ void k_output2(int n0, int n1, const Remap2<Real>* remap, const Vec4<Real>* tab, float* out) {
  const long long n = (long long)n0 * n1;
  const long long node = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (node >= n) return;
  const Remap2<Real> m = remap[b * n + node];
  Real v[3] = {0, 0, 0};
  if (tab) interp2(tab + b * n, n0, n1, m.u, m.s, v);
  float* o = out + 3 * (b * n + node);
  o[0] = (float)v[0];
  o[1] = (float)v[1];
  o[2] = (float)v[2];
}

template <class Real>
__global__ void k_add_to_sum(long long n, const Vec4<Real>* J, Vec4<float>* jsum, bool first) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  Vec4<float> o;
  if (first) {
    o.x = 0;
    o.y = 0;
    o.z = 0;
    o.w = 0;
  } else {
    o = jsum[t];
  }
  const Vec4<Real> j = J[t];
  o.x += (float)j.x;
  o.y += (float)j.y;
  o.z += (float)j.z;
  jsum[t] = o;
}

template <class Real>
__global__ void k_export(long long n, const Vec4<Real>* tab, float* out) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const Vec4<Real> v = tab[t];
  out[3 * t] = (float)v.x;
  out[3 * t + 1] = (float)v.y;
  out[3 * t + 2] = (float)v.z;
}

static inline dim3 grid1(long long n, int block, int B) { return dim3((unsigned)((n + block - 1) / block), B); }

template <class Real>
void launch_accumulate4(const BuildDims& d, const SetupBuffers<Real>& maps, const Vec4<Real>* a, const Vec4<Real>* b,
                        Vec4<Real>* out, cudaStream_t st) {
  k_accumulate4<Real><<<grid1(d.n4(), 256, d.B), 256, 0, st>>>(d, maps.rowmap, maps.prow, maps.angle, a, b, out);
}

template <class Real>
void launch_accumulate2(int B, int n0, int n1, const Remap2<Real>* remap, const Vec4<Real>* a, const Vec4<Real>* b,
                        Vec4<Real>* out, cudaStream_t st) {
  k_accumulate2<Real><<<grid1((long long)n0 * n1, 256, B), 256, 0, st>>>(n0, n1, remap, a, b, out);
}

template <class Real>
void launch_output4(const BuildDims& d, const SetupBuffers<Real>& maps, const Vec4<Real>* tab, float* out,
                    cudaStream_t st) {
  k_output4<Real><<<grid1(d.n4(), 256, d.B), 256, 0, st>>>(d, maps.rowmap, maps.prow, maps.angle, tab, out);
}

template <class Real>
void launch_output2(int B, int n0, int n1, const Remap2<Real>* remap, const Vec4<Real>* tab, float* out,
                    cudaStream_t st) {
  k_output2<Real><<<grid1((long long)n0 * n1, 256, B), 256, 0, st>>>(n0, n1, remap, tab, out);
}

template <class Real>
void launch_add_to_sum(long long n, const Vec4<Real>* J, Vec4<float>* jsum, bool first, cudaStream_t st) {
  k_add_to_sum<Real><<<grid1(n, 256, 1), 256, 0, st>>>(n, J, jsum, first);
}

template <class Real>
void launch_export(long long n, const Vec4<Real>* tab, float* out, cudaStream_t st) {
  k_export<Real><<<grid1(n, 256, 1), 256, 0, st>>>(n, tab, out);
}

#define SFSIM_INSTANTIATE(Real)                                                                                     \
  template void launch_accumulate4<Real>(const BuildDims&, const SetupBuffers<Real>&, const Vec4<Real>*,           \
                                         const Vec4<Real>*, Vec4<Real>*, cudaStream_t);                            \
  template void launch_accumulate2<Real>(int, int, int, const Remap2<Real>*, const Vec4<Real>*, const Vec4<Real>*, \
                                         Vec4<Real>*, cudaStream_t);                                               \
  template void launch_output4<Real>(const BuildDims&, const SetupBuffers<Real>&, const Vec4<Real>*, float*,       \
                                     cudaStream_t);                                                                \
  template void launch_output2<Real>(int, int, int, const Remap2<Real>*, const Vec4<Real>*, float*, cudaStream_t);  \
  template void launch_export<Real>(long long, const Vec4<Real>*, float*, cudaStream_t);                           \
  template void launch_add_to_sum<Real>(long long, const Vec4<Real>*, Vec4<float>*, bool, cudaStream_t);

SFSIM_INSTANTIATE(float)
SFSIM_INSTANTIATE(double)

}  // namespace sfsim
