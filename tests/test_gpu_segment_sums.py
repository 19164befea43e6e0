"""segment_depth_warp (the optical depth to point scatter's ground points, a
warp a segment) sums its samples as segment_depth does, compensated: against
the same FP32 samples added in FP64 the sum is within Kahan's bound, two units
roundoff (2 * 2^-24) of its value, whatever the number of samples."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "atmo_device.cuh"
using namespace sfsim;

// one warp a case: the depth of unit extinction and unit sample length is the sum itself
__global__ void sums(const AtmoParams* P, int steps, int cases, double* worst) {
  const int c = blockIdx.x, lane = threadIdx.x;
  const d3 x = mk3(P->R + 90.0 * (c % 97), 0, 0);
  const d3 D = mul3(mk3(-0.8 + 1.7 * c / cases, 0.6 + 0.3 * c / cases, 0.1), (double)steps);
  const d3 unit = mul3(D, steps / mag3(D));
  float tau[3];
  segment_depth_warp<float>(*P, x, unit, steps, lane, tau);
  const double c0 = (mag3(x) - P->R) * (mag3(x) + P->R), du = 1.0 / steps;
  const QForm f = segment_q_form(c0, dot3(x, unit), dot3(unit, unit), du);
  double exact = 0;
  for (int n = 0; n < steps; n++) {
    const float w = fmaf((float)n, (float)du, (float)f.w0);
    const float q = fmaf(w, fmaf(w, (float)f.C, (float)f.B), (float)f.A);
    const float h = height_from_q<float, 5>(q, P->f_hpoly, P->f_alpha, P->f_beta);
    exact += (double)Bulk<float>::exp2(h * P->f_kr);
  }
  const float length = (float)(mag3(unit) / steps);
  if (lane == 0) worst[c] = length == 1.0f ? fabs(tau[0] / exact - 1.0) * 16777216.0 : 0.0;
}

int main() {
  AtmoParams h;
  memset(&h, 0, sizeof h);
  h.R = 6378000.0;
  h.f_ray_ext[0] = 1.0f;
  h.f_kr = -0.01f;
  h.f_km = -0.01f;
  h.f_hpoly[0] = 1.0f / (2.0f * 6378000.0f);
  AtmoParams* P;
  double* w;
  const int cases = 4096;
  cudaMalloc(&P, sizeof h);
  cudaMalloc(&w, cases * sizeof(double));
  cudaMemcpy(P, &h, sizeof h, cudaMemcpyHostToDevice);
  for (int steps : {24, 33, 64, 100, 128, 1000}) {
    sums<<<cases, 32>>>(P, steps, cases, w);
    static double r[cases];
    if (cudaMemcpy(r, w, sizeof r, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    double worst = 0;
    int used = 0;
    for (double v : r) worst = v > worst || v != v ? v : worst, used += v > 0;
    printf("%d %d %.4f\n", steps, used, worst);
  }
  return 0;
}
"""


def test_within_two_roundoffs(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "sums.cu", tmp_path / "sums"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(root, "sfsim_gb300", "csrc"), "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True).stdout.split("\n")
    rows = [line.split() for line in out if line]
    assert len(rows) == 6
    for steps, used, worst in rows:
        assert int(used) > 1000 and float(worst) <= 2.0, (steps, used, worst)
