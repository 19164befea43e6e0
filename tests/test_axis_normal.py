"""Point scatter's directions are unit vectors for every radius that a
configuration may have.

It forms offsets into shared memory from a direction's cosine with the light,
so a direction that is no unit vector (radii whose squares overflow or vanish
gave NaN) reads outside its tables.  Host code of the device functions: the
frame at every height and the directions of a ring, over radii from 1e-300 to
1e300 with thin and thick atmospheres, and the products of what the ground
term's sun elevation is formed from."""
import os
import shutil
import subprocess

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "atmo_device.cuh"
using namespace sfsim;

int main() {
  int bad = 0, cases = 0;
  for (int e = -300; e <= 300; e++)
    for (double thick : {1e-30, 1e-12, 1e-3, 0.05}) {
      AtmoParams P;
      memset(&P, 0, sizeof P);
      P.R = 3.7 * pow(10.0, e), P.H = P.R * thick, P.top = P.R + P.H;
      if (!(P.H > 0) || !std::isfinite(P.top)) continue;
      P.R2 = P.R * P.R, P.top2 = P.top * P.top, P.Hh = sqrt(P.top2 - P.R2), P.Hh2 = P.Hh * P.Hh;
      for (int i = 0; i < 5; i++) {
        const d3 x = mk3(index_to_radius(P, 5, (double)i), 0, 0);
        const d3 n = axis_normal(P, x), o1 = orthogonal(n), o2 = cross3(n, o1);
        for (int k = 0; k < 12; k++) {
          const double t = 0.1 + 0.25 * k, p = 0.7 * k;
          const d3 w = to_world(n, o1, o2, DirLocal{cos(t), sin(t) * cos(p), sin(t) * sin(p), 1.0});
          const double m = mag3(w);
          bad += !(m > 1 - 1e-9 && m < 1 + 1e-9);
          cases++;
        }
        // the sun elevation's sine at the ground point of a ray straight down: 1 for a light overhead
        if (ordinary_radii(P)) {
          const double down = (x.x - P.R) / P.R, sine = x.x / P.R - down;
          bad += !(sine > 1 - 1e-9 && sine < 1 + 1e-9);
        }
      }
    }
  printf("%d %d\n", cases, bad);
  return 0;
}
"""


def test_directions_are_unit_vectors(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src, exe = tmp_path / "axis.cu", tmp_path / "axis"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(root, "sfsim_gb300", "csrc"), "-o", str(exe), str(src)], check=True)
    cases, bad = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120, check=True).stdout.split()
    assert int(cases) > 50000 and int(bad) == 0, (cases, bad)
