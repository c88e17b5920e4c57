"""The departure search finds a point's leaf from its cells along the two face
coordinates (leaf_by_cells); the reference's descent through the levels decides
ties on panel boundaries by comparisons of xi and eta together.  Both, compiled
for the host, give the same leaf and bounds on every combination of boundaries
and their neighbouring doubles, and at random points, at levels 1 to 12."""
import os
import shutil
import subprocess
import textwrap

import pytest

from conftest import ROOT

PROGRAM = textwrap.dedent(r"""
    #include <algorithm>
    #include <cmath>
    #include <cstdio>
    #include <random>
    #include <vector>

    #include "geometry.cuh"

    using namespace sbslpm;

    int main() {
      std::mt19937_64 rng(7);
      long points = 0;
      for (int levels = 1; levels <= 12; levels++) {
        const int n = 1 << (levels - 1);
        std::vector<int> cut;  // boundaries: all of a small level, else those of the coarse cuts, the ends and some more
        if (n <= 32) {
          for (int b = 0; b <= n; b++) cut.push_back(b);
        } else {
          for (int b = 0; b <= n; b += n / 16) cut.insert(cut.end(), {b, std::min(b + 1, n), std::max(b - 1, 0)});
          for (int k = 0; k < 20; k++) cut.push_back((int)(rng() % (n + 1)));
        }
        std::vector<double> at;
        for (int b : cut) {
          const double t = kPi / 4.0 * (b * (2.0 / n) - 1.0);
          for (double u : {std::nextafter(t, -1.0), t, std::nextafter(t, 1.0)})
            if (std::fabs(u) <= kPi / 4.0) at.push_back(u);
        }
        std::uniform_real_distribution<double> uniform(-kPi / 4.0, kPi / 4.0);
        for (int k = 0; k < 40; k++) at.push_back(uniform(rng));
        for (double xi : at)
          for (double eta : at)
            for (int face : {0, 5}) {
              unsigned err = 0;
              Bounds a, b;
              const int id = descend_to_leaf(face, xi, eta, levels, a, err);
              const unsigned leaf = leaf_by_cells(xi, eta, levels, b);
              points++;
              if (err || id != level_start(levels - 1) + face * n * n + (int)leaf || a.min_xi != b.min_xi ||
                  a.max_xi != b.max_xi || a.min_eta != b.min_eta || a.max_eta != b.max_eta) {
                std::printf("levels %d face %d xi %.17g eta %.17g: %d, by cells %u\n", levels, face, xi, eta, id, leaf);
                return 1;
              }
            }
      }
      std::printf("%ld points\n", points);
      return points > 500000 ? 0 : 2;
    }
""")


def test_leaf_by_cells_is_the_descents(tmp_path):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("the CUDA headers are not installed")
    src, exe = tmp_path / "location.cpp", tmp_path / "location"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-w", f"-I{cuda}", f"-I{ROOT}/spectral-bslpm_b200/csrc",
                    f"-I{ROOT}/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
