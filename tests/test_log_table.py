"""The Poisson sums' logarithm by table, compiled for the host (its operations
are correctly rounded ones, the same on both sides), against long double: from
2^-51, below the smallest 1 - x.y the sums take (1e-15), to 2, at the table's
interval ends, powers of two and arguments next to 1.

Tolerance: relative 1.5 * 2^-53 by the derivation beside the function, 1/32
more for its terms of order r^2; rms 2^-53 / sqrt(3), that of a rounding error
spread evenly over its whole range."""
import os
import shutil
import subprocess
import textwrap

import pytest

from conftest import ROOT

PROGRAM = textwrap.dedent(r"""
    #include <cstdio>
    #include <random>

    #include "log_table.cuh"

    using namespace sbslpm;

    int main() {
      const std::vector<double> t = log_table();
      const double2* cv = reinterpret_cast<const double2*>(t.data());
      const double* lo = t.data() + 2 * kLogN;
      std::mt19937_64 rng(3);
      std::uniform_real_distribution<double> uniform(0, 1);
      double worst = 0, at = 0;
      long double square = 0;
      long n = 0, random = 0;
      auto check = [&](double a, bool counted) {
        const double got = table_log(a, cv, lo);
        if (a == 1.0) {
          if (got != 0) worst = 1, at = a;
          return;
        }
        const long double want = std::log((long double)a);
        const double e = (double)(((long double)got - want) / want);
        n++;
        if (counted) square += (long double)e * e, random++;
        if (!(std::fabs(e) <= worst)) worst = std::fabs(e), at = a;
      };
      for (int k = 0; k < 1000000; k++) {
        check(2 * (1 - uniform(rng)), true);                       // as 1 - x.y of scattered points
        check(std::ldexp(1 + uniform(rng), -1 - (k % 51)), true);  // every power down to 2^-51
      }
      for (int e = -51; e <= 1; e++)
        for (int i = 0; i < kLogN; i++) {
          const double a = std::ldexp(with_high_word(0.0, kLogFirst + (i << (20 - kLogBits))), e + 1);
          for (double b : {std::nextafter(a, 0.0), a, std::nextafter(a, 4.0)})
            if (b <= 2) check(b, false);
        }
      for (int k = 1; k < 200000; k++)
        for (double s : {-1.0, 1.0}) {
          check(1 + s * std::ldexp((double)k, -53), false);
          check(1 + s * std::ldexp(uniform(rng), -(k % 50)), false);
        }
      const double rms = (double)std::sqrt(square / random), u = std::ldexp(1.0, -53);
      std::printf("%ld values: worst %.3g at %a, rms %.3g\n", n, worst, at, rms);
      return worst <= 1.5 * u * (1 + 1.0 / 32) && rms <= u / std::sqrt(3.0) ? 0 : 1;
    }
""")


def test_table_log_error(tmp_path):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("the CUDA headers are not installed")
    src, exe = tmp_path / "log.cpp", tmp_path / "log"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-w", f"-I{cuda}", f"-I{ROOT}/spectral-bslpm_b200/csrc",
                    f"-I{ROOT}/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(out.stdout)
    assert out.returncode == 0, out.stdout
