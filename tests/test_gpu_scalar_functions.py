"""The kernels' own reciprocals and logarithm on the device, value by value.

Tolerances, relative: recip_nr the last rounding's 2^-53 and the cube of the
hardware approximation's 2^-20, together 2^-53 (1 + 2^-7); recip_full 2^-53
(1 + 2^-50); both checked on the residual 1 - d r, which one fused multiply-add
gives to 2^-53 of itself (the bounds here allow 2^-6 and 2^-20).  table_log
1.5 * 2^-53 (1 + 1/32) as derived beside it, against torch's log, whose own
error is at most one unit (CUDA's documented bound), 2^-52."""
import ctypes
import os
import subprocess
import textwrap

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
NVCC = "/usr/local/cuda/bin/nvcc"

SOURCE = textwrap.dedent(r"""
    #include "device_common.cuh"
    #include "log_table.cuh"
    using namespace sbslpm;

    __global__ void k_recip(long n, const double* d, double* nr, double* full, double* res_nr, double* res_full) {
      const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
      if (i >= n) return;
      nr[i] = dev::recip_nr(d[i]);
      full[i] = dev::recip_full(d[i]);
      res_nr[i] = fma(-d[i], nr[i], 1.0);
      res_full[i] = fma(-d[i], full[i], 1.0);
    }

    __global__ void k_log(long n, const double* a, const double* table, double* out) {
      const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
      if (i < n) out[i] = table_log(a[i], reinterpret_cast<const double2*>(table), table + 2 * kLogN);
    }

    extern "C" int run_recip(long n, const double* d, double* nr, double* full, double* res_nr, double* res_full) {
      k_recip<<<dev::blocks_for(n, 256), 256>>>(n, d, nr, full, res_nr, res_full);
      return cudaDeviceSynchronize();
    }
    extern "C" int log_table_size() { return (int)log_table().size(); }
    extern "C" void fill_log_table(double* to) {
      const std::vector<double> t = log_table();
      std::memcpy(to, t.data(), sizeof(double) * t.size());
    }
    extern "C" int run_log(long n, const double* a, const double* table, double* out) {
      k_log<<<dev::blocks_for(n, 256), 256>>>(n, a, table, out);
      return cudaDeviceSynchronize();
    }
""")


@pytest.fixture(scope="module")
def functions(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("scalar")
    (d / "f.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", f"-I{ROOT}/spectral-bslpm_b200/csrc", f"-I{ROOT}/include",
                    str(d / "f.cu"), "-o", str(d / "libf.so")], check=True)
    return ctypes.CDLL(str(d / "libf.so"))


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def test_reciprocals(functions):
    rng = np.random.default_rng(5)
    n = 1 << 21
    mantissa = 1 + rng.random(n)
    mantissa[:4096] = 1 + np.arange(4096) * 2.0 ** -52  # just above a power of two, and just below
    mantissa[4096:8192] = 2 - (1 + np.arange(4096)) * 2.0 ** -52
    d = torch.from_numpy(np.ldexp(mantissa, rng.integers(-900, 900, n)) * rng.choice([-1.0, 1.0], n)).cuda()
    out = [torch.empty_like(d) for _ in range(4)]
    assert functions.run_recip(ctypes.c_long(n), ptr(d), *[ptr(o) for o in out]) == 0
    u = 2.0 ** -53
    assert float(out[2].abs().max()) <= u * (1 + 2.0 ** -6)
    assert float(out[3].abs().max()) <= u * (1 + 2.0 ** -20)
    assert float(((out[0] - 1 / d) * d).abs().max()) <= 2 * u * (1 + 2.0 ** -6)
    assert float(((out[1] - 1 / d) * d).abs().max()) <= 2 * u * (1 + 2.0 ** -20)


def test_table_log(functions):
    rng = np.random.default_rng(6)
    k = np.arange(1, 100001)
    near = np.ldexp(rng.random(400000), -(np.arange(400000) % 50))
    a = np.concatenate([2 * rng.random(1 << 20) + 1e-15, np.ldexp(1 + rng.random(1 << 20), rng.integers(-51, 1, 1 << 20)),
                        np.ldexp(1.0, np.arange(-51, 2)), 1 + k * 2.0 ** -52, 1 - k * 2.0 ** -53, 1 + near, 1 - near,
                        [1.0]])
    a = torch.from_numpy(a[(a >= 2.0 ** -51) & (a <= 2)]).cuda()
    table = np.empty(functions.log_table_size())
    functions.fill_log_table(ctypes.c_void_p(table.ctypes.data))
    table = torch.from_numpy(table).cuda()
    got = torch.empty_like(a)
    torch.cuda.synchronize()
    assert functions.run_log(ctypes.c_long(a.numel()), ptr(a), ptr(table), ptr(got)) == 0
    want = torch.log(a)
    assert not got[a == 1].any()
    at = a != 1
    bound = (1.5 * (1 + 1 / 32) + 2) * 2.0 ** -53 * want[at].abs()
    assert bool(((got[at] - want[at]).abs() <= bound).all())
