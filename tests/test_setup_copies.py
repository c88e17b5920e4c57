"""Set-up tables are on the device when the call that fills them returns.

A copy from pageable memory may return once its bytes are staged, and a memset
before it has run, and the streams that read the buffers do not wait for the
legacy stream.  Here the CUDA runtime is a stand-in that takes this to the
limit: "device" memory changes only when the stream is waited for."""
import os
import shutil
import subprocess
import textwrap

import pytest

from conftest import ROOT

PROGRAM = textwrap.dedent(r"""
    #include <cstdio>
    #include <cstdlib>
    #include <functional>
    #include <vector>

    #include "context_internal.hpp"

    static std::vector<std::function<void()>> pending;  // the legacy stream's work

    extern "C" {
    cudaError_t cudaMalloc(void** p, size_t n) {
      *p = std::malloc(n);
      std::memset(*p, 0x5a, n);
      return cudaSuccess;
    }
    cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind) {
      std::vector<char> staged((const char*)from, (const char*)from + n);
      pending.push_back([=] { std::memcpy(to, staged.data(), n); });
      return cudaSuccess;
    }
    cudaError_t cudaMemset(void* to, int v, size_t n) {
      pending.push_back([=] { std::memset(to, v, n); });
      return cudaSuccess;
    }
    cudaError_t cudaStreamSynchronize(cudaStream_t st) {
      if (st == nullptr)
        for (auto& f : pending) f();
      pending.clear();
      return cudaSuccess;
    }
    const char* cudaGetErrorString(cudaError_t) { return ""; }
    }
    namespace sbslpm {
    void set_last_error(const std::string&) {}
    }  // namespace sbslpm

    int main() {
      using namespace sbslpm;
      const std::vector<double> h = {1.5, -2.0, 3.25};
      double* table = nullptr;
      if (upload(&table, h) != SBSLPM_OK || std::memcmp(table, h.data(), sizeof(double) * h.size())) return 1;
      double* none = table;
      if (upload(&none, std::vector<double>()) != SBSLPM_OK || none) return 2;
      float4* packed = nullptr;
      if (alloc_packed(&packed, 3, 9) != SBSLPM_OK) return 3;
      for (int k = 0; k < 3 * packed_stride(9); k++)
        if (packed[k].x != 0 || packed[k].w != 0) return 4;
      return 0;
    }
""")


def test_set_up_waits_for_its_copies(tmp_path):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("the CUDA headers are not installed")
    src, exe = tmp_path / "copies.cpp", tmp_path / "copies"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-w", f"-I{cuda}", f"-I{ROOT}/spectral-bslpm_b200/csrc", f"-I{ROOT}/include",
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
