"""launch_after (csrc/common.cuh) takes what a call of the kernel would take and nothing else. Compiled, not run: no GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

CODE = r"""
#include "common.cuh"
#include <utility>
using namespace epsp;
__global__ void k(const double* in, float* out, long n, double4 v, bool on, const double* maybe) { pdl_wait(); }
double* d; const double* cd; float* f; const float* cf; int i; unsigned char* u; double4 v;
template <class... A>
auto takes_t(int, A&&... a) -> decltype(launch_after(cudaStream_t(), k, dim3(1), dim3(1), 0, std::forward<A>(a)...), char(0));
template <class... A>
int takes_t(long, A&&...);
#define TAKES(...) (sizeof(takes_t(0, __VA_ARGS__)) == 1)
static_assert(TAKES(d, f, i, v, true, nullptr), "as a call: const added, int to long, nullptr");
static_assert(TAKES(cd, f, 3u, v, i > 0, cd), "as a call");
static_assert(!TAKES(f, f, i, v, true, nullptr), "float* for const double*");
static_assert(!TAKES(d, d, i, v, true, nullptr), "double* for float*");
static_assert(!TAKES(d, cf, i, v, true, nullptr), "const lost");
static_assert(!TAKES(d, f, i, v, true, u), "unsigned char* for const double*");
static_assert(!TAKES(d, f, f, v, true, nullptr), "a pointer for a number");
static_assert(!TAKES(d, i, i, v, true, nullptr), "a number for a pointer");
static_assert(!TAKES(d, f, i, v, true), "an argument short");
"""


def test_arguments_convert_as_in_a_call(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "launch_types.cu"
    src.write_text(CODE)
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.join(PKG, "csrc"),
                        "-c", str(src), "-o", str(tmp_path / "launch_types.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
