"""step_launch (csrc/common.cuh) checks a kernel's arguments as a <<<>>> launch does:
what converts implicitly is taken, a pointer of another type or a dropped const is
not.  Compiled here, never run.
"""
import shutil
import subprocess

import pytest

from conftest import PKG

CODE = """
#include "common.cuh"
#include <utility>
template <typename... A>
constexpr auto launches(int) -> decltype(ehd::step_launch(
    (void (*)(const double *, float *, int, double))nullptr, dim3(1), dim3(1), size_t(0),
    cudaStream_t(nullptr), std::declval<A>()...), true) { return true; }
template <typename... A> constexpr bool launches(long) { return false; }
static_assert(launches<const double *, float *, int, double>(0), "the parameters themselves");
static_assert(launches<double *, float *, long long, float>(0), "implicit conversions");
static_assert(launches<std::nullptr_t, float *, int, int>(0), "null pointers");
static_assert(!launches<float *, float *, int, double>(0), "another pointer type");
static_assert(!launches<const double *, const float *, int, double>(0), "a dropped const");
static_assert(!launches<float *, const double *, int, double>(0), "swapped pointers");
static_assert(!launches<const double *, float *, float *, double>(0), "a pointer as a number");
static_assert(!launches<const double *, float *, int>(0), "too few");
"""


def test_launch_arguments_are_checked(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "launch.cu"
    src.write_text(CODE)
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                        "--expt-relaxed-constexpr", "-I", str(PKG / "csrc"), "-I",
                        str(PKG.parent / "include"), "-c", str(src), "-o", str(tmp_path / "launch.o")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
