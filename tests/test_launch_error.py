"""A pass kernel that cannot be launched: the call returns the error, and the
runtime's last error is as if nothing had happened (the caller's next check of
its own launches does not find it).  pfgb_launch.h compiled with g++ against a
fake of the two runtime calls."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pencilffts.jl_gb300" / "csrc"

FAKE = r"""
#pragma once
#include <cstddef>
#include <cstdint>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidConfiguration = 9 };
typedef void* cudaStream_t;
struct dim3 { unsigned x, y, z; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
enum cudaLaunchAttributeID { cudaLaunchAttributeProgrammaticStreamSerialization };
struct cudaLaunchAttribute { cudaLaunchAttributeID id; struct { int programmaticStreamSerializationAllowed; } val; };
struct cudaLaunchConfig_t {
  dim3 gridDim, blockDim;
  size_t dynamicSmemBytes;
  cudaStream_t stream;
  cudaLaunchAttribute* attrs;
  unsigned numAttrs;
};
inline cudaError_t last_error = cudaSuccess;
inline cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
template <typename A>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t* c, void (*)(A), const A&) {
  return c->blockDim.x > 1024 ? last_error = cudaErrorInvalidConfiguration : cudaSuccess;
}
"""

DRIVER = r"""
#include "pfgb_launch.h"
static void kernel(int) {}
int main() {
  if (pfgb::launch_pass_kernel(kernel, 1, 128, 0, nullptr, 1) != cudaSuccess) return 1;
  if (pfgb::launch_pass_kernel(kernel, 1, 4096, 0, nullptr, 1) != cudaErrorInvalidConfiguration) return 2;
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_failed_launch_leaves_no_error_behind(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "launch.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", str(CSRC), str(tmp_path / "launch.cpp"), "-o",
                    str(tmp_path / "launch")], check=True)
    assert subprocess.run([str(tmp_path / "launch")]).returncode == 0
