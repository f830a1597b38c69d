"""A launch that the runtime refuses is reported by the call and does not stay behind as the thread's last error, where the next
check of another library that shares the runtime would find it."""

import os
import shutil
import subprocess

import pytest

from rbf_attention_b200 import build

SOURCE = r"""
#include <cstdio>
#include "launch.h"
__global__ void kernel(float* x) { x[0] = 1.f; }
int main() {
  const cudaError_t e = rbf::launch_dependent(kernel, dim3(1), 4096 /* threads: too many */, 0, nullptr, static_cast<float*>(nullptr));
  std::printf("%d %d", static_cast<int>(e), static_cast<int>(cudaPeekAtLastError()));
  return 0;
}
"""


@pytest.mark.gpu             # (without a driver the runtime's own start-up error cannot be taken back)
def test_a_refused_launch_leaves_no_error_behind(tmp_path):
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    (tmp_path / "launch.cu").write_text(SOURCE)
    program = str(tmp_path / "launch")
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-O0", f"-I{build.CSRC}", str(tmp_path / "launch.cu"), "-o", program], check=True,
                   env={**os.environ, "TMPDIR": str(tmp_path)}, capture_output=True)
    returned, left = subprocess.run([program], check=True, capture_output=True, text=True).stdout.split()
    assert int(returned) == 9 and int(left) == 0        # cudaErrorInvalidConfiguration
