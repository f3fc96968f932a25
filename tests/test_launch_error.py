"""A refused kernel launch is reported once: launch_k (csrc/common.cuh) returns its error and leaves the
thread's last error clear, so the cudaGetLastError() after the next launch does not report it again.
The runtime refuses a block of 4096 threads on the host; without a driver every call reports the missing
driver, so this needs a device."""
import os
import subprocess
import tempfile

import pytest

from fluxo_b200 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "common.cuh"
__global__ void k(int) {}
int main() {
  for (int pdl = 0; pdl < 2; ++pdl) {
    const cudaError_t e = fluxo::launch_k(pdl != 0, k, 1u, 4096u, 0, (cudaStream_t)0, 1);
    std::printf("%d %d\n", e != cudaSuccess, cudaGetLastError() != cudaSuccess);
  }
}
"""


@pytest.mark.timeout(120)
def test_refused_launch_is_reported_once(gpu_lib):
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cu"), os.path.join(d, "t")
        with open(src, "w") as f:
            f.write(PROGRAM)
        subprocess.run([build._nvcc()] + build.NVCC_FLAGS + [src, "-o", exe], check=True, capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["1", "0"] * 2
