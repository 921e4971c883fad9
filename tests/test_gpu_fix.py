"""The functions of phs_fix.h as the device evaluates them (its own estimates of 1/x and
1/sqrt(x)) against the library's correctly rounded ones."""
import os
import subprocess

import pytest

from gpu_phs_gb300 import build

pytestmark = pytest.mark.gpu

DRIVER = r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "phs_fix.h"
// mantissas next to 1, 2 and 4, where the estimates change their binade, and in between
__global__ void compare(int n, int *rcp, int *root) {
  const FxRegs k = fx_regs();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double x;
    const double c = i & 1 ? 1.0 : (i & 2 ? 2.0 : 4.0);
    switch (i >> 2 & 3) {
      case 0: x = c + c * (i >> 4) * 0x1p-44; break;
      case 1: x = c - c * (1 + (i >> 4)) * 0x1p-45; break;
      case 2: x = c * (1 + (i >> 4) * 0x1p-22); break;
      default: x = __longlong_as_double(__double_as_longlong(c) - 1 - (i >> 4) * 8191ll);
    }
    const long long dr = __double_as_longlong(fx_rcp(x, k)) - __double_as_longlong(__drcp_rn(x));
    const long long ds = __double_as_longlong(fx_sqrt(x, k)) - __double_as_longlong(__dsqrt_rn(x));
    atomicMax(rcp, (int)min(llabs(dr), 1000000ll));
    atomicMax(root, (int)min(llabs(ds), 1000000ll));
  }
}
int main() {
  int *d, h[2] = {-1, -1};
  if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 1;
  compare<<<304, 256>>>(1 << 26, d, d + 1);
  if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  std::printf("%d %d\n", h[0], h[1]);
}
"""


def test_root_and_reciprocal_where_the_estimates_change_binade(tmp_path):
    """Both within an ulp of the correctly rounded value (next to 4 roots lie so near to a rounding
    boundary that fx_sqrt does not promise the last bit)."""
    src, exe = str(tmp_path / "f.cu"), str(tmp_path / "f")
    with open(src, "w") as fh:
        fh.write(DRIVER)
    subprocess.run([build.NVCC, *build.ARCH, "-O2", "-std=c++17", "-I", build.CSRC, src, "-o", exe], check=True)
    rcp, root = subprocess.run([exe], check=True, capture_output=True, text=True,
                               env=dict(os.environ)).stdout.split()
    assert int(rcp) <= 1
    assert int(root) <= 1
