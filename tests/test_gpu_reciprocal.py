"""recip_1_2 of the FP32 logistic kernel is the correctly rounded reciprocal for every float of [1, 2]."""
import os
import subprocess

import pytest

torch = pytest.importorskip("torch")

from numpyro_gb300 import build as B  # noqa: E402

SOURCE = r"""
#include <cstdio>
#include "logreg_fp32.cuh"
__global__ void compare(unsigned long long* wrong) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > (1u << 23)) return;
  const float d = __uint_as_float(0x3f800000u + i);
  if (__float_as_uint(gbn::recip_1_2(d)) != __float_as_uint(1.0f / d)) atomicAdd(wrong, 1ull);
}
int main() {
  unsigned long long* wrong = nullptr;
  unsigned long long n = ~0ull;
  if (cudaMalloc(&wrong, sizeof n) != cudaSuccess || cudaMemset(wrong, 0, sizeof n) != cudaSuccess) return 2;
  compare<<<(1 << 23) / 256 + 1, 256>>>(wrong);
  if (cudaMemcpy(&n, wrong, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu\n", n);
  return 0;
}
"""


@pytest.mark.gpu
def test_every_float_from_1_to_2(tmp_path):
    src, exe = str(tmp_path / "recip.cu"), str(tmp_path / "recip")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([B.nvcc()] + B.ARCH + B.NVCC_FLAGS + [src, "-o", exe], check=True, env=dict(os.environ))
    done = subprocess.run([exe], check=True, capture_output=True, text=True)
    assert int(done.stdout) == 0
