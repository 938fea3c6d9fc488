"""The activation functions of the GEMM epilogues against 64-bit values, in 32 bits (a layer's 16-bit results would hide the loss
of half the bits).  The bounds follow from the documented errors of what the functions are made of."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = """
#include "common.cuh"
__global__ void run(const float* x, float* s, float* silu, float* dsilu, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  s[i] = moe::sigmoidf_fast(x[i]);
  silu[i] = moe::silu_f(x[i]);
  dsilu[i] = moe::dsilu_f(x[i]);
}
extern "C" int activations(const float* x, float* s, float* silu, float* dsilu, int n, void* stream) {
  run<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, s, silu, dsilu, n);
  return static_cast<int>(cudaGetLastError());
}
"""


@pytest.fixture(scope="module")
def activations(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "moe-explore_b200"))
    import build_native

    out = tmp_path_factory.mktemp("activations")
    (out / "a.cu").write_text(SOURCE)
    subprocess.run([build_native._nvcc()] + build_native.NVCC_FLAGS +
                   ["-I", build_native.CSRC, "-shared", "-o", str(out / "a.so"), str(out / "a.cu")], check=True)
    fn = ctypes.CDLL(str(out / "a.so")).activations
    fn.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_int, ctypes.c_void_p]

    def call(x):
        ys = [torch.empty_like(x) for _ in range(3)]
        assert fn(x.data_ptr(), *[y.data_ptr() for y in ys], x.numel(), torch.cuda.current_stream().cuda_stream) == 0
        return [y.double() for y in ys]
    return call


def test_sigmoid_and_silu_to_their_last_places(activations):
    edges = [0.0, -0.0, 20.0, -20.0, 87.0, -87.0, -87.3, -87.4, -88.0, -88.6, 89.0, -89.0, 104.0, -104.0, 1e30, -1e30]
    x = torch.cat([torch.tensor(edges), torch.linspace(-110, 110, 400001), torch.linspace(-4, 4, 400001)]).cuda()
    s, silu, dsilu = activations(x)
    x = x.double()
    e = torch.exp(-x.abs())
    ref = torch.where(x >= 0, 1 / (1 + e), e / (1 + e))
    ulp = 2.0 ** -23
    # __expf(-x) is within 2 + 1.173 |x| units (CUDA's table of intrinsics), and counts by the share of e^-x in 1 + e^-x, which is
    # 1 - sigmoid; the sum and the reciprocal add one unit each.  Past -88.7 e^-x exceeds 32 bits and the result is 0, off by at
    # most 1 / FLT_MAX = 2^-128.
    bound = ref * ulp * (2 + (1 - ref) * (2 + 1.173 * x.abs())) + 2.0 ** -128
    assert bool(((s - ref).abs() <= bound).all())
    # x * s: one more rounding; s (1 + x (1 - s)): the error of s through its derivative, three more roundings of its terms
    assert bool(((silu - x * ref).abs() <= x.abs() * bound + (x * ref).abs() * ulp).all())
    exact = ref * (1 + x * (1 - ref))
    spread = (1 + x - 2 * x * ref).abs() * bound + 3 * ulp * ref * (1 + x.abs() * (1 - ref).clamp_min(ulp))
    assert bool(((dsilu - exact).abs() <= spread).all())


def test_infinities_and_nan(activations):
    s, silu, dsilu = activations(torch.tensor([float("inf"), float("-inf"), float("nan")], device="cuda"))
    assert s[:2].tolist() == [1.0, 0.0] and bool(s[2].isnan())
    assert float(silu[0]) == float("inf") and bool(silu[2].isnan()) and bool(dsilu[2].isnan())
