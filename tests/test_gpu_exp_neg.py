"""exp_neg_slab itself (rg_exp.cuh), compiled into a kernel of the test: bit for bit the float nearest to double
precision's exp(-sig dt) for every density sum whose product lies in [2e-4, 1/4], with the eight samples of a slab
near each other and spread over the range, and in slabs that mix them with zeros, sums beyond 1/4 and infinity."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT

pytestmark = pytest.mark.gpu
CSRC = os.path.join(ROOT, "ray_gauss_b200", "csrc")
SOURCE = r"""
#include "rg_exp.cuh"
using namespace rg;
// Slab i of n: sample k has the density sum with bits first + i + k * stride, or special[k] where its bit of `mix` is set.
__global__ void k_check(unsigned first, unsigned n, unsigned stride, unsigned mix, const float* special, f2 nz,
                        unsigned long long* wrong) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float sig[kBuf];
    for (int k = 0; k < kBuf; ++k) sig[k] = (mix >> k) & 1u ? special[k] : __uint_as_float(first + i + k * stride);
    f2 in[kPairs], out[kPairs];
    for (int p = 0; p < kPairs; ++p) in[p] = pk(sig[2 * p], sig[2 * p + 1]);
    exp_neg_slab(in, out, nz);
    unsigned bad = 0;
    for (int k = 0; k < kBuf; ++k) {
        const float want = (float)exp(-(double)__fmul_rn(sig[k], kDt));
        bad += __float_as_uint(rg::half2(out[k >> 1], k & 1)) != __float_as_uint(want);
    }
    if (bad) atomicAdd(wrong, (unsigned long long)bad);
}
extern "C" int check(unsigned first, unsigned n, unsigned stride, unsigned mix, const float* special, unsigned long long* wrong) {
    k_check<<<(n + 255) / 256, 256>>>(first, n, stride, mix, special, 0x8000000080000000ull, wrong);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("exp")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", CSRC, "-I", os.path.join(ROOT, "include"), str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    lib = ctypes.CDLL(str(d / "t.so"))
    lib.check.argtypes = [ctypes.c_uint32] * 4 + [ctypes.c_void_p] * 2

    def run(first, n, stride, mix=0, special=(0.0,) * 8):
        wrong = torch.zeros(1, dtype=torch.int64, device="cuda")
        sp = torch.tensor(special, dtype=torch.float32, device="cuda")
        assert lib.check(first, n, stride, mix, sp.data_ptr(), wrong.data_ptr()) == 0
        return int(wrong)
    return run


FIRST, LAST = (int(np.float32(v).view(np.uint32)) for v in (0.08, 100.0))   # sums whose product with dt is in the range


def test_every_sum_of_the_range(cuda, check):
    n = LAST - FIRST + 1
    assert n > 80_000_000
    assert check(FIRST, n - 7, 1) == 0                    # neighbours in a slab
    assert check(FIRST, n // 8, n // 8) == 0              # a slab's samples spread over the range


@pytest.mark.parametrize("mix,special", [
    (0b10101010, (0.0,) * 8), (0b00000001, (0.0,) * 8), (0b01111111, (0.0,) * 8),
    (0b00100000, (100.1,) * 8), (0b11000011, (5000.0, 40000.0, 0.0, 0.0, 0.0, 0.0, 101.0, 3e38)),
    (0b00010010, (0.0, float("inf"), 0.0, 0.0, float("inf"), 0.0, 0.0, 0.0))])
def test_mixed_slabs(cuda, check, mix, special):
    assert check(FIRST, LAST - FIRST - 7 * 1009, 1009, mix, special) == 0
