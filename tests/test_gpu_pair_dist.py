"""The distance that picks a mean-force bin (pair_dist) and the correctly rounded root
it stands for, which the oracle and the adjoint take: the table jumps at half-bin
edges, so one ulp moves a bin.  Compared for every float between 1e-6 and 1e4 A^2
(a thousandth of an angstrom to a hundred), in a program built with the library's
flags."""
import subprocess

import pytest

import build as engine_build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "device_common.cuh"
__global__ void differ(unsigned lo, unsigned hi, unsigned long long *out) {
    unsigned long long bad = 0;
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned long long b = lo + blockIdx.x * blockDim.x + threadIdx.x; b <= hi; b += stride) {
        const float d2 = __uint_as_float((unsigned)b);
        bad += __float_as_uint(isspa::pair_dist(d2, rsqrtf(d2))) != __float_as_uint(__fsqrt_rn(d2));
    }
    atomicAdd(out, bad);
    atomicAdd(out + 1, 1ull);
}
int main() {
    const float lo = 1e-6f, hi = 1e4f;
    unsigned l, h;
    memcpy(&l, &lo, 4);
    memcpy(&h, &hi, 4);
    unsigned long long *d, r[2] = {0, 0};
    if (cudaMalloc(&d, sizeof r) != cudaSuccess || cudaMemset(d, 0, sizeof r) != cudaSuccess) return 1;
    differ<<<1024, 256>>>(l, h, d);
    if (cudaMemcpy(r, d, sizeof r, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::printf("%u %llu %llu\n", h - l + 1, r[0], r[1]);
    return 0;
}
"""


def test_pair_dist_is_the_rounded_root(tmp_path):
    src, exe = tmp_path / "pair_dist.cu", tmp_path / "pair_dist"
    src.write_text(PROGRAM)
    subprocess.run([engine_build.nvcc()] + engine_build._flags() + [str(src), "-o", str(exe)], check=True)
    values, differ, threads = map(int, subprocess.run([str(exe)], check=True, capture_output=True,
                                                      text=True).stdout.split())
    assert values > 270_000_000 and threads == 1024 * 256
    assert differ == 0
