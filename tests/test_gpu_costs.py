"""Block matching's two evaluations of one cost (csrc/level.cuh): a run's first test evaluates two vectors as the
lanes of packed arithmetic, the next ones a vector each, and the sweep compares the ones with the others. Both must
give the same bits, in the strict build and in the fast mode's: a small program of the two, built with each one's
flags."""
import subprocess

import pytest

from twixtor_b200 import buildlib

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "kernels.cuh"
#include "level.cuh"
constexpr int W = 64, H = 64, N = 1 << 16;
__device__ unsigned rnd(unsigned& s) { s = s * 1664525u + 1013904223u; return s >> 8; }
__device__ float unit(unsigned& s) { return (float)rnd(s) / 16777216.0f; }
__global__ void fill(float* b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned s = i * 2654435761u + 1;
    if (i < W * H) b[i] = 255.0f * (unit(s) - 0.5f);
}
template <bool COLS>
__device__ bool differ(const float* b, unsigned s, float z) {
    float p[9];
    for (int k = 0; k < 9; k++) p[k] = 255.0f * (unit(s) - 0.5f);
    const float2 fx = make_float2(unit(s), rnd(s) % 4 ? unit(s) : 1.0f), fy = make_float2(rnd(s) % 4 ? unit(s) : 0.0f, unit(s));
    const int at0 = rnd(s) % (H - 3) * W + rnd(s) % (W - 3), at1 = rnd(s) % (H - 3) * W + rnd(s) % (W - 3);
    const float2 c = tw::bm_cost2<COLS>(b, W, p, fx, fy, at0, at1, z);
    const float c0 = tw::bm_cost1<COLS>(b, W, p, fx.x, fy.x, at0), c1 = tw::bm_cost1<COLS>(b, W, p, fx.y, fy.y, at1);
    return !tw::same_bits(c, make_float2(c0, c1));
}
__global__ void check(const float* b, float z, int* bad) {
    unsigned s = (blockIdx.x * blockDim.x + threadIdx.x) * 747796405u + 7;
    if (differ<false>(b, s, z) || differ<true>(b, s + 99, z)) atomicAdd(bad, 1);
}
int main() {
    float* b;
    int *bad, n = -1;
    cudaMalloc(&b, W * H * sizeof(float));
    cudaMalloc(&bad, sizeof(int));
    cudaMemset(bad, 0, sizeof(int));
    fill<<<W * H / 256, 256>>>(b);
    check<<<N / 256, 256>>>(b, -0.0f, bad);
    cudaMemcpy(&n, bad, sizeof n, cudaMemcpyDeviceToHost);
    printf("%s %d\n", cudaGetErrorString(cudaGetLastError()), n);
}
"""


@pytest.mark.parametrize("fast", [False, True])
def test_both_evaluations_of_a_cost_give_the_same_bits(fast, tmp_path):
    flags = [f for f in buildlib.FLAGS if f not in ("-shared", "-cudart", "shared")]
    if fast:
        flags = buildlib.fast_flags(flags)
    (tmp_path / "costs.cu").write_text(SOURCE)
    subprocess.run([buildlib.NVCC] + flags + ["-I", buildlib.CSRC, "-o", str(tmp_path / "costs"), str(tmp_path / "costs.cu")],
                   check=True)
    r = subprocess.run([str(tmp_path / "costs")], capture_output=True, text=True, check=True)
    assert r.stdout.strip() == "no error 0"
