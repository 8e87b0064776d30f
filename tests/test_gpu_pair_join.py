"""The float pairs' join into doubles on the integer pipe (f2_to_double,
fargocpt_gb300/csrc/fp64_pair.cuh) against numpy's h + l in FP64, which rounds
the same exact sum once: equal bit patterns for every pair a pair operation
leaves (|l| at most ulp(h)), over h from 2^-74 to 2^127, powers of two of both
signs with low parts on either side (the binade below), ties, zero low parts,
and zero, infinite and NaN high parts.  A small program with the header's
device function, compiled with nvcc."""
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <vector>
#include "fp64_pair.cuh"
__global__ void k(const float2 *a, double *o, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) o[i] = fgpu::f2_to_double(fgpu::f2{a[i].x, a[i].y});
}
int main(int, char **v)
{
    FILE *f = fopen(v[1], "rb");
    fseek(f, 0, SEEK_END);
    const int n = (int)(ftell(f) / 8);
    rewind(f);
    std::vector<float2> h(n);
    if (fread(h.data(), 8, n, f) != (size_t)n) return 2;
    fclose(f);
    float2 *a;
    double *o;
    if (cudaMalloc(&a, 8 * n) || cudaMalloc(&o, 8 * n)) return 3;
    cudaMemcpy(a, h.data(), 8 * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(a, o, n);
    std::vector<double> r(n);
    if (cudaMemcpy(r.data(), o, 8 * n, cudaMemcpyDeviceToHost)) return 4;
    f = fopen(v[2], "wb");
    fwrite(r.data(), 8, n, f);
    return fclose(f);
}
"""


def pairs():
    rng = np.random.default_rng(5)
    n = 200_000
    exp = rng.integers(53, 254, n)
    man = rng.integers(0, 1 << 23, n)
    man[::7], man[1::7] = 0, (1 << 23) - 1
    h = ((exp << 23) | man).astype(np.uint32).view(np.float32)
    h = np.where(rng.random(n) < 0.5, -h, h).astype(np.float32)
    ulp = np.ldexp(1.0, exp - 150)
    u = rng.uniform(-1.0, 1.0, n)
    u[::11], u[3::11], u[5::13] = 0.0, -0.5, 0.5
    u[7::17] = rng.integers(-64, 65, u[7::17].size) / 2.0 ** 30  # ties at the double's last place
    low = (ulp * u).astype(np.float32)
    return h, low


@pytest.mark.gpu
def test_join_is_the_fp64_sum(tmp_path):
    h, low = pairs()
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan], dtype=np.float32)
    a = np.zeros((h.size + special.size, 2), dtype=np.float32)
    a[:h.size, 0], a[:h.size, 1] = h, low
    a[h.size:, 0] = special
    src, exe = tmp_path / "join.cu", tmp_path / "join"
    src.write_text(SRC)
    nvcc = "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc if os.path.exists(nvcc) else "nvcc", "-std=c++17", "-O2", "-gencode",
                    "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(REPO, "fargocpt_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    a.tofile(tmp_path / "in")
    subprocess.run([str(exe), str(tmp_path / "in"), str(tmp_path / "out")], check=True)
    got = np.fromfile(tmp_path / "out", dtype=np.float64)
    want = h.astype(np.float64) + low.astype(np.float64)
    assert np.array_equal(got[:h.size].view(np.uint64), want.view(np.uint64))
    tail = got[h.size:]
    assert tail[0] == 0.0 and tail[1] == 0.0 and np.isnan(tail[2:]).all()
