"""The round-off maximum of a warp (ErrMax and warp_max of llg_device.cuh, in a kernel of their own) is
the largest |difference| to the last bit, whichever lane and operand holds it: the bound, the reported
maximum and the logs are no shorter than the differences themselves."""
import math
import os
import random
import struct
import subprocess

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "llg_device.cuh"
__global__ void k(const double* x, int n, unsigned long long* out) {
    llg::ErrMax<COUNT> e;
    for (int i = 0; i < n; ++i) e.add(x[2 * (32 * i + threadIdx.x)], x[2 * (32 * i + threadIdx.x) + 1]);
    const unsigned long long w = llg::warp_max(e.value());
    if (threadIdx.x == 0) *out = w;
}
int main() {
    int n;
    double* d;
    unsigned long long *o, h;
    cudaMalloc(&d, 64 * 8 * sizeof(double));
    cudaMalloc(&o, sizeof *o);
    while (scanf("%d", &n) == 1 && n >= 1 && n <= 8) {  // 64 n doubles, as their bits
        std::vector<unsigned long long> v(64 * n);
        for (auto& x : v)
            if (scanf("%llx", &x) != 1) return 2;
        cudaMemcpy(d, v.data(), v.size() * 8, cudaMemcpyHostToDevice);
        k<<<1, 32>>>(d, n, o);
        if (cudaMemcpy(&h, o, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        printf("%016llx\n", h);
    }
    return 0;
}
"""


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


@pytest.mark.parametrize("chains", [1, 2])
def test_warp_maximum_is_exact(gpu, tmp_path, chains):
    src, exe = tmp_path / "m.cu", tmp_path / "m"
    src.write_text(SOURCE.replace("COUNT", str(chains)))
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(PKG, "csrc"), str(src), "-o", str(exe)], check=True)
    rng = random.Random(5)
    cases = []
    for n in (1, 2, 8):
        size = 64 * n
        cases.append([0.0] * size)
        cases.append([rng.uniform(-0.5, 0.5) for _ in range(size)])
        cases.append([rng.randrange(-64, 65) / 4096 for _ in range(size)])  # a few bits each
        for at in (0, 1, 2, size // 2 + 1, size - 2, size - 1):
            # all within the last two bits of one another, the largest at `at`, of either sign
            top = math.nextafter(0.3, 1.0)
            v = [rng.choice((-1, 1)) * rng.choice((0.3, math.nextafter(0.3, 0.0))) for _ in range(size)]
            v[at] = rng.choice((-1, 1)) * top
            cases.append(v)
        v = [rng.uniform(-0.5, 0.5) for _ in range(size)]
        v[size - 1] = math.inf
        cases.append(v)
        v = [5e-324 * rng.randrange(4) for _ in range(size)]  # subnormal
        cases.append(v)
    text = "\n".join(f"{len(v) // 64} " + " ".join(f"{_bits(x):x}" for x in v) for v in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert [int(x, 16) for x in out] == [_bits(max(abs(x) for x in v)) for v in cases]
    # not a number (it spreads to a whole transform's outputs) exceeds every bound
    nan = "1 " + " ".join(f"{_bits(math.nan):x}" for _ in range(64))
    out = subprocess.run([str(exe)], input=nan, capture_output=True, text=True, check=True).stdout.split()
    assert int(out[0], 16) == _bits(math.inf)
