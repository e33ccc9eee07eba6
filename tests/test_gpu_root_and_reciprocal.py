"""The pair distance's root and reciprocal root and the pivots' reciprocal, as the
kernels use them (compiled here from their headers), against extended precision.

Tolerances.  Both start from a single-precision value good to 2^-21 and end with a
multiply-add, so the last rounding (half a unit) and what enters it remain: the root
after its Newton correction within one unit in the last place of the correctly
rounded one, the reciprocal root (whose residual carries the rounding of r2 y) within
two, the reciprocal within one.  The reciprocal also through the batched inverse of
1 x 1 matrices, on both sides of the switch to the division (2^-111, 2^109) and for
the smallest, subnormal and largest numbers.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, build, capi, configs

pytestmark = pytest.mark.gpu
LD = np.longdouble

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "dmc_walker.cuh"

__global__ void eval(const double* in, double* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r, ri;
    dmc::walker::inv_dist(in[2 * i], r, ri);
    out[3 * i] = r;
    out[3 * i + 1] = ri;
    out[3 * i + 2] = dmc::walker::pivot_rcp(in[2 * i + 1]);
}

int main(int argc, char** argv)
{
    FILE* f = std::fopen(argv[1], "rb");
    if (argc < 3 || !f) return 1;
    std::fseek(f, 0, SEEK_END);
    const int n = (int)(std::ftell(f) / 16);
    std::rewind(f);
    std::vector<double> in(2 * n), out(3 * n);
    if ((int)std::fread(in.data(), 16, n, f) != n) return 2;
    std::fclose(f);
    double *din, *dout;
    if (cudaMalloc(&din, n * 16) || cudaMalloc(&dout, n * 24)) return 3;
    if (cudaMemcpy(din, in.data(), n * 16, cudaMemcpyHostToDevice)) return 4;
    eval<<<(n + 255) / 256, 256>>>(din, dout, n);
    if (cudaMemcpy(out.data(), dout, n * 24, cudaMemcpyDeviceToHost)) return 5;
    FILE* g = std::fopen(argv[2], "wb");
    return !g || (int)std::fwrite(out.data(), 24, n, g) != n || std::fclose(g) ? 6 : 0;
}
"""


def units(got, exact):
    """|got - exact| in units of the last place of the correctly rounded value."""
    return float(np.max(np.abs(got.astype(LD) - exact) / np.spacing(np.abs(exact).astype(np.float64)).astype(LD)))


def test_root_and_reciprocal(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "eval.cu", tmp_path / "eval"
    src.write_text(SOURCE)
    subprocess.run([nvcc, *build.ARCH, "-O3", "-std=c++17", "-I", build.CSRC, "-I", build.INCLUDE, str(src), "-o", str(exe)], check=True)
    rng = np.random.default_rng(1)
    m = 200000
    r2 = 2.0 ** rng.uniform(-126.0, 128.0, m)
    r2[:8] = [1.0, 2.0 ** -126, np.nextafter(2.0 ** 128, 0.0), 4.0, np.nextafter(4.0, 0.0), 2.0 ** 126, 3.0 * 2.0 ** 126, 2.0]
    r2[8:1000] = rng.integers(1, 2 ** 26, 992).astype(float) ** 2        # exact squares: exact roots
    p = 2.0 ** rng.uniform(-111.0, 109.0, m) * rng.choice([-1.0, 1.0], m)
    p[:8] = [2.0 ** -111, np.nextafter(2.0 ** 109, 0.0), np.nextafter(2.0 ** -111, 0.0), 2.0 ** 109, 1.0, np.nextafter(1.0, 0.0), -3.0, 49.0]
    np.stack([r2, p], 1).tofile(tmp_path / "in")
    subprocess.run([str(exe), str(tmp_path / "in"), str(tmp_path / "out")], check=True, timeout=120)
    out = np.fromfile(tmp_path / "out").reshape(m, 3)
    assert units(out[:, 0], np.sqrt(r2.astype(LD))) <= 1.0
    assert np.array_equal(out[8:1000, 0], np.sqrt(r2[8:1000]))
    assert units(out[:, 1], 1 / np.sqrt(r2.astype(LD))) <= 2.0
    assert units(out[:, 2], 1 / p.astype(LD)) <= 1.0


def test_reciprocal_of_any_pivot():
    rng = np.random.default_rng(2)
    p = np.concatenate([2.0 ** rng.uniform(-1022.0, 1022.0, 4000), [2.0 ** k * f for k in (-112, -111, -110, 108, 109, 110) for f in (1.0, 1.5, np.nextafter(2.0, 0.0))],
                        [2.0 ** -1022, 2.0 ** -1024, 1.7e308, np.inf]])
    p = p * rng.choice([-1.0, 1.0], p.size)
    with capi.Context(abi.make_system(configs.system_params(7, 7, 5)), abi.make_run(configs.run_params(4, 0.001))) as ctx:
        inv, logdet, sign = ctx.matinv(p.reshape(-1, 1, 1))
    inv = inv.reshape(-1)
    assert np.array_equal(sign, np.sign(p).astype(np.int32))
    finite = np.isfinite(p) & (np.abs(p) >= 2.0 ** -1022)
    assert units(inv[finite], 1 / p[finite].astype(LD)) <= 1.0
    assert inv[-1] == 0.0 and inv[-3] == np.copysign(np.inf, p[-3])   # infinity; 2^-1024
