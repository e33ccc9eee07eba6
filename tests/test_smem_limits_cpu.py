"""The dynamic shared-memory limit of every kernel whose need depends on the
system only grows (CPU only).

The limit belongs to the function on the device; contexts of any sizes launch it
from their own host threads.  This test links the library's own launchers of the
sweeps, the operators, the shell derivatives and the adjoint gradients against a
stand-in for the CUDA runtime that records limits and launches, runs a large
system, then a small one, then the large one again: no call may lower a limit, and
every launch must be within its kernel's.
"""
import os
import shutil
import subprocess

import pytest

from dmcbcs_project_gb300 import build

# the runtime's entry points that nvcc's host code and the launchers call
RUNTIME = r"""
#include <cstdio>
#include <map>

struct Dim { unsigned x, y, z; };
static std::map<const void*, int> limit;   // by kernel
static int lowered = 0, refused = 0, launches = 0;
static Dim cg, cb;
static size_t cs;
static void* cst;

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaInitModule(void**) {}
unsigned __cudaPushCallConfiguration(Dim g, Dim b, size_t s, void* st) { cg = g; cb = b; cs = s; cst = st; return 0; }
int __cudaPopCallConfiguration(Dim* g, Dim* b, size_t* s, void* st) { *g = cg; *b = cb; *s = cs; *(void**)st = cst; return 0; }
int __cudaGetKernel(const void** k, const void* f) { *k = f; return 0; }
int __cudaLaunchKernel(const void* k, Dim, Dim, void**, size_t smem, void*)
{
    ++launches;
    const auto it = limit.find(k);
    if (smem > (size_t)(it == limit.end() ? 48 * 1024 : it->second)) ++refused;
    return 0;
}
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int) { *v = a == 16 ? 152 : 227 * 1024; return 0; }   // 16: SM count
int cudaFuncSetAttribute(const void* f, int a, int v)
{
    if (a != 8) return 0;   // 8: the dynamic shared-memory limit
    if (limit.count(f) && v < limit[f]) ++lowered;
    limit[f] = v;
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned)
{
    *n = (int)(228 * 1024 / (smem + 1024));
    if (*n > 4) *n = 4;
    return 0;
}
int cudaGetLastError() { return 0; }
int report()
{
    std::printf("kernels %d lowered %d refused %d launches %d\n", (int)limit.size(), lowered, refused, launches);
    return lowered || refused || limit.size() < 9;
}
}
"""

DRIVER = r"""
#include <cstring>
#include "dmc_kernels.h"

extern "C" int report();
static_assert(cudaDevAttrMultiProcessorCount == 16 && cudaFuncAttributeMaxDynamicSharedMemorySize == 8, "as in the stand-in");
using namespace dmc;

static int all(int up, int nk, bool big)
{
    DevParams p;
    std::memset(&p, 0, sizeof p);
    p.nup = p.ndn = p.npair = p.nd = up;
    p.npart = 2 * up;
    p.nk = nk;
    p.norb = 7;
    p.nmax = 2;
    OpsDev o;
    std::memset(&o, 0, sizeof o);
    o.ntabg = big ? 1000 : 20;
    o.nqtot = 4;
    o.nsamp = 1;
    o.ntabk = 4;
    o.nnk = big ? 8 : 2;
    o.nkv = big ? 200 : 10;
    double d[2] = {0.0, 0.0};
    DevStack st;
    std::memset(&st, 0, sizeof st);
    int e = 0;
    for (int n : {1, 1 << 20})
        e |= launch_sweeps(p, st, n, 1, d, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, d, 0);
    e |= launch_ops_walker(p, o, d, 4, nullptr, nullptr, d, 4, 0);
    for (bool sym : {false, true}) {
        e |= launch_ops_enk(p, o, nullptr, nullptr, nullptr, nullptr, nullptr, sym, d, nullptr, d, 4, d, 152, 0);
        e |= launch_derbcs(p, nullptr, d, d, d, 4, 4, 0, -1, 0, sym);
        if (pgrad_grid(p, 4, 152, 227 * 1024, sym) < 1) e |= 1;
        e |= launch_pgrad(p, nullptr, nullptr, d, d, d, d, d, d, 4, p.norb, 1.0, nullptr, nullptr, 0, 0, sym, 4, nullptr, d,
                          227 * 1024, 0);
    }
    return e;
}

int main()
{
    const int e = all(60, 41, true) | all(5, 3, false) | all(60, 41, true);
    return report() || e;
}
"""


def test_limits_only_grow(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    objs = [os.path.join(build.BUILD, o) for o in ("dmc_sweep.o", "dmc_ops.o", "dmc_single.o")]
    build.build(force=not all(os.path.exists(o) for o in objs))
    driver, runtime, exe = tmp_path / "limits.cu", tmp_path / "runtime.cpp", tmp_path / "limits"
    driver.write_text(DRIVER)
    runtime.write_text(RUNTIME)
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-cudart", "none", "-I", build.CSRC, "-I", build.INCLUDE,
                    str(driver), str(runtime), *objs, "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.stdout, r.stderr)
