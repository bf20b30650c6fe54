"""Launch plans are kept per device: the functions of csrc/march.cu that keep
them, compiled for the host over a stand-in for the CUDA runtime with two
devices of different sizes.  A kernel's attributes are set on each device that
runs it, and no device gets what was found on another."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <atomic>
#include <cstddef>
#include <cstdio>
#include <map>
#include <mutex>
#include <vector>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum { cudaFuncAttributeMaxDynamicSharedMemorySize, cudaFuncAttributeNonPortableClusterSizeAllowed };
enum { cudaDevAttrMultiProcessorCount, cudaLaunchAttributeClusterDimension };
struct dim3 { unsigned x, y, z; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
struct cudaLaunchAttribute { int id; struct { struct { unsigned x, y, z; } clusterDim; } val; };
struct cudaLaunchConfig_t { dim3 gridDim, blockDim; size_t dynamicSmemBytes; cudaLaunchAttribute *attrs; int numAttrs; };
constexpr int FWI_ECUDA = -2, FWI_ERANGE = -3, kResThreads = 512;
static int set_error(int c, const char *, ...) { return c; }
static const char *cudaGetErrorString(cudaError_t) { return ""; }
static cudaError_t cudaGetLastError() { return cudaSuccess; }
static int device = 0;
static std::map<int, std::map<int, int>> attr[2];  // device -> kernel -> attribute -> value
static cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
static cudaError_t cudaDeviceGetAttribute(int *v, int, int d) { *v = d ? 20 : 148; return cudaSuccess; }
static cudaError_t cudaFuncSetAttribute(int kernel, int a, int v) { attr[device][kernel][a] = v; return cudaSuccess; }
static bool fits(int kernel, size_t b) {
    return b <= 49152 || (size_t)attr[device][kernel][cudaFuncAttributeMaxDynamicSharedMemorySize] >= b;
}
static cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, int kernel, int, size_t b) {
    if (!fits(kernel, b)) return cudaErrorInvalidValue;
    *n = device ? 1 : 3;
    return cudaSuccess;
}
static cudaError_t cudaOccupancyMaxActiveClusters(int *n, int kernel, const cudaLaunchConfig_t *c) {
    if (!fits(kernel, c->dynamicSmemBytes)) return cudaErrorInvalidValue;
    if (c->gridDim.x > 8 && !attr[device][kernel][cudaFuncAttributeNonPortableClusterSizeAllowed]) return cudaErrorInvalidValue;
    *n = device ? 1 : 9;
    return cudaSuccess;
}
template <int MODE, int WIDE, bool SEG> constexpr int march_kernel = 1;
template <int MODE, int I> constexpr int resident_kernel = 2;
static size_t march_bytes(int, int, int n) { return 30000u * n; }
"""

MAIN = r"""
int main() {
    for (int pass = 0; pass < 2; pass++)
        for (device = 0; device < 2; device++) {
            MarchPlan p{};
            const int rc = march_choose<1, 0, false>(128, 136, 0, &p);
            printf("%d %d %d ", rc, p.occ, sm_count());
            printf("%d %d %d ", resident_clusters<1, 2>(4, 40000), resident_clusters<1, 2>(16, 40000), resident_clusters<1, 2>(16, 200000));
            printf("%d %d\n", (int)fits(1, 220000), (int)fits(2, 220000));
        }
    return 0;
}
"""


def _function(text, pattern):
    m = re.search(pattern, text, re.S | re.M)
    assert m, pattern
    return m.group(0)


def test_every_device_gets_its_own_attributes_and_plans(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    text = open(os.path.join(ROOT, "seispie_b200", "csrc", "march.cu")).read()
    parts = [_function(text, r"^constexpr size_t kMaxSmem = .*?;\n")]
    if "current_device" in text:
        parts.append(_function(text, r"^static int current_device\(\) \{.*?\n\}\n"))
    parts += [_function(text, r"^struct MarchPlan \{.*?\n\};\n"),
              _function(text, r"^template <int MODE, int WIDE, bool SEG>\nstatic int march_choose\(.*?\n\}\n"),
              _function(text, r"^static int sm_count\(\) \{.*?\n\}\n"),
              _function(text, r"^template <int MODE, int I>\nstatic int resident_clusters\(.*?\n\}\n")]
    src, out = tmp_path / "plans.cpp", tmp_path / "plans"
    src.write_text(SHIM + "\n".join(parts) + MAIN)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", str(src), "-o", str(out)], check=True)
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0
    rows = [[int(q) for q in line.split()] for line in r.stdout.splitlines()]
    assert rows == [[0, 3, 148, 9, 9, 9, 1, 1], [0, 1, 20, 1, 1, 1, 1, 1]] * 2
