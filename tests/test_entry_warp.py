"""The warp that adds a shot's entries in the transposed step, run on the CPU:
the functions' text from csrc/step.cu is compiled for the host with 32 threads
for the lanes and warp-wide operations that need every lane, so an operation
that some lanes never reach is found instead of waited for."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
using std::min;
#define __device__
#define __forceinline__ inline
constexpr int kThreads = 256;
struct Dim { int x; };
static thread_local Dim threadIdx;

// 32 lanes meet here with a value each; a lane that waits for two seconds is waiting for one that never comes
static std::mutex mu;
static std::condition_variable cv;
static int arrived = 0;
static long generation = 0;
static int slot[2][32];
static int *meet(int v) {
    std::unique_lock<std::mutex> l(mu);
    const long g = generation;
    int *s = slot[g & 1];
    s[threadIdx.x] = v;
    if (++arrived == 32) {
        arrived = 0;
        generation++;
        cv.notify_all();
    } else if (!cv.wait_for(l, std::chrono::seconds(2), [&] { return generation != g; })) {
        printf("HANG\n");
        fflush(stdout);
        _Exit(3);
    }
    return s;
}
static int __shfl_up_sync(unsigned, int v, int d) { int *s = meet(v); return s[threadIdx.x >= d ? threadIdx.x - d : threadIdx.x]; }
static bool __all_sync(unsigned, bool p) { int *s = meet(p); return std::all_of(s, s + 32, [](int q) { return q != 0; }); }
static void __syncwarp() { meet(0); }
static unsigned landed_lanes;
static bool mbar_wait(uint64_t *, uint32_t) { return (landed_lanes >> threadIdx.x) & 1; }
"""

MAIN = r"""
int main(int argc, char **argv) {
    landed_lanes = (unsigned)strtoul(argv[1], nullptr, 0);
    const int n = atoi(argv[2]), distinct = atoi(argv[3]);
    std::vector<float> v(64, 0.f), val(kThreads);
    std::vector<int> loc(kThreads);
    for (int i = 0; i < n; i++) {
        loc[i] = distinct ? i : (7 * i) % 10;
        val[i] = 1.f + i;
    }
    int ok[32];
    std::vector<std::thread> t;
    for (int i = 0; i < 32; i++)
        t.emplace_back([&, i] {
            threadIdx.x = i;
            ok[i] = wait_and_add<1, 64>(nullptr, 0, true, v.data(), n, loc.data(), val.data(), 2.f);
        });
    for (auto &q : t) q.join();
    for (int i = 0; i < 32; i++) printf("%d ", ok[i]);
    for (float x : v) printf("%.1f ", x);
    return 0;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host compiler")
    text = open(os.path.join(ROOT, "seispie_b200", "csrc", "step.cu")).read()
    parts = []
    for name in ("add_entries", "wait_and_add"):
        m = re.search(r"template <[^>]*>\n__device__ __forceinline__ \w+ %s\(.*?\n}\n" % name, text, re.S)
        assert m, name
        parts.append(m.group(0))
    d = tmp_path_factory.mktemp("warp")
    src, out = d / "warp.cpp", d / "warp"
    src.write_text(SHIM + "\n".join(parts) + MAIN)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-Wno-unknown-pragmas", str(src), "-o", str(out)], check=True)
    return str(out)


def _run(exe, landed, n, distinct):
    r = subprocess.run([exe, str(landed), str(n), str(distinct)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-200:]
    x = r.stdout.split()
    return [int(q) for q in x[:32]], [float(q) for q in x[32:]]


@pytest.mark.parametrize("landed", [0x0, 0x1, 0xfffffffe, 0x0000ffff, 0x7fffffff])
@pytest.mark.parametrize("n", [1, 32, 40])
def test_a_wait_that_gives_up_in_some_lanes_gives_up_in_all(exe, landed, n):
    ok, v = _run(exe, landed, n, 1)
    assert ok == [0] * 32 and v == [0.0] * 64


@pytest.mark.parametrize("n,distinct", [(0, 1), (1, 1), (32, 1), (45, 1), (33, 0), (64, 0)])
def test_entries_are_added_once_the_copies_have_landed(exe, n, distinct):
    ok, v = _run(exe, 0xffffffff, n, distinct)
    want = [0.0] * 64
    for i in range(n):
        want[i if distinct else (7 * i) % 10] += 2.0 * (1 + i)
    assert ok == [1] * 32 and v == want
