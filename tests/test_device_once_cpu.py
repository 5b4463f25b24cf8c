"""The opt-in to large shared memory (csrc/device_once.cuh) against a fake of the two runtime calls: once per device and
kernel, again after a failure, and on every call - not refused - for device ordinals beyond the table.  A limit that
follows the calls is only ever raised: a thread that has looked at the occupancy still has its launch before it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#pragma once
#include <cstddef>
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern int g_device, g_sets, g_fail;
inline cudaError_t cudaGetDevice(int* d) { *d = g_device; return 0; }
template<class F> inline cudaError_t cudaFuncSetAttribute(F, int, int) { ++g_sets; return g_fail; }
"""
MAIN = r"""
#include "device_once.cuh"
int g_device = 0, g_sets = 0, g_fail = 0;
static void kernel() {}
static std::atomic<bool> done[ftb200::kDevicesKnown];
static int sets(int device, int fail, int want)
{
    g_device = device, g_fail = fail, g_sets = 0;
    return ftb200::opt_in_smem(kernel, 1000, done) == fail && g_sets == want ? 0 : 1;
}
int main()
{
    if (sets(0, 0, 1) || sets(0, 0, 0)) return 1;   // once
    if (sets(63, 0, 1) || sets(63, 0, 0)) return 2;
    if (sets(64, 0, 1) || sets(64, 0, 1)) return 3; // beyond the table: every time
    if (sets(7, 2, 1) || sets(7, 0, 1) || sets(7, 0, 0)) return 4;  // a failure is reported and not remembered
    // a larger need raises the limit, a smaller one after it does not lower it, a failure is not remembered
    size_t highest = 0;
    auto   raise   = [&](size_t bytes, int fail, int want) {
        g_fail = fail, g_sets = 0;
        return ftb200::raise_smem(kernel, bytes, highest) == fail && g_sets == want ? 0 : 1;
    };
    if (raise(60000, 0, 1) || raise(68000, 0, 1) || raise(60000, 0, 0) || raise(68000, 0, 0)) return 5;
    if (raise(90000, 1, 1) || raise(80000, 0, 1) || raise(90000, 0, 1) || highest != 90000) return 6;
    return 0;
}
"""


def test_opt_in_per_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    src, exe = tmp_path / "main.cc", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-I", str(tmp_path), "-I", os.path.join(ROOT, "fastertransformer_b200", "csrc"),
                           str(src), "-o", str(exe)])
    assert subprocess.call([str(exe)]) == 0
