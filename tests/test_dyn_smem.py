"""The opt-in to more than 48 KB of dynamic shared memory is made once for each kernel and device,
by every host thread that launches: csrc/dyn_smem.h is compiled with stand-ins for the two runtime
calls it makes, and no other source remembers an opt-in by itself."""
import glob
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "slope_stability_octave_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <thread>
#include "dyn_smem.h"
static thread_local int device = 0;
static std::map<std::pair<const void *, int>, int> limit;   // what the two devices have been told
static int calls = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaErrorInvalidValue;
    ++calls;
    if (v > 227 * 1024) return cudaErrorInvalidValue;
    limit[{f, device}] = v;
    return cudaSuccess;
}
static void one(int) {}
static void two(int) {}
#define EXPECT(c) if (!(c)) { std::printf("line %d\n", __LINE__); return 1; }
int main() {
    using sg::allow_dynamic_smem;
    EXPECT(allow_dynamic_smem(one, 48 * 1024) == cudaSuccess && calls == 0);
    EXPECT(allow_dynamic_smem(one, 60000) == cudaSuccess && calls == 1);
    EXPECT(allow_dynamic_smem(one, 50000) == cudaSuccess && calls == 1);
    EXPECT(allow_dynamic_smem(two, 60000) == cudaSuccess && calls == 2);
    device = 1;                                              // the same thread, another device
    EXPECT(allow_dynamic_smem(one, 60000) == cudaSuccess && calls == 3);
    EXPECT((limit[{(const void *)one, 1}] == 60000));
    EXPECT(allow_dynamic_smem(one, 90000) == cudaSuccess && calls == 4);
    device = 0;                                              // and back: its limit is still the smaller one
    EXPECT(allow_dynamic_smem(one, 60000) == cudaSuccess && calls == 4);
    EXPECT(allow_dynamic_smem(one, 90000) == cudaSuccess && calls == 5);
    EXPECT(allow_dynamic_smem(one, 300000) == cudaErrorInvalidValue && calls == 6);   // refused: not remembered
    EXPECT(allow_dynamic_smem(one, 300000) == cudaErrorInvalidValue && calls == 7);
    std::thread([] { device = 1; sg::allow_dynamic_smem(two, 60000); }).join();
    EXPECT((limit[{(const void *)two, 1}] == 60000) && calls == 8);
    for (device = 2; device < 100; ++device)                 // more pairs than a thread remembers
        EXPECT(allow_dynamic_smem(one, 60000) == cudaSuccess && (limit[{(const void *)one, device}] == 60000));
    return 0;
}
"""


def test_limit_is_raised_per_kernel_and_device(tmp_path):
    cc = next((c for c in ("/usr/bin/g++", shutil.which("g++")) if c and os.path.exists(c)), None)
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if cc is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cc, "-std=c++17", "-pthread", "-I" + CSRC, "-I" + include, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_every_opt_in_goes_through_it():
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if os.path.isfile(path) and os.path.basename(path) != "dyn_smem.h":
            assert "cudaFuncSetAttribute" not in open(path).read(), path
