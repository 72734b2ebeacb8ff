"""What a launcher does once on every device, against a runtime that keeps a kernel's limit per device as CUDA's does."""

from __future__ import annotations

import re
import shutil
import subprocess
from pathlib import Path

import pytest

from litinfer_b200.csrc import build

CSRC = build.CSRC

PROGRAM = r"""
#include "device_once.h"
#include <cassert>
#include <map>
#include <thread>
#include <vector>

static thread_local int current = 0;
static std::atomic<int> raises{0};
static std::atomic<int> limit[100];
static bool fail = false;

extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
    assert(f && a == cudaFuncAttributeMaxDynamicSharedMemorySize);
    if (fail) return cudaErrorInvalidValue;
    ++raises;
    limit[current] = v;
    return cudaSuccess;
}
extern "C" cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) {
    assert(a == cudaDevAttrMultiProcessorCount);
    *v = 100 + d;
    return cudaSuccess;
}

int main() {
    static int kernel;
    static LiOncePerDevice once;
    for (int call = 0; call < 3; ++call)
        for (current = 0; current < 3; ++current) {
            assert(li_raise_shared(once, &kernel, 101376) == cudaSuccess);
            assert(limit[current] == 101376);
            assert(li_multiprocessors() == 100 + current);
        }
    assert(raises == 3);                                   // once on each of three devices
    current = 70;                                          // beyond the marks: every time
    assert(li_raise_shared(once, &kernel, 5) == cudaSuccess && li_raise_shared(once, &kernel, 5) == cudaSuccess && limit[70] == 5 && raises == 5);
    assert(li_multiprocessors() == 170);
    static LiOncePerDevice other;
    current = 1;
    fail = true;                                           // a failure is told and tried again
    assert(li_raise_shared(other, &kernel, 7) != cudaSuccess);
    fail = false;
    assert(li_raise_shared(other, &kernel, 7) == cudaSuccess && limit[1] == 7);
    std::vector<std::thread> threads;
    static LiOncePerDevice many;
    for (int t = 0; t < 16; ++t)
        threads.emplace_back([t] {
            current = 10 + t % 4;
            for (int i = 0; i < 1000; ++i) assert(li_raise_shared(many, &kernel, 9) == cudaSuccess && limit[current] == 9);
        });
    for (auto& t : threads) t.join();
    return 0;
}
"""


def test_once_on_every_device(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    try:
        include = Path(build.find_nvcc()).resolve().parent.parent / "include"
    except build.BuildError:
        include = None
    if cxx is None or include is None or not (include / "cuda_runtime_api.h").is_file():
        pytest.skip("no C++ compiler or no CUDA headers")
    (tmp_path / "p.cpp").write_text(PROGRAM)
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), "-I", str(include), str(tmp_path / "p.cpp"), "-o", str(tmp_path / "p")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(tmp_path / "p")], timeout=60).returncode == 0


def test_no_launcher_keeps_a_mark_for_the_whole_process():
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        assert not re.search(r"static (const )?(int|bool) (sms|raised|attr_set)\b", text), f"{f.name}: limits and counts belong to a device (device_once.h)"
