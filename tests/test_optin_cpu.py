"""The record of the shared memory that kernels are opted in to (ib_optin.h), with a fake of the attribute call: one
value per device, never lowered, under threads with different sizes; and no launcher that keeps a record of its own."""
import glob
import os
import re
import subprocess

import gpuimogen_b200.build as build

SRC = r'''
#include "ib_optin.h"
#include <cassert>
#include <thread>
#include <vector>
static std::atomic<size_t> attr[4];
static std::atomic<int> calls{0};
int main()
{
    ib::SmemOptIn s;
    auto set = [](int dev) { return [dev](size_t b) { attr[dev] = b; calls++; return 0; }; };
    assert(s.raise(0, 100, set(0)) == 0 && attr[0] == 100 && attr[1] == 0);
    assert(s.raise(1, 60, set(1)) == 0 && attr[1] == 60);          // a second device has its own
    assert(s.raise(0, 80, set(0)) == 0 && attr[0] == 100);         // never lowered
    assert(calls == 2);
    assert(s.raise(2, 10, [](size_t) { return -7; }) == -7);       // a failure is passed on and not recorded
    assert(s.raise(2, 10, set(2)) == 0 && attr[2] == 10);
    assert(s.raise(1000, 10, [](size_t) { return 0; }) == 0);      // a device past the record: set each time
    std::vector<std::thread> t;
    for (int k = 0; k < 16; k++)
        t.emplace_back([&, k] {
            for (size_t b = 1; b < 2000; b++) {
                const size_t want = 1000 + (b * 37 + k * 101) % 5000;
                s.raise(3, want, set(3));
                assert(attr[3] >= want);                           // what this launch needs is set
            }
        });
    for (auto &x : t) x.join();
    return 0;
}
'''


def test_record(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + build.CSRC, "-o", str(exe), str(src)], check=True)
    subprocess.run([str(exe)], check=True, timeout=120)


def test_every_launcher_uses_it():
    calls = []
    for path in glob.glob(os.path.join(build.CSRC, "*.cu*")):
        with open(path) as f:
            text = f.read()
        calls += [os.path.basename(path)] * len(re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize", text))
    assert calls == ["ib_internal.cuh"], calls
