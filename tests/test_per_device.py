"""Host state of the kernels' launchers that belongs to a device: each device of a process has its own."""
import glob
import os
import re
import shutil
import subprocess

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini_rsglang_b200", "csrc", "kernels")

FAKE_RUNTIME = """
#pragma once
typedef int cudaError_t;
constexpr cudaError_t cudaSuccess = 0;
extern int current_device, broken;
inline cudaError_t cudaGetDevice(int* device) { *device = current_device; return broken; }
"""

PROGRAM = """
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int current_device = 0, broken = 0;
int launches(PerDevice& configured) {          // what a launcher does: its attributes once a device
    if (configured.get()) return 0;
    configured.set(1);
    return 1;
}
#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s\\n", __LINE__, #x); return 1; } } while (0)
int main() {
    static PerDevice configured, clusters;
    for (int round = 0; round < 2; ++round)
        for (current_device = 0; current_device < 64; ++current_device) EXPECT(launches(configured) == (round == 0));
    EXPECT(clusters.get() == 0);
    current_device = 3; clusters.set(33);
    current_device = 4; EXPECT(clusters.get() == 0); clusters.set(-1);
    current_device = 3; EXPECT(clusters.get() == 33);
    current_device = 64; EXPECT(launches(configured) == 1 && launches(configured) == 1);      // no place in the table: done every time
    current_device = -1; EXPECT(launches(configured) == 1);
    current_device = 3; broken = 1; EXPECT(clusters.get() == 0);
    broken = 0;
    static PerDevice shared;
    std::vector<std::thread> threads;
    current_device = 7;
    for (int i = 0; i < 4; ++i) threads.emplace_back([] { for (int k = 0; k < 1000; ++k) if (shared.get() == 0) shared.set(5); });
    for (auto& t : threads) t.join();
    EXPECT(shared.get() == 5);
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="no C++ compiler")
def test_a_number_a_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE_RUNTIME)
    (tmp_path / "main.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{tmp_path}", f"-I{KERNELS}", str(tmp_path / "main.cc"), "-o", str(tmp_path / "main")], check=True)
    done = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout


def test_no_launcher_keeps_a_devices_state_for_the_whole_process():
    """Where kernels' attributes are set or residency is asked for, what is remembered of it is remembered a device: no flag or number of
    the process beside it (a static constant, as a switch of the environment, is none)."""
    looked = 0
    for path in glob.glob(os.path.join(KERNELS, "*.cu")):
        source = open(path).read()
        if "cudaFuncSetAttribute" not in source:
            continue
        looked += 1
        kept = re.findall(r"^ +static (?:bool|int|unsigned|size_t)\b[^;(]*;", source, re.M)
        assert not kept, f"{os.path.basename(path)}: {kept}"
        assert "PerDevice" in source, os.path.basename(path)
    assert looked >= 10
