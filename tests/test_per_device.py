"""Kernel attributes and device sizes belong to a device: a process that uses a second one
sets and asks for them there too.

CPU only: a small program over csrc/tc_perdev.h whose "current device" is a variable; and
no launch code keeps such a setting once per process.
"""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tracer_code_gb300", "csrc")

PROGRAM = r"""
#include "tc_perdev.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int device = 0;
int tc_current_device() { return device; }
#define CHECK(x) if (!(x)) { std::printf("%s\n", #x); return 1; }
int main() {
    static PerDevice set, sms, refused;
    int calls[3] = {0, 0, 0};
    for (int round = 0; round < 3; round++)
        for (device = 0; device < 3; device++) {
            CHECK(set.get([&] { calls[device]++; return 0; }) == 0);
            CHECK(sms.get([&] { return 100 + device; }) == 100 + device);
        }
    CHECK(calls[0] == 1 && calls[1] == 1 && calls[2] == 1);
    // a setting that was refused is tried again, on that device only
    device = 1;
    CHECK(refused.get([] { return -1; }) == -1);
    CHECK(refused.get([] { return -1; }) == -1);
    CHECK(refused.get([] { return 7; }) == 7);
    CHECK(refused.get([] { return -1; }) == 7);
    device = 0;
    CHECK(refused.get([] { return -1; }) == -1);
    // devices beyond those remembered are asked each time
    device = 1000;
    CHECK(sms.get([] { return 5; }) == 5 && sms.get([] { return 6; }) == 6);
    device = -1;
    CHECK(sms.get([] { return 5; }) == 5 && sms.get([] { return 6; }) == 6);
    std::vector<std::thread> pool;
    static PerDevice shared;
    static std::atomic<int> bad{0};
    for (int t = 0; t < 8; t++)
        pool.emplace_back([t] {
            device = t % 4;
            for (int n = 0; n < 1000; n++)
                if (shared.get([t] { return 10 * (t % 4); }) != 10 * (t % 4)) bad++;
        });
    for (auto& t : pool) t.join();
    CHECK(bad == 0);
    return 0;
}
"""


def test_settings_are_kept_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "per_device.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "per_device")
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_setting_is_kept_per_process():
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        s = open(f).read()
        for m in re.finditer(r"^[ \t]+static (const )?(bool|int) (\w+)( =|;)", s, re.M):
            pytest.fail(f"{os.path.basename(f)}: {m.group(0).strip()}")
