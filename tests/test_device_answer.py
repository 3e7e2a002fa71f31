"""A question about a device is asked on each device (csrc/device_answer.h): a host
program stands in for the devices."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pbe-fixed-pivot-cuda_gb300", "csrc")

DRIVER = r"""
#include "device_answer.h"
#include <cstdio>
using pbe_gb300::DeviceAnswer;
static DeviceAnswer answer;
static int asked[70];
static int truth[70];
static bool on(int dev) { return answer.get(dev, [&]() { ++asked[dev]; return truth[dev]; }); }
#define CHECK(c) do { if (!(c)) { std::printf("line %d\n", __LINE__); return 1; } } while (0)
int main()
{
    truth[0] = 1; truth[1] = -1; truth[2] = 1;
    for (int r = 0; r < 3; ++r) CHECK(on(0) && !on(1) && on(2));
    CHECK(asked[0] == 1 && asked[1] == 1 && asked[2] == 1);      // every device is asked, once
    truth[3] = 0;                                                // could not be found out
    CHECK(!on(3) && !on(3) && asked[3] == 2);
    truth[3] = 1;
    CHECK(on(3) && on(3) && asked[3] == 3);
    truth[65] = 1;                                               // beyond the table
    CHECK(on(65) && on(65) && asked[65] == 2);
    return 0;
}
"""


def test_every_device_is_asked(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "d.cpp", tmp_path / "d"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_cluster_size_is_asked_per_device():
    """The one kernel that launches clusters beyond the portable size goes by it."""
    with open(os.path.join(CSRC, "aggregation.cu")) as f:
        body = f.read().split("bool small_cluster_ok", 1)[1].split("template <int K, int KIND>", 1)[0]
    assert "NonPortableClusterSizeAllowed" in body
    assert "static const bool" not in body and "DeviceAnswer" in body
