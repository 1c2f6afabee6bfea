"""Set-up once per device (superman_b200/csrc/per_device.h), as the batched
walk's launcher does it, on the CPU: each device runs its own, and one device's
failure is not another's."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "superman_b200", "csrc")

PROGRAM = r"""
#include <thread>
#include <vector>
#include "per_device.h"
static int launch(int dev, int status, int* runs)
{
    static spb::OncePerDevice<int> ready;
    return ready(dev, [&] { ++runs[dev]; return status; });
}
int main()
{
    int runs[4] = {0, 0, 0, 0};
    if (launch(1, 7, runs) != 7 || launch(0, 0, runs) != 0) return 1;  // device 1 fails, device 0 does not
    if (launch(1, 0, runs) != 7 || launch(0, 9, runs) != 0) return 2;  // kept, each its own
    std::vector<std::thread> t;
    for (int k = 0; k < 8; ++k) t.emplace_back([&] { launch(3, 0, runs); });
    for (auto& x : t) x.join();
    return runs[0] == 1 && runs[1] == 1 && runs[2] == 0 && runs[3] == 1 ? 0 : 3;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_batched_launcher_sets_up_per_device():
    """The launcher keeps no outcome of its own for the whole process."""
    text = open(os.path.join(CSRC, "batch.cu")).read()
    assert "static cudaError_t" not in text and "OncePerDevice" in text
