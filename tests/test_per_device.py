"""per_device.h: what a launcher sets or asks once per device, compiled for the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "univeral_3d_reconstruction_system_b200" / "csrc"

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>

int main()
{
    static u3dg::PerDevice values;
    int made[80] = {};
    auto ask = [&](int device) { return values.get(device, [&] { ++made[device + 1]; return 100 + device; }); };
    for (int turn = 0; turn < 3; ++turn)
        for (int device : {0, 3, 63, 1, 0})
            if (ask(device) != 100 + device)
                return 1;
    for (int device : {0, 1, 3, 63})
        if (made[device + 1] != 1) // once for each device, not once for the process
            return 2;
    for (int device : {-1, 64, 70}) // (devices it has no place for are asked every time)
        if (ask(device) != 100 + device || ask(device) != 100 + device || made[device + 1] != 2)
            return 3;
    static u3dg::PerDevice shared;
    std::vector<std::thread> threads;
    int wrong[8] = {};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int k = 0; k < 1000; ++k)
                wrong[t] += shared.get(k % 5, [&] { return 7 + k % 5; }) != 7 + k % 5;
        });
    for (auto &t : threads)
        t.join();
    for (int w : wrong)
        if (w)
            return 4;
    return 0;
}
"""


def _compile(tmp_path, name, text):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src = tmp_path / f"{name}.cpp"
    src.write_text(text)
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", f"-I{CSRC}", str(src), "-o", str(tmp_path / name)], check=True)
    return tmp_path / name


def test_a_value_is_made_once_for_each_device(tmp_path):
    assert subprocess.run([str(_compile(tmp_path, "per_device", PROGRAM))]).returncode == 0


def test_launchers_keep_no_device_value_per_process():
    # A function-local static that is computed once holds the first device's value for all others.
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for call in ("cudaFuncSetAttribute", "cudaOccupancyMaxActiveBlocksPerMultiprocessor", "cudaDeviceGetAttribute"):
            at = text.find(call)
            while at >= 0:
                before = text[:at].rsplit("\n}\n", 1)[-1]
                assert "static const int" not in before, (path.name, call)
                at = text.find(call, at + 1)
