"""Per-device set-up of the CUDA kernels: run once for each device, again after
a failure, and under threads once only.  cudaFuncSetAttribute applies to the
current device, so nothing that sets an attribute may be guarded by a flag of
the process.
"""

import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "quant-kernel_b200" / "csrc"

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "device_once.h"
int main() {
    qkb::DeviceOnce once;
    std::atomic<int> runs[3] = {};
    auto ok = [&](int d) { return once.run(d, [&] { ++runs[d]; return 0; }); };
    if (ok(0) || ok(0) || ok(2) || ok(2)) return 1;
    if (runs[0] != 1 || runs[1] != 0 || runs[2] != 1) return 2;
    // a failure is reported and tried again
    int tries = 0;
    if (once.run(1, [&] { ++tries; return 7; }) != 7) return 3;
    if (once.run(1, [&] { ++tries; return 0; }) != 0 || tries != 2) return 4;
    if (once.run(1, [&] { ++tries; return 7; }) != 0 || tries != 2) return 5;
    // devices past the table run every time rather than never
    int far = 0;
    for (int i = 0; i < 2; ++i) once.run(qkb::DeviceOnce::kDevices, [&] { ++far; return 0; });
    for (int i = 0; i < 2; ++i) once.run(-1, [&] { ++far; return 0; });
    if (far != 4) return 6;
    qkb::DeviceOnce shared;
    std::atomic<int> n{0};
    std::vector<std::thread> pool;
    for (int i = 0; i < 8; ++i)
        pool.emplace_back([&] { for (int d = 0; d < 8; ++d) shared.run(d, [&] { ++n; return 0; }); });
    for (auto& t : pool) t.join();
    return n == 8 ? 0 : 7;
}
"""


def test_once_per_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "once"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe),
                    "-pthread"], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_attribute_under_a_process_wide_flag():
    for path in sorted(CSRC.glob("*.cu")):
        for call in re.finditer(r"std::call_once\((?:[^;]|;(?!\s*\n\s*\}\);))*", path.read_text()):
            assert "cudaFuncSetAttribute" not in call.group(0), (path.name, call.group(0)[:80])
