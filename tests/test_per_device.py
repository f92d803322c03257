"""What is set once per device (per_device.h): on every device of a process,
again after a failure, and not again once it held."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "kiraray_gb300" / "csrc"

MAIN = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "per_device.h"

int main() {
    krr::OncePerDevice once;
    int calls[80] = {}, status = 0;
    auto on = [&](int dev) { return once(dev, [&] { ++calls[dev]; return status; }); };
    for (int k = 0; k < 3; ++k) assert(on(0) == 0);
    assert(calls[0] == 1);
    assert(on(1) == 0 && calls[1] == 1);      // the second device of the process
    assert(on(63) == 0 && on(63) == 0 && calls[63] == 1);
    status = 7;                               // a failure is reported and not kept
    assert(on(2) == 7 && on(2) == 7 && calls[2] == 2);
    status = 0;
    assert(on(2) == 0 && on(2) == 0 && calls[2] == 3);
    assert(on(0) == 0 && calls[0] == 1);
    assert(on(70) == 0 && on(70) == 0 && calls[70] == 2);
    krr::OncePerDevice other;                 // another kernel's
    int n = 0;
    assert(other(0, [&] { ++n; return 0; }) == 0 && n == 1);
    krr::OncePerDevice shared;
    std::vector<std::thread> threads;
    for (int k = 0; k < 8; ++k)
        threads.emplace_back([&, k] { for (int i = 0; i < 1000; ++i) assert(shared((k + i) % 64, [] { return 0; }) == 0); });
    for (auto &t : threads) t.join();
    for (int d = 0; d < 64; ++d) shared(d, [&] { ++n; return 0; });
    assert(n == 1);
    return 0;
}
"""


def test_once_per_device(tmp_path):
    src = tmp_path / "main.cpp"
    src.write_text(MAIN)
    exe = tmp_path / "main"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", str(CSRC), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr


def test_limits_are_set_per_device():
    """No kernel's limit is raised but through it."""
    for f in sorted(CSRC.glob("*.cu")):
        assert "cudaFuncSetAttribute" not in f.read_text(), f.name
