"""Which readers a writer has to wait for (stream_use.h)."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "kiraray_gb300" / "csrc"

MAIN = r"""
#include <cassert>
#include <thread>
#include <vector>
#include "stream_use.h"

int main() {
    krr::StreamUse u;
    assert(u.alone_on(7));                      // nobody reads
    u.read(7);
    u.read(7);
    assert(u.alone_on(7) && !u.alone_on(8));    // a stream waits for itself
    u.start_over();
    assert(u.alone_on(8));
    u.read(0);
    assert(u.alone_on(0) && !u.alone_on(1));
    u.read(1);
    assert(!u.alone_on(0) && !u.alone_on(1));   // two streams
    u.read(1);
    assert(!u.alone_on(1));
    u.start_over();
    u.read(1);
    assert(u.alone_on(1));
    u.read_captured();                          // a graph may run anywhere, and again
    assert(!u.alone_on(1));
    u.start_over();
    assert(!u.alone_on(1));
    for (int k = 0; k < 200; ++k) {             // readers on several threads
        krr::StreamUse v;
        std::vector<std::thread> t;
        for (int i = 0; i < 4; ++i) t.emplace_back([&v, i] { for (int j = 0; j < 50; ++j) v.read(i); });
        for (auto &x : t) x.join();
        for (int i = 0; i < 4; ++i) assert(!v.alone_on(i));
    }
    return 0;
}
"""


def test_stream_use(tmp_path):
    src = tmp_path / "main.cpp"
    src.write_text(MAIN)
    exe = tmp_path / "main"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", str(CSRC), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr


def test_every_view_names_its_stream():
    """Kernels get the instance tree from instanced_view() alone."""
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        if f.name != "instanced.cu":
            assert "tlas_nodes" not in text and "tlas->d_nodes" not in text.replace("a.tlas->d_nodes, a.tlas->d_tris", ""), f.name
