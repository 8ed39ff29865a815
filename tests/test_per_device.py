"""The guard of per-device kernel settings (csrc/gx_per_device.h): a setting made on one device does not count for
another, a larger value is set again, and no kernel launcher keeps such a guard per process."""

from __future__ import annotations

import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "giaoint_gb300" / "csrc"

PROGRAM = r"""
#include "gx_per_device.h"
#include <cassert>
#include <thread>
#include <vector>
int main() {
    gx::PerDevice p;
    assert(p.needs(0, 100) && p.needs(1, 100));
    p.done(0, 100);
    assert(!p.needs(0, 100) && !p.needs(0, 50) && p.needs(0, 101));
    assert(p.needs(1, 100));
    p.done(0, 50);
    assert(!p.needs(0, 100));
    p.done(1000, 100);
    assert(p.needs(1000, 100) && p.needs(-1, 1));
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&p, t] { for (int v = 1; v <= 1000; ++v) p.done(2, v * 8 + t); });
    for (auto& t : threads) t.join();
    assert(!p.needs(2, 8007) && p.needs(2, 8008));
}
"""


def test_guard(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++20", "-pthread", "-I", str(CSRC), str(src), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True, timeout=60)


def test_no_launcher_keeps_a_process_wide_guard():
    for path in sorted(CSRC.glob("gx_*.cu*")):
        text = path.read_text()
        if "cudaFuncSetAttribute" in text:
            assert not re.search(r"static\s+(std::atomic<|bool|size_t|int\b(?! device))[^;()]*\b(ready|configured)", text), path
