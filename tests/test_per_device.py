"""What the kernel library asks or sets once on every device (csrc/per_device.h), compiled and run on the host."""
import os
import re
import shutil
import subprocess

import pytest

import rocml_b200

CSRC = os.path.join(os.path.dirname(rocml_b200.__file__), "csrc")

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    rb::PerDevice<int> known;
    int asked = 0;
    const int* v = nullptr;
    auto ask = [&](int& value) { value = 10 + asked++; return 0; };
    if (known.get(0, &v, [](int&) { return 7; }) != 7 || v != nullptr) return 1;          // an error is passed on ...
    if (known.get(0, &v, ask) || *v != 10) return 2;                                      // ... and not kept
    const int* first = v;
    if (known.get(1, &v, ask) || *v != 11) return 3;                                      // a second device is asked itself
    if (known.get(100, &v, ask) || *v != 12) return 4;
    if (known.get(0, &v, ask) || v != first || *v != 10 || asked != 3) return 5;          // each once
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] { for (int d = 200; d < 300; ++d) { const int* w = nullptr; known.get(d, &w, ask); } });
    for (auto& t : threads) t.join();
    return asked == 103 ? 0 : 6;
}
"""


def test_every_device_is_asked_once_and_an_error_is_not_kept(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cc").write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-pthread", "-I", CSRC, str(tmp_path / "t.cc"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


def test_the_32_bit_product_of_more_rows_keeps_its_settings_by_device():
    """Its large shared memory has to be allowed on each: nothing of its launch is kept once a process."""
    with open(os.path.join(CSRC, "gemm_generic.cu")) as f:
        text = f.read()
    body = text[text.index("int launch_f32("):]
    body = body[:body.index("\n}\n")]
    assert "cudaFuncAttributeMaxDynamicSharedMemorySize" in body
    assert [s for s in re.findall(r"\bstatic\b[^;(]*", body) if "PerDevice" not in s] == []
