"""A device's answers are its own: the LU panel's cluster kernel asks (and sets the kernel's attributes)
once on each device, not once in a process. Compiled with the host compiler against a count."""
from __future__ import annotations

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "remora_b200" / "csrc"

PROGRAM = r"""
#include "per_device.cuh"
#include <cstdio>
static rc::PerDevice<5> fits;
int main() {
    int asked = 0, wrong = 0;
    auto get = [&](int dev, int which, bool answer) {
        if (fits.get(dev, which, [&] { ++asked; return answer; }) != answer) ++wrong;
    };
    for (int dev = 0; dev < 64; ++dev)
        for (int q = 0; q < 5; ++q) get(dev, q, (dev + q) % 2 == 0);   // every device is asked
    const int first = asked;
    for (int dev = 0; dev < 64; ++dev)
        for (int q = 0; q < 5; ++q) get(dev, q, (dev + q) % 2 == 0);   // and only once
    const int again = asked;
    get(64, 0, true);    // beyond the table: asked each time
    get(64, 0, false);
    get(-1, 4, true);
    std::printf("%d %d %d %d", first, again, asked, wrong);
}
"""


def test_every_device_is_asked_once(tmp_path):
    src, exe = tmp_path / "a.cpp", tmp_path / "a.out"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "320 320 323 0"


def test_no_kernel_attribute_is_kept_for_a_whole_process():
    """Host code that remembers something about a device has the device in its key."""
    text = (CSRC / "lu.cu").read_text()
    assert "static std::atomic" not in text and "static PerDevice<" in text
