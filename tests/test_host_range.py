"""Which host buffers the GPU may read and write itself (csrc/host_range.h), on the CPU with made-up answers of the driver:
a buffer whose page-locked range starts late or ends early, one across two ranges, managed and device memory."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include "host_range.h"
#include <cstdio>
using pxb::HostRange;
using pxb::range_holds;
static int bad = 0;
static void expect(bool want, const HostRange &r, unsigned long long at, size_t bytes, const char *what) {
    if (range_holds(r, reinterpret_cast<const void *>(at), bytes) != want) {
        std::printf("%s\n", what);
        ++bad;
    }
}
int main() {
    const HostRange r{1, 0, 0x10000, 0x2000};
    expect(true, r, 0x10000, 0x2000, "the whole range");
    expect(true, r, 0x10008, 0x1ff8, "up to its end");
    expect(true, r, 0x12000, 0, "nothing, at its end");
    expect(false, r, 0x10000, 0x2001, "one byte past it");
    expect(false, r, 0x11ff8, 16, "first byte inside, last one not");
    expect(false, r, 0xfff8, 16, "first byte before it");
    expect(false, r, 0x12008, 8, "behind it");
    expect(false, r, 0x10000, ~(size_t)0, "a size that wraps");
    expect(false, HostRange{1, 1, 0x10000, 0x2000}, 0x10000, 8, "managed memory");
    expect(false, HostRange{2, 0, 0x10000, 0x2000}, 0x10000, 8, "device memory");
    expect(false, HostRange{}, 0x10000, 8, "memory that the driver does not know");
    return bad;
}
"""


def test_range_holds_whole_buffers_only(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++20", "-I", os.path.join(ROOT, "perix_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
