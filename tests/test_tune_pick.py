"""The autotuner's choice among schedules timed one step at a time and in a loop (csrc/tune_pick.h), on the CPU with made-up
times."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include "tune_pick.h"
#include <cstdio>
static int bad = 0;
static void expect(int want, int flushed, std::vector<float> step, std::vector<float> loop, const char *what,
                   int exact = 0) {
    const int got = pxb::pick_by_loop(step, flushed, exact, [&](int v, float *t) {
        if (loop[v] == -2.f) { std::printf("%s: schedule %d timed\n", what, v); ++bad; }
        *t = loop[v];
        return loop[v] < 0.f ? -1 : loop[v] == 0.f ? 0 : 1;
    });
    if (got != want) { std::printf("%s: %d, not %d\n", what, got, want); ++bad; }
}
int main() {
    expect(2, 1, {1.05f, 1.0f, 1.09f, 1.2f}, {3.f, 4.f, 2.f, -2.f}, "the fastest loop within a tenth");
    expect(1, 1, {1.05f, 1.0f, 1.09f}, {3.f, 4.f, -1.f}, "a loop fails after another has ended");
    expect(1, 1, {1.05f, 1.0f, 1.09f}, {-1.f, -2.f, -2.f}, "the first loop fails");
    expect(0, 1, {1.05f, 1.0f, 1.09f}, {3.f, 4.f, 0.f}, "one is not to be had");
    expect(1, 1, {1.05f, 1.0f, 1e30f}, {0.f, 0.f, -2.f}, "none is");
    // the first two are the more accurate ones
    expect(1, 2, {1.05f, 1.0f, 1.0f, 1.09f}, {3.f, 2.03f, 2.1f, 2.f}, "a tie goes to them", 2);
    expect(3, 2, {1.05f, 1.0f, 1.0f, 1.09f}, {3.f, 2.2f, 2.1f, 2.f}, "more than a tie does not", 2);
    expect(3, 2, {1.5f, 1.4f, 1.0f, 1.09f}, {-2.f, -2.f, 2.1f, 2.f}, "they are far off", 2);
    expect(2, 2, {1.05f, 1.0f, 1.0f}, {2.f, -1.f, 2.f}, "one of their loops fails", 2);
    expect(0, 2, {1.05f, 1.0f, 1.0f}, {2.f, 0.f, 2.01f}, "one is not to be had", 2);
    return bad;
}
"""


def test_loop_times_decide_only_together(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++20", "-I", os.path.join(ROOT, "perix_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
