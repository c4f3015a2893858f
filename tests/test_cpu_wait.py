"""The kernels' waits with a limit (csrc/wait.cuh), on the CPU: a thread that
waits for many phases which never come, or several that share its flag, poll
one limit's worth and then a burst of 64 per phase, and say so each time; waits
that end poll until their phase is there."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include "wait.cuh"
int main() {
    long polls = 0;
    bool any = false;
    int out = 0;
    for (int k = 0; k < 5000; ++k) any |= uva::bounded_wait([&]() { ++polls; return false; }, 1000, out);
    std::printf("%ld %d %d\n", polls, any, out);
    long ok = 0;
    polls = 0;
    out = 0;
    for (int k = 0; k < 5000; ++k) {
        int left = k % 1000;
        ok += uva::bounded_wait([&]() { ++polls; return left-- == 0; }, 1000, out);
    }
    std::printf("%ld %ld %d\n", ok, polls, out);
    int left = 10;   // the phase comes after the limit: later waits poll a burst
    const bool first = uva::bounded_wait([&]() { return left-- == 0; }, 10, out);
    polls = 0;
    const bool second = uva::bounded_wait([&]() { ++polls; return true; }, 10, out);
    const bool third = uva::bounded_wait([&]() { ++polls; return false; }, 1000, out);
    std::printf("%d %d %d %ld %d\n", first, second, third, polls, out);
}
"""


def test_waits_share_one_limit(tmp_path):
    here = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "w.cpp").write_text(SRC)
    exe = str(tmp_path / "w")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(here, "ultimate_uv_artist_b200", "csrc"),
                    str(tmp_path / "w.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split("\n")
    assert out[0] == f"{1000 + 4999 * 64} 0 2"
    assert out[1] == f"5000 {5 * sum(range(1, 1001))} 0"
    assert out[2] == "0 1 0 65 2"
