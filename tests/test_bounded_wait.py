"""The loop of the GEMM's bounded waits (lt_wait.cuh), compiled for the host with a barrier that never completes."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))

PROGRAM = r"""
#include <cstdio>
#include "lt_wait.cuh"
static long long t;
static int sleeps, given_up;
static void wait(volatile int* flag, int after) {     // the barrier completes at the after-th look (0: never); a look takes 100 clocks
    sleeps = 0;
    lt::tc::bounded_wait([&] { t += 100; return ++sleeps == after; }, [] { return t; }, 1000, flag, [&] { *flag = 1; given_up++; });
    std::printf("%d %d\n", sleeps, given_up);
}
int main() {
    volatile int flag = 0;
    wait(&flag, 1);      // complete at once
    wait(&flag, 3);      // after a while
    wait(&flag, 0);      // runs out of time
    wait(&flag, 0);      // later waits do not sleep
    wait(&flag, 1);
}
"""


def test_waits_after_a_timeout_return_without_a_sleep(tmp_path):
    src, exe = tmp_path / "w.cpp", str(tmp_path / "w")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(HERE, "..", "llamatov_b200", "csrc"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout.split("\n")[:5]
    assert out == ["1 0", "3 0", "12 1", "0 1", "0 1"]
