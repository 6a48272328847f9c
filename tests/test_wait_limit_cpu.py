"""The test that every bounded device-side wait makes against its limit (csrc/wait_limit.h; no GPU needed)."""

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "frac-ssm-kernels_b200", "csrc")
LIMIT = 2_000_000_000
CASES = [  # start, now, gives up
    (1000, 1000, 0), (1000, 1000 + LIMIT, 0), (1000, 1001 + LIMIT, 1),
    (1000, 999, 0), (1000, 0, 0), (5 * LIMIT, 5 * LIMIT - 1024, 0),      # a reading before the start: nothing has passed
    (2 ** 64 - 10, 20, 0), (2 ** 64 - 10, LIMIT, 1),                     # the timer wraps
]


def test_only_time_that_has_passed_counts(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    calls = "".join(f"std::putchar('0' + fracssm::umma::past_limit({s}ull, {n}ull, {LIMIT}ull));" for s, n, _ in CASES)
    src.write_text(f'#include <cstdio>\n#include "wait_limit.h"\nint main() {{ {calls} }}\n')
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    got = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert got == "".join(str(g) for *_, g in CASES)


def test_no_wait_subtracts_the_timer_itself():
    """(such a difference would be unsigned)"""
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            assert "global_ns() -" not in open(os.path.join(CSRC, name)).read(), name
