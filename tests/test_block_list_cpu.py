"""How long the blocks of a decode step wait for one another (csrc/wait_limit.h; no GPU needed)."""

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "frac-ssm-kernels_b200", "csrc")


def _values(tmp_path, calls):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    lines = "".join(f'std::printf("%llu\\n", (unsigned long long)fracssm::{c});' for c in calls)
    src.write_text(f'#include <cstdio>\n#include "wait_limit.h"\nint main() {{ {lines} }}\n')
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return [int(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]


def test_the_list_stays_open_no_longer_than_the_missing_blocks_are_worth(tmp_path):
    work = 500_000
    counts = [148, 147, 140, 74, 2, 1]
    got = _values(tmp_path, [f"list_patience_ns({n}u, 148u, {work}ull)" for n in counts])
    # with n of 148 blocks the work takes 148 / n times as long
    assert got == [10_000 + work * (148 - n) // n for n in counts]
    assert got[0] == 10_000 and got == sorted(got)
    # the longest work of a launch, 32 layers whose weights fill the device's memory, and nobody else: still an end
    assert 0 < _values(tmp_path, [f"list_patience_ns(1u, 148u, {50_000_000_000}ull)"])[0] < 2 ** 63


def test_the_limit_covers_the_work_of_all_by_one(tmp_path):
    work = [640_000, 50_000_000_000]      # 24 layers of hidden 768; layers whose weights fill the device's memory
    got = _values(tmp_path, [f"list_limit_ns(148u, {w}ull, 2000000000ull)" for w in work])
    assert got == [2_000_000_000 + 148 * w for w in work] and got[-1] < 2 ** 63
    # and with it the time that the list may stay open
    assert all(g > p for g, p in zip(got, _values(tmp_path, [f"list_patience_ns(1u, 148u, {w}ull)" for w in work])))
