"""The loop of the tensor-core GEMMs' waits (csrc/bounded_wait.cuh) with a barrier that is counted instead of tried: a wait ends after the
budget that the bulk-copy kernels' waits have, and once one has run out the others of the CTA end at once."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "mnemocuda_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "bounded_wait.cuh"
static void go(uint32_t ready_at, int raised)
{
    volatile int flag = raised;
    uint32_t tries = 0;
    mb200::bounded_wait([&] { return ++tries == ready_at; }, [] {}, &flag);
    std::printf("%u %d\n", tries, static_cast<int>(flag));
}
int main()
{
    std::printf("%u\n", mb200::kWaitBudget);
    go(1, 0);  // ready at once
    go(1, 1);
    go(200, 0);
    go(0, 0);  // never
    go(0, 1);  // never, after another wait ran out
}
"""


def test_a_wait_ends(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    budget = int(lines[0])
    out = [tuple(map(int, l.split())) for l in lines[1:6]]
    assert out[:3] == [(1, 0), (1, 1), (200, 0)]
    tries, flag = out[3]
    assert flag == 1 and budget <= tries <= budget + 1
    tries, flag = out[4]
    assert flag == 1 and tries <= 2
