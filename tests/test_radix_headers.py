"""The numpy restatement of the row transform (test_row_transform) and the build's list of kernel sets
hold the library's own numbers: the radix plans, row splits and twiddle tables of
radix_plan.h and kernel_table.h, printed by a host program compiled from them."""
import os
import re
import subprocess

from conftest import ROOT
from mm_propagation_b200 import build
from test_row_transform import PLANS, max_split

CSRC = os.path.join(ROOT, "mm_propagation_b200", "csrc")

PROGRAM = """
#include "kernel_table.h"
#include <cstdio>
using namespace mmp;
int main() {
  for (int L = kMinLogN; L <= kMaxLogN; ++L) {
    const RadixPlan p = radix_plan(L);
    std::printf("%d %d %d %zu %zu", L, max_split(false, L), max_split(true, L), twiddle_entries(L), twiddle_offset(L));
    for (int i = 0; i < p.n; ++i) std::printf(" %d", p.r[i]);
    std::printf("\\n");
  }
}
"""


def test_plans_and_splits_are_the_headers(tmp_path):
    src, exe = tmp_path / "plans.cpp", tmp_path / "plans"
    src.write_text(PROGRAM)
    subprocess.run([build.CXX, "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    offset = 0
    for line, L in zip(lines, range(6, 17), strict=True):
        v = [int(x) for x in line.split()]
        r = PLANS[L]
        left = [L]
        for x in r:
            left.append(left[-1] - x)
        entries = sum(1 << x for x in left[:len(r) - 1])  # every pass but the last
        assert left[-1] == 0
        assert v == [L, max_split(0, L), max_split(1, L), entries, offset, *r]
        assert build._max_split(False, L) == max_split(0, L) and build._max_split(True, L) == max_split(1, L)
        offset += entries


def test_every_built_kernel_set_is_listed():
    text = open(os.path.join(CSRC, "solver.cu")).read()
    listed = re.findall(r"X\((f32|f64), (\d+), (\d+)\)", text)
    want = [(tag, L, x) for tag, fp64 in (("f32", 0), ("f64", 1)) for L in range(6, 17)
            for x in range(max_split(fp64, L) + 1)]
    assert sorted((t, int(L), int(x)) for t, L, x in listed) == sorted(want)
