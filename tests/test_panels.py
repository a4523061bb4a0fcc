"""The on-chip solvers' shared-memory budget (csrc/panels.h): how many of a CTA's panels each of its slices
keeps, for slices of every width down to one block, against what the kernels rely on."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <vector>
#include "panels.h"
int main() {  // lines "cap n w0 w1 ..." -> the kept panels of each slice
    int cap, n;
    while (scanf("%d %d", &cap, &n) == 2) {
        std::vector<int> w(n), k(n);
        for (int& x : w) if (scanf("%d", &x) != 1) return 1;
        keptPanels(w.data(), n, cap, k.data());
        for (int x : k) printf("%d ", x);
        printf("\n");
    }
    return 0;
}
"""


def kept(tmp_path, cases):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "k.cpp").write_text(SRC)
    subprocess.run([cxx, "-O1", "-I", os.path.join(ROOT, "clothsimulator_b200", "csrc"), str(tmp_path / "k.cpp"), "-o",
                    str(tmp_path / "k")], check=True)
    text = "\n".join(f"{cap} {len(w)} " + " ".join(map(str, w)) for cap, w in cases)
    out = subprocess.run([str(tmp_path / "k")], input=text, capture_output=True, text=True, check=True).stdout
    return [list(map(int, ln.split())) for ln in out.splitlines()]


def even(cap, w):
    """The even deal alone: a narrow slice's remainder goes nowhere."""
    over, n = max(sum(w) - cap, 0), len(w)
    return [x - min(x, over * (j + 1) // n - over * j // n) for j, x in enumerate(w)]


def test_kept_panels_fill_the_budget_and_no_more(tmp_path):
    rng = np.random.default_rng(0)
    # nodes without a face make slices of one block per row: the even deal alone exceeds the budget
    narrow = (179, [13] * 14 + [14, 1])
    assert sum(even(*narrow)) > narrow[0]
    cases = [narrow, (165, [1, 1] + [13] * 13 + [11]), (0, [1, 1, 1]), (5, [3]), (40, [13, 13, 13])]
    for _ in range(400):
        n = int(rng.integers(1, 17))
        w = [int(x) for x in rng.choice([1, 1, 2, 9, 13, 16, 18], n)]
        cases.append((int(rng.integers(0, sum(w) + 3)), w))
    for (cap, w), k in zip(cases, kept(tmp_path, cases)):
        assert sum(k) == min(cap, sum(w)), (cap, w, k)
        assert all(0 <= a <= b for a, b in zip(k, w)), (cap, w, k)
        if sum(even(cap, w)) == min(cap, sum(w)):  # no slice is narrower than its share
            assert k == even(cap, w)
