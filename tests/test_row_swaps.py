"""row_swaps.h: the coarsest inverse's row swaps undone, and a table of swaps that no
elimination wrote (the device's, after a kernel that did not run) refused before
anything is indexed by it."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "curvib_old_gb300" / "csrc"

# perm and map end at the end of the arrays, guard values around them
MAIN = r"""
#include <cstdio>
#include <vector>
#include "row_swaps.h"
int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    std::vector<int> perm(n), map(n + 2, -7);
    for (int &v : perm) if (std::scanf("%d", &v) != 1) return 1;
    const bool ok = cvb::undo_row_swaps(perm.data(), n, map.data() + 1);
    if (map[0] != -7 || map[n + 1] != -7) return 1;
    std::printf("%d", ok);
    for (int q = 0; ok && q < n; q++) std::printf(" %d", map[q + 1]);
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("row_swaps")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(perms):
        text = "".join(f"{len(p)} {' '.join(map(str, p))}\n" for p in perms)
        r = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True)
        assert r.returncode == 0
        return [[int(v) for v in line.split()] for line in r.stdout.splitlines()]
    return run


def test_swaps_are_undone(program):
    rng = np.random.default_rng(4)
    perms = [[int(rng.integers(c, n)) for c in range(n)] for n in (1, 2, 3, 7, 64, 216)]
    for p, (ok, *got) in zip(perms, program(perms)):
        # rows swapped: P A; its inverse is A^-1 P^-1, so column q of A^-1 is column
        # (where row q went) of it
        rows = np.arange(len(p))
        for c, r in enumerate(p):
            rows[[c, r]] = rows[[r, c]]
        assert ok and got == np.argsort(rows).tolist()


@pytest.mark.parametrize("n", [1, 2, 9])
def test_no_row_is_refused(program, n):
    bad = []
    for c in range(n):
        for v in (-1, c - 1, n, 2**31 - 1, -2**31):
            p = list(range(n))
            p[c] = v
            bad.append(p)
    assert all(r == [0] for r in program(bad))


def test_the_device_inverse_uses_it():
    text = (CSRC / "kernels_setup.cu").read_text()
    assert "undo_row_swaps(h_perm.data(), n, map.data())" in text and "map[h_perm" not in text
