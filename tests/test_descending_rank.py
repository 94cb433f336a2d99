"""The order in which rg_green.cu stores eigenvalues and vectors: a permutation for every input, non-finite ones too
(anything else would leave slots that later index memory unset)."""
import itertools
import os
import subprocess

import numpy as np
import pytest

from recurgreen_gb300 import build

SRC = r"""
#include "rg_internal.h"
#include <cstdio>
int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    std::vector<double> t(n);
    for (double& x : t) std::scanf("%lf", &x);
    for (int v = 0; v < n; ++v) std::printf("%d ", rg::descending_rank(t.data(), n, v));
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def ranks(tmp_path_factory):
    d = tmp_path_factory.mktemp("rank")
    (d / "rank.cpp").write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run([build.cxx(), "-std=c++17", "-I", build.CSRC, "-I", inc, str(d / "rank.cpp"), "-o", str(d / "rank")],
                   check=True)

    def run(rows):
        text = "\n".join(f"{len(r)} " + " ".join(repr(float(x)) for x in r) for r in rows)
        out = subprocess.run([str(d / "rank")], input=text, capture_output=True, text=True, check=True).stdout
        return [[int(x) for x in line.split()] for line in out.splitlines()]

    return run


def test_rank_is_a_permutation_with_nan_last(ranks):
    rows = [list(p) for n in (1, 2, 3, 4) for p in itertools.product([0.5, 0.0, np.nan, np.inf], repeat=n)]
    for t, k in zip(rows, ranks(rows), strict=True):
        assert sorted(k) == list(range(len(t)))
        key = sorted(range(len(t)), key=lambda v: (np.isnan(t[v]), -t[v] if t[v] == t[v] else 0.0, v))
        assert [k[v] for v in key] == list(range(len(t)))
