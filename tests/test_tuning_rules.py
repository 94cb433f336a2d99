"""The rules of the launch tuner (rg_internal.h): which choices are timed, and which guides share them."""
import os
import subprocess

import pytest

from recurgreen_gb300 import build

SRC = r"""
#include "rg_internal.h"
#include <cstdio>
int main() {
  int m, symmetric, tensor, split, periodic;
  while (std::scanf("%d %d %d %d %d", &m, &symmetric, &tensor, &split, &periodic) == 5) {
    rg::SweepArgs a{};
    a.max_M = m, a.symmetric = symmetric, a.tensor_r = tensor, a.split_inverse = split;
    std::printf("%d %d\n", rg::row_split_matters(a, periodic) ? 1 : 0, rg::tuned_kernel(a, periodic));
  }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "tune.cpp").write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run([build.cxx(), "-std=c++17", "-I", build.CSRC, "-I", inc, str(d / "tune.cpp"), "-o", str(d / "tune")],
                   check=True)

    def run(*form):
        out = subprocess.run([str(d / "tune")], input=" ".join(map(str, form)), capture_output=True, text=True, check=True)
        return tuple(map(int, out.stdout.split()))

    return run


def test_row_splits_are_timed_only_where_slices_are_eliminated(rules):
    # modes, symmetric, tensor product, split levels, periodic
    assert rules(100, 1, 1, 3, 0)[0] == 0 and rules(512, 1, 1, 3, 0)[0] == 0
    assert rules(64, 1, 1, 2, 0)[0] == 0 and rules(100, 0, 1, 2, 0)[0] == 0 and rules(100, 1, 1, 2, 1)[0] == 0
    for form in ((100, 1, 0, 3, 0), (513, 1, 1, 3, 0), (100, 1, 1, 0, 0), (300, 1, 1, 1, 0), (300, 1, 1, 2, 0)):
        assert rules(*form)[0] == 1


def test_other_kernels_have_choices_of_their_own(rules):
    forms = [(100, s, t, l, p) for s in (0, 1) for t in (0, 1) for l in (0, 1, 2, 3) for p in (0, 1)]
    kernels = {}
    for s, t, l, p in (f[1:] for f in forms):
        runs = ("symmetric", t, l) if s and not p else ("pivoted", p)
        kernels.setdefault(rules(100, s, t, l, p)[1], set()).add(runs)
    assert all(len(v) == 1 for v in kernels.values()) and len(kernels) == len(set().union(*kernels.values()))
    assert rules(51, 1, 1, 3, 1)[1] != rules(51, 0, 1, 3, 1)[1]
