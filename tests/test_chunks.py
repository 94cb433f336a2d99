"""Realizations per launch where device memory is short (rg_internal.h): their buffers and the sweep's workspace, which
above 64 modes is of the same order, have to fit together."""
import os
import subprocess

import pytest

from recurgreen_gb300 import build

SRC = r"""
#include "rg_internal.h"
#include <algorithm>
#include <cstdio>
int main() {
  long long c, item, free_bytes, work, slots;
  while (std::scanf("%lld %lld %lld %lld %lld", &c, &item, &free_bytes, &work, &slots) == 5)
    std::printf("%d\n", rg::fitting_chunk((int)c, item, free_bytes,
                                          [&](int k) { return (size_t)(work * std::min<long long>(k, slots)); }));
}
"""
MB, GB = 1 << 20, 1 << 30


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunk")
    (d / "chunk.cpp").write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run([build.cxx(), "-std=c++17", "-I", build.CSRC, "-I", inc, str(d / "chunk.cpp"), "-o", str(d / "chunk")],
                   check=True)

    def run(*a):
        return int(subprocess.run([str(d / "chunk")], input=" ".join(map(str, a)), capture_output=True, text=True,
                                  check=True).stdout)

    return run


def test_workspace_fits_beside_the_realizations(chunk):
    for c, item, free, work in ((250, 20 * MB, 10 * GB, 42 * MB), (37, 138 * MB, 10 * GB, 42 * MB), (300, 4 * MB, 2 * GB, 11 * MB),
                                (1, 9 * GB, 10 * GB, 4 * GB), (2, 4 * GB, 10 * GB, 4 * GB)):
        k = chunk(c, item, free, work, 304)
        assert 1 <= k <= c
        assert k == 1 or k * item + work * min(k, 304) <= free * 15 // 16
        more = k + (k + 2) // 3 + 1
        assert k == c or more > c or more * item + work * min(more, 304) > free * 11 // 16  # nothing much is given away


def test_plenty_of_memory_changes_nothing(chunk):
    assert chunk(608, 20 * MB, 270 * GB, 42 * MB, 304) == 608
