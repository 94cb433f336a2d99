"""Handles on threads of their own.  A kernel's limit of dynamic shared memory belongs to the kernel, not to a launch: one
thread's plan for few modes must not lower it between another's plan and launch for many."""
import glob
import os
import threading

import numpy as np
import pytest

import recurgreen_gb300 as rg
from recurgreen_gb300 import build


def test_limits_are_set_in_one_place():
    users = [os.path.basename(f) for f in glob.glob(os.path.join(build.CSRC, "*"))
             if "cudaFuncAttributeMaxDynamicSharedMemorySize" in open(f).read()]
    assert users == ["rg_internal.h"]


@pytest.mark.gpu
def test_sizes_on_concurrent_threads():
    def guide(m):
        return rg.Waveguide("dirichlet", nxdiso=2, nxfree=0, wol=(m + 0.5) / 2, exfac=1.0, aratio=1.0, dscat=3.0, ny=m)

    calls = {66: 400, 100: 300, 300: 60, 512: 30}
    want = {m: guide(m).tdistrib_batch(np.arange(1, 6, dtype=np.int32)).reshape(5, -1) for m in calls}
    wrong = []

    def work(m):
        g = guide(m)
        out = np.zeros(5 * g.neigv)
        try:
            for k in range(calls[m]):
                g.compute_tdistrib(1 + k % 5, out)
                if not np.array_equal(out.reshape(5, -1)[k % 5], want[m][k % 5]):
                    wrong.append((m, k, "other values"))
        except rg.RecurGreenError as e:
            wrong.append((m, str(e)))

    threads = [threading.Thread(target=work, args=(m,)) for m in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
