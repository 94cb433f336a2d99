"""The blocked symmetric sweep of more than 64 modes (rg_sweep_large_sym.cu): its 2 x 2 block inverse at sizes whose
halves are odd, at each change of depth, at leaves of one mode more or less than a 16-mode tile, and products of one
row more or less than a 64-row block.  Bars as in test_gpu_parity.py: t and r within 1e-10 of the oracle (relative
Frobenius), T within 1e-9; no realization may need the pivoted kernel."""
import numpy as np
import pytest

import oracle as O
import recurgreen_gb300 as rg

pytestmark = pytest.mark.gpu


def guide(m, ny, nx, **kw):
    return dict(boundtype="dirichlet", nxdiso=nx, nxfree=1, wol=(m + 0.5) / 2, exfac=1.0, aratio=1.0, dscat=3.0, ny=ny,
                **kw)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("m", [65, 66, 67, 71, 95, 96, 97, 127, 128, 129, 131, 161, 191, 193, 255, 256, 257, 300])
def test_sizes_of_the_blocks(m):
    kw = guide(m, m + 3, 4, dabso=0.2)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    u = o.potential(4)
    ro, to = o.refl_trans_v1_upot(u)
    r, t = g.refl_trans_v1_upot(u, want_r=True)
    assert rel(t, to) <= 1e-10 and rel(r, ro) <= 1e-10
    T = g.tdistrib_batch(np.array([9, 4, 7], np.int32)).reshape(3, -1)
    assert g.last_batch_info()["kernel"] == "blocked_symmetric" and g.last_batch_info()["rerun"] == 0
    assert np.max(np.abs(T[1] - o.tdistrib_upot(u))) <= 1e-9


@pytest.mark.parametrize("m", [449, 511, 512])
def test_deepest_split(m):
    kw = guide(m, m, 2, dabso=0.0)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    u = o.potential(2)
    assert rel(g.refl_trans_v1_upot(u), o.refl_trans_v1_upot(u)[1]) <= 1e-10


@pytest.mark.parametrize("m,n", [(65, 400), (130, 200), (257, 160)])
def test_batch_is_the_single_call(m, n):
    """More realizations than clusters fit at once, one CTA each, against one realization spread over a cluster."""
    g = rg.Waveguide(**guide(m, m, 3))
    T = g.tdistrib_batch(np.arange(1, n + 1, dtype=np.int32)).reshape(n, -1)
    for k in (0, n // 2, n - 1):
        np.testing.assert_array_equal(T[k], g.tdistrib_batch(np.array([k + 1], np.int32)))
