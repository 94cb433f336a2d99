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


@pytest.mark.parametrize("m,nx,dscat,n,bar", [(65, 20, 300.0, 600, 1e-11), (65, 20, 30000.0, 600, 3e-10), (100, 12, 3000.0, 400, 8e-11),
                                              (200, 8, 3000.0, 300, 2e-10), (200, 8, 30000.0, 300, 1e-8)])
def test_block_inverse_under_strong_disorder(monkeypatch, m, nx, dscat, n, bar):
    """T against the pivoted kernel's where leading blocks are often nearly singular: within 30 times what the symmetric
    elimination of the whole matrix differs from it by (3.5e-13, 1.1e-11, 2.7e-12, 6.9e-12 and 4.7e-10 at most)."""
    g = rg.Waveguide("dirichlet", nxdiso=nx, nxfree=0, wol=(m + 0.5) / 2, exfac=1.0, aratio=1.0, dscat=dscat, ny=m + 2)
    seeds = np.arange(1, n + 1, dtype=np.int32)
    T = g.tdistrib_batch(seeds)
    assert g.last_batch_info()["rerun"] < n // 2  # most T are this kernel's own
    monkeypatch.setenv("RG_SYMMETRIC", "0")
    assert np.max(np.abs(T - g.tdistrib_batch(seeds))) <= bar


@pytest.mark.parametrize("levels", ["0", "1", "2"])
@pytest.mark.parametrize("m", [67, 128, 130, 300])
def test_fewer_block_levels(monkeypatch, levels, m):
    """RG_SPLIT_INVERSE=0, 1, 2: the blocks left are eliminated, whole ones of more than 64 modes among them."""
    monkeypatch.setenv("RG_SPLIT_INVERSE", levels)
    kw = guide(m, m + 3, 3, dabso=0.2)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    u = o.potential(4)
    ro, to = o.refl_trans_v1_upot(u)
    r, t = g.refl_trans_v1_upot(u, want_r=True)
    assert rel(t, to) <= 1e-10 and rel(r, ro) <= 1e-10
