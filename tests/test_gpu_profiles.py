"""Profiles of open transmission eigenstates (rg_green.cu) at the sizes where their kernels change: one mode, the edges
of the 16-mode tiles, the largest matrix whose vectors are found in shared memory (78 modes) and the next.  Bars as in
test_green.py: 1e-9 of the oracle, relative."""
import numpy as np
import pytest

import oracle as O
import recurgreen_gb300 as rg

pytestmark = pytest.mark.gpu


def window(tv, lo, hi):
    """The window's edges moved to the middle of the gaps between the eigenvalues next to them."""
    def mid(x):
        s = np.concatenate([[0.0], np.sort(tv), [1.0]])
        k = np.searchsorted(s, x)
        return (s[k - 1] + s[k]) / 2 if 0 < k < s.size and s[k] - s[k - 1] > 1e-6 else x
    return mid(lo), mid(hi)


@pytest.mark.parametrize("bt,m", [("periodic", m) for m in (1, 17, 63, 81)] + [
    ("dirichlet", m) for m in (1, 2, 7, 15, 16, 17, 32, 33, 48, 49, 63, 64, 65, 77, 78, 79, 101)])
def test_profiles_at_kernel_edges(bt, m):
    wol = (m + 0.5) / 2 if bt == "dirichlet" else m // 2 + 0.4
    kw = dict(boundtype=bt, nxdiso=9, nxfree=1, wol=wol, exfac=1.0, aratio=1.0, dscat=4.0, ny=m + 2)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    assert g.nmu == m
    u = o.potential(3)
    tv = np.linalg.svd(o.refl_trans_v1_upot(u)[1], compute_uv=False) ** 2
    lo, hi = window(tv, 0.05, 0.97)
    p, nt = g.compute_tprofile(3, lo, hi)
    po, nto = o.tprofile_upot(u, lo, hi)
    assert nt == nto
    assert np.linalg.norm(p - po) <= 1e-9 * max(np.linalg.norm(po), 1.0)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_matrix_that_is_not_finite_has_no_decomposition(bad):
    a = np.ones((5, 4), complex)
    a[2, 1] = bad
    with pytest.raises(rg.RecurGreenError):
        rg.diagonalize_ahca(a)
