"""The tensor-core sweep of up to 64 modes (rg_sweep_sym.cu) at the edges of its 16-mode tiles: one mode short of a
tile, a full one and one more, for every tile count; odd and tiny transverse grids; the shortest guides; the
deposition matrix, whose source slice lies inside the guide.  Bars as in test_gpu_parity.py: t and r within 1e-10 of
the oracle (relative Frobenius), T within 1e-9; no realization may need the pivoted kernel."""
import numpy as np
import pytest

import oracle as O
import recurgreen_gb300 as rg

pytestmark = pytest.mark.gpu


def guide(m, ny, nx, **kw):
    return dict(boundtype="dirichlet", nxdiso=nx, nxfree=kw.pop("nxfree", 1), wol=(m + 0.5) / 2, exfac=1.0, aratio=1.0,
                dscat=3.0, ny=ny, **kw)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dabso", [0.0, 0.4])
@pytest.mark.parametrize("m", [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64])
def test_tile_edges(m, dabso):
    kw = guide(m, 2 * m + 1, 6, dabso=dabso)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    u = o.potential(4)
    ro, to = o.refl_trans_v1_upot(u)
    r, t = g.refl_trans_v1_upot(u, want_r=True)
    assert rel(t, to) <= 1e-10 and rel(r, ro) <= 1e-10
    T = g.tdistrib_batch(np.array([9, 4, 7], np.int32)).reshape(3, -1)
    assert g.last_batch_info()["kernel"] == "symmetric" and g.last_batch_info()["rerun"] == 0
    assert np.max(np.abs(T[1] - o.tdistrib_upot(u))) <= 1e-9


@pytest.mark.parametrize("m,ny,nx", [(3, 1, 4), (9, 2, 2), (20, 5, 3), (50, 301, 2), (64, 64, 3)])
def test_small_grids_and_short_guides(m, ny, nx):
    kw = guide(m, ny, nx, nxfree=0)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    u = o.potential(2)
    assert rel(g.refl_trans_v1_upot(u), o.refl_trans_v1_upot(u)[1]) <= 1e-10


@pytest.mark.parametrize("m", [8, 24, 40, 64])
def test_source_inside_the_guide(m):
    kw = guide(m, m, 7)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    for fpos, ipos in ((9, 1), (3, 5), (7, 4)):
        assert rel(g.compute_deposition(3, fpos, ipos), o.deposition_upot(o.potential(3), fpos, ipos)) <= 1e-10


def test_classes_that_share_a_pivoted_kernel():
    """Guides of 33 to 48 and of 49 to 64 modes are different launches of one multi call, but share the pivoted
    kernel, whose shared memory follows the widest grid of either."""
    gs = [rg.Waveguide(**guide(60, 240, 5)), rg.Waveguide(**guide(40, 40, 5))]
    res, st = rg.tdistrib_multi([(gs[k % 2], 1 + k) for k in range(4)], return_status=True)
    assert np.all(st == 0) and all(np.any(T > 0) for T in res)
    for k, T in enumerate(res):
        one = np.zeros((1 + k) * gs[k % 2].neigv)
        gs[k % 2].compute_tdistrib(1 + k, one)
        np.testing.assert_array_equal(T, one[k * gs[k % 2].neigv:])


@pytest.mark.parametrize("m,napera,naperb", [(1, 1.0, 1.0), (2, 1.0, 0.6), (13, 0.5, 1.0), (33, 1.0, 0.7), (64, 0.9, 0.8),
                                             (65, 1.0, 1.0), (72, 0.6, 1.0), (100, 1.0, 0.5), (130, 0.03, 1.0)])
def test_eigenvalues_are_the_squared_singular_values_of_t(m, napera, naperb):
    """Tall, wide and square filter windows: every singular value within 64 eps ||t|| of LAPACK's for the same t (both
    reductions are backward stable), whatever the number of CTAs a realization gets."""
    kw = guide(m, m + 3, 4, dabso=0.2, napera=napera, naperb=naperb)
    g = rg.Waveguide(**kw)
    T, t = g.tdistrib_upot(O.Waveguide(**kw).potential(6), want_t=True)
    s = np.linalg.svd(t, compute_uv=False)
    assert np.all(np.diff(T) <= 0)
    assert np.max(np.abs(np.sqrt(T) - s[: T.size])) <= 64 * np.finfo(float).eps * s[0]
    many = g.tdistrib_batch(np.arange(1, 301, dtype=np.int32)).reshape(300, -1)
    np.testing.assert_array_equal(many[5], g.tdistrib_batch(np.array([6], np.int32)))


@pytest.mark.parametrize("dabso,exfac", [(0.0, 1.0), (0.4, 1.3)])
@pytest.mark.parametrize("m,ny,nxfree", [(1, 1, 0), (1, 6, 1), (3, 3, 1), (15, 15, 0), (17, 40, 2), (31, 33, 1), (33, 16, 0),
                                         (47, 47, 1), (49, 101, 0), (63, 64, 1)])
def test_periodic_guides_in_real_modes(m, ny, nxfree, dabso, exfac):
    """t, r and filtered T of periodic guides, which this kernel sweeps in the modes cos and sin, at tile edges, with
    closed channels, and on odd, even and tiny grids; a batch gives the single call's bits.  (Closed channels decay by
    exp(10) over one of these long slices: there the kernel may pass realizations on.)"""
    kw = dict(boundtype="periodic", nxdiso=6, nxfree=nxfree, wol=(m // 2 + 0.45) / exfac, exfac=exfac, aratio=1.0,
              dscat=3.0, dabso=dabso, ny=ny, napera=0.8, naperb=0.6)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    assert g.nmu == m
    u = o.potential(4)
    ro, to = o.refl_trans_v1_upot(u)
    r, t = g.refl_trans_v1_upot(u, want_r=True)
    assert rel(t, to) <= 1e-10 and rel(r, ro) <= 1e-10
    T = g.tdistrib_batch(np.arange(1, 401, dtype=np.int32)).reshape(400, -1)
    info = g.last_batch_info()
    assert info["kernel"] == "symmetric" and (info["rerun"] == 0 or exfac > 1.0)
    assert np.max(np.abs(T[3] - o.tdistrib_upot(u))) <= 1e-9
    np.testing.assert_array_equal(T[3], g.tdistrib_batch(np.array([4], np.int32)))


@pytest.mark.parametrize("m,nabs", [(3, 1), (16, 1), (16, 2), (64, 3), (70, 2), (100, 4)])
def test_transmission_of_strongly_absorbing_guides(m, nabs):
    """A clean absorbing guide transmits T_k = exp(-2 Im mu_k (nx - 1) kdx) exactly, down to values whose root, or its
    square, underflows: the eigenvalue and eigenvector stages scale t, so no value is lost (relative error of nx slices
    of M-term sums below 1e-10) and none is NaN."""
    nx, dabso = 40, 700.0 * nabs
    wol = (m + 0.5) / 2
    kl = 2 * np.pi * wol
    mu = np.sqrt(1 - (0.5 * np.arange(1, m + 1) / wol) ** 2 + 1j * dabso / kl)
    want = np.sort(np.exp(-2 * mu.imag * kl * (nx - 1) / nx))[::-1]
    g = rg.Waveguide(**dict(guide(m, 2 * m + 1, nx, nxfree=0, dabso=dabso), dscat=0.0))
    T = np.asarray(g.tdistrib_batch(np.array([1], np.int32))).ravel()
    assert np.all(np.isfinite(T))
    assert np.all(np.abs(T - want) <= 1e-10 * want + 1e-300)
    p, nt = g.compute_tprofile(1, 0.0, 0.1)
    assert nt == m and np.all(np.isfinite(p))


@pytest.mark.parametrize("m,dabso", [(40, 700.0), (70, 700.0), (100, 400.0), (33, 300.0)])
def test_small_transmissions_of_clean_guides_keep_their_digits(m, dabso):
    """Where modes do not mix, every T has the relative accuracy of its own mode, however much smaller than the
    largest it is (here by up to 1e-63; nx slices of M-term sums: below 1e-10)."""
    nx = 40
    wol = (m + 0.5) / 2
    kl = 2 * np.pi * wol
    mu = np.sqrt(1 - (0.5 * np.arange(1, m + 1) / wol) ** 2 + 1j * dabso / kl)
    want = np.sort(np.exp(-2 * mu.imag * kl * (nx - 1) / nx))[::-1]
    T = np.asarray(rg.Waveguide(**dict(guide(m, m, nx, nxfree=0, dabso=dabso), dscat=0.0)).tdistrib_batch(
        np.array([1], np.int32))).ravel()
    assert np.all(np.abs(T - want) <= 1e-10 * want)


@pytest.mark.parametrize("bt,m,nx,dscat,seeds", [
    ("dirichlet", 20, 60, 20.0, (4035, 5037, 5194)), ("dirichlet", 20, 60, 30.0, (769, 1121, 1472)),
    ("dirichlet", 20, 60, 100.0, (2643, 2666)), ("periodic", 19, 60, 30.0, (68, 1836, 4053)),
    ("periodic", 19, 60, 50.0, (3880, 4274, 4640)), ("dirichlet", 32, 60, 30.0, (1908, 2396)),
    ("periodic", 31, 60, 20.0, (630,)), ("dirichlet", 40, 40, 100.0, (1644, 2022)), ("periodic", 39, 40, 60.0, (550, 856)),
    ("dirichlet", 64, 30, 100.0, (22, 1272, 1464)), ("periodic", 63, 30, 100.0, (593,))])
def test_inverses_with_rows_of_very_different_size(bt, m, nx, dscat, seeds):
    """Strong disorder: realizations in which some slice's inverse has entries beyond what the fixed point of their row
    holds (found among thousands by comparison with the pivoted kernel; they gave T up to 7000)."""
    kw = dict(boundtype=bt, nxdiso=nx, nxfree=0, wol=(m + 0.5) / 2 if bt == "dirichlet" else m // 2 + 0.45, exfac=1.0,
              aratio=1.0, dscat=dscat, ny=m + 2)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    T = g.tdistrib_batch(np.array(seeds, np.int32)).reshape(len(seeds), -1)
    for k, s in enumerate(seeds):
        assert np.max(np.abs(T[k] - o.tdistrib_upot(o.potential(s)))) <= 1e-9


@pytest.mark.parametrize("bt", ["dirichlet", "periodic"])
@pytest.mark.parametrize("m,nx,aratio,exfac,dabso", [(11, 3, 1.0, 1.3, 0.0), (21, 5, 1.0, 1.3, 0.0), (33, 5, 1.0, 2.0, 0.3),
                                                     (47, 12, 2.0, 1.1, 0.0), (49, 4, 1.0, 1.3, 0.5), (63, 40, 3.0, 1.3, 0.0),
                                                     (63, 2, 1.0, 2.0, 0.0)])
def test_closed_channels_on_coarse_slices(bt, m, nx, aratio, exfac, dabso):
    """Closed channels that decay by up to exp(60) over a slice: t, r, the filtered T and the deposition matrix from this
    kernel, none passed on (but for small pivots in the guide of two slices, which share an optical depth of 3)."""
    wol = ((m + 0.5) / 2 if bt == "dirichlet" else m // 2 + 0.45) / exfac
    kw = dict(boundtype=bt, nxdiso=nx, nxfree=1, wol=wol, exfac=exfac, aratio=aratio, dscat=3.0, dabso=dabso, ny=m + 2)
    o, g = O.Waveguide(**kw), rg.Waveguide(**kw)
    assert g.nmu == m
    u = o.potential(4)
    ro, to = o.refl_trans_v1_upot(u)
    r, t = g.refl_trans_v1_upot(u, want_r=True)
    assert rel(t, to) <= 1e-10 and rel(r, ro) <= 1e-10
    T = g.tdistrib_batch(np.arange(1, 201, dtype=np.int32)).reshape(200, -1)
    info = g.last_batch_info()
    assert info["kernel"] == "symmetric" and (info["rerun"] == 0 or (nx == 2 and info["rerun"] < 100))
    assert np.max(np.abs(T[3] - o.tdistrib_upot(u))) <= 1e-9
    np.testing.assert_array_equal(T[3], g.tdistrib_batch(np.array([4], np.int32)))
    assert rel(g.compute_deposition(4, nx, 2), o.deposition_upot(u, nx, 2)) <= 1e-10
