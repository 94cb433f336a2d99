"""The tensor-core sweeps round to fixed point without a bias.  Without absorption t^H t + r^H r = 1; rounding makes
each slice gain or lose some 2^-55 of it at random, which averages out over slices and realizations, where a bias of one
sign grows with the number of slices (ties rounded away from zero: the mean of trace(t^H t + r^H r - 1) / M was 2e-17 to 1e-16 a
slice)."""
import numpy as np
import pytest

import recurgreen_gb300 as rg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,ny,nx,dscat", [(37, 37, 150, 6.0), (48, 100, 80, 5.0), (64, 256, 300, 3.0), (81, 200, 60, 8.0)])
def test_flux_has_no_drift(m, ny, nx, dscat):
    """Bar: a mean over 24 realizations of at most a quarter of what ties away from zero give, 5e-18 a slice."""
    g = rg.Waveguide("dirichlet", nxdiso=nx, nxfree=0, wol=(m + 0.5) / 2, exfac=1.0, aratio=1.0, dscat=dscat, ny=ny)
    r, t = g.refl_trans_v1_batch(np.arange(1, 25, dtype=np.int32))
    flux = (np.sum(np.abs(t) ** 2, axis=(1, 2)) + np.sum(np.abs(r) ** 2, axis=(1, 2))) / m - 1
    assert abs(np.mean(flux)) <= 5e-18 * nx
