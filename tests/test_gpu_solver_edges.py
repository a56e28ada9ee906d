"""The HMC predecessor's congrad (csrc/hmc_planes.cuh) and the Thirring
multi-shift solver (csrc/thirring.cu) at the edges of their launches: odd and
ragged lattices, less than a block of points and many blocks, one pole, poles
that are no multiple of the four a thread takes, solves that end inside a chunk
of iterations.  Against the oracle; congrad's x to 1e-5 of its maximum, which
its REAL*4 vectors set."""
import numpy as np
import pytest

import pyoracle as po
import chiralheisenberg_b200 as chb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 5, 3), (5, 4, 7), (2, 7, 2), (13, 6, 5)])
@pytest.mark.parametrize("imass", [1, 3])
def test_hmc_congrad_shapes(shape, imass):
    L, Lt, Ls = shape
    rng = np.random.default_rng(L * 100 + Lt * 10 + Ls)
    sh = (2, 4, Lt, L, L, Ls)
    Phi = (rng.standard_normal(sh) + 1j * rng.standard_normal(sh)).astype(np.complex64)
    chi = (0.7 * rng.standard_normal((3, L * L * Lt))).astype(np.float32)
    lat = po.make_lat(L, Lt, Ls, beta=0.475)
    xo, ito, capo = po.hmc_congrad(lat, Phi, chi, Phi, 1e-6, imass)
    h = chb.Hmc(L, Lt, Ls, 0.1, 0.475, 1.0, 0.0, imass, 5)
    try:
        for _ in range(2):                # a replayed graph too
            xg, itg, capg = h.congrad(Phi, chi, Phi, 1e-6)
    finally:
        h.close()
    assert capo == capg
    assert abs(itg - ito) <= max(3, 0.1 * ito), (itg, ito)
    if not capo:
        assert np.abs(xg - xo).max() <= 1e-5 * np.abs(xo).max()


@pytest.mark.parametrize("shape", [(2, 3, 4), (3, 2, 5), (5, 3, 4), (9, 7, 6)])
@pytest.mark.parametrize("npole", [1, 5, 12])
@pytest.mark.parametrize("imass", [1, 3, 5])
def test_thirring_qmrherm_shapes(remez, shape, npole, imass):
    """Every x_k solves (M^dagger M + sigma_k) x_k = R with the oracle's
    operator.  The solve stops when its residual estimate is below 2 sqrt(n) res,
    1.4e-6 of |R| = sqrt(2 n); beta enters the recurrences rounded to REAL*4,
    which adds at most 6e-8 |R| an iteration.  x is the weighted sum of the x_k in FP64."""
    L, Lt, Ls = shape
    lat = po.make_lat(L, Lt, Ls)
    rng = np.random.default_rng(L * 100 + Lt * 10 + Ls + npole)
    sh = po.thr_shape(lat)
    R = rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    theta = (0.3 * rng.standard_normal((3, po.kvol(lat)))).astype(np.float32)
    u = po.thr_coef(lat, theta)
    am = np.float32(0.2)
    g = remez["remez2g"]
    num, den = g["anum"][:npole + 1], g["aden"][:npole]
    h = chb.Thirring(L, Lt, Ls, 0.1, 0.5, 1.0, float(am), imass, 4)
    try:
        for _ in range(2):                # a replayed graph too
            x, its, capped, P0, _ = h.qmrherm(R, u, 1e-6, am, imass, num, den, iflag=1)
    finally:
        h.close()
    assert not capped
    total = num[0] * R
    for k in range(npole):
        mx = po.thr_dslash(lat, P0[k], u, am, imass)
        r = R - po.thr_dslash(lat, mx, u, am, imass, dag=True) - den[k] * P0[k]
        assert np.linalg.norm(r) <= (1.4143e-6 + its * 6e-8) * np.linalg.norm(R), k
        total = total + num[k + 1] * P0[k]
    assert np.linalg.norm(x - total) <= 1e-13 * np.linalg.norm(total)
