"""The HMC predecessor's congrad on the smallest lattices (csrc/hmc_planes.cuh): two
sites a row, both walls next to each other.  With weak fields it converges below its
cap of kthird*kvol iterations, so x itself is checked: M^dagger M x, by the oracle's
operator, is Phi up to the residual at which the solve stops, sqrt(kferm) res, and
what REAL*4 vectors lose: half an ulp of terms of at most ||M||^2 ||x|| an iteration,
||M|| <= 11 (diagonal 3, six hops of norm 1, two s hops)."""
import numpy as np
import pytest

import pyoracle as po
import chiralheisenberg_b200 as chb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 7, 2), (2, 9, 3), (3, 4, 2)])
@pytest.mark.parametrize("imass", [1, 3])
def test_hmc_congrad_converges_on_the_smallest_lattices(shape, imass):
    L, Lt, Ls = shape
    rng = np.random.default_rng(L * 100 + Lt * 10 + Ls)
    sh = (2, 4, Lt, L, L, Ls)
    Phi = (rng.standard_normal(sh) + 1j * rng.standard_normal(sh)).astype(np.complex64)
    chi = (0.05 * rng.standard_normal((3, L * L * Lt))).astype(np.float32)
    lat = po.make_lat(L, Lt, Ls, beta=0.475)
    res = 1e-4
    xo, ito, capo = po.hmc_congrad(lat, Phi, chi, Phi, res, imass)
    h = chb.Hmc(L, Lt, Ls, 0.1, 0.475, 1.0, 0.0, imass, 5)
    try:
        xg, itg, capg = h.congrad(Phi, chi, Phi, res)
    finally:
        h.close()
    assert not capo and not capg
    assert abs(itg - ito) <= max(3, 0.1 * ito), (itg, ito)
    for x, it in ((xo, ito), (xg, itg)):
        mx = po.hmc_dslash(lat, x.astype(np.complex64), chi, imass)
        r = Phi - po.hmc_dslash(lat, mx, chi, imass, dag=True)
        bound = np.sqrt(Phi.size) * res + it * 2.0 ** -24 * 121 * np.linalg.norm(x)
        assert np.linalg.norm(r) <= bound, (np.linalg.norm(r), bound)
