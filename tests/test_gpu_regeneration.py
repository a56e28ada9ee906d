"""Multi-shift solves that outgrow the stored basis (csrc/lanczos.cu): pass 2
regenerates the Lanczos vectors and takes them into x three at a time, from the
ring of residuals.  x has the bits of the solve with a store, whatever the number
of iterations is modulo three and however many vectors a short store keeps, and
a vector costs two kernels and a third."""
import ctypes as C

import numpy as np
import pytest

import chiralheisenberg_b200 as chb
from conftest import random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (5, 3, 7), (6, 6, 2), (8, 6, 5)])
@pytest.mark.parametrize("imass", [1, 3])
def test_regenerated_solution_has_the_stored_one_s_bits(remez, L, Lt, Ls, imass):
    lib = chb.load_library()
    r = remez["remez2g"]
    Phi, chi = random_fields(L, Lt, Ls, seed=61, chi_scale=0.4)
    vec = 16.0 * Phi.size
    seen = set()
    for res in (1e-2, 3e-3, 1e-3, 3e-4, 1e-4, 1e-5):
        out = []
        for store in (-1.0, 0.0, 8.5 * vec, 9.5 * vec):
            gl = chb.Lattice(L, Lt, Ls, beta=0.475)
            gl.set_basis_store(store)
            n0 = lib.chdwf_kernel_launches()
            x, it, _ = gl.qmrherm(Phi, res, r["anum"], r["aden"], 0, chi, imass=imass)
            out.append((x, it, lib.chdwf_kernel_launches() - n0))
            gl.close()
        m = out[0][1]
        seen.add(m % 3)
        for x, it, n in out[1:]:
            assert it == m
            assert np.array_equal(x, out[0][0]), (res, m)
        # beyond the store's own launches: M and M^dagger for all but the last
        # vector, and one more kernel for three
        assert out[1][2] - out[0][2] <= 2 * (m - 1) + (m + 2) // 3, (m, out[1][2], out[0][2])
    assert len(seen) > 1


@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (5, 3, 7)])
def test_regeneration_from_fp32_vectors(remez, L, Lt, Ls):
    """The Hamiltonian's solve with FP32 vectors: S, a sum over x, is the same number."""
    lib = chb.load_library()
    rng = np.random.default_rng(3)
    chi = rng.standard_normal((3, L * L * Lt))
    ps = (rng.standard_normal((8 * Ls, 2, L * L * Lt)) * np.sqrt(0.5)).astype(np.float32)
    hs = []
    for store in (-1.0, 0.0):
        gl = chb.Lattice(L, Lt, Ls, beta=0.475)
        gl.set_basis_store(store)
        assert lib.chdwf_set_precision(gl.h, 0, 1) == 0
        for which, name, n in ((2, "remez2", 25), (4, "remez4", 25), (22, "remez2g", 12)):
            q = remez[name]
            assert lib.chdwf_traj_set_remez(
                gl.h, which, *(np.ascontiguousarray(q[k]).ctypes.data_as(C.c_void_p)
                               for k in ("anum", "aden", "bnum", "bden")), n) == 0
        assert lib.chdwf_traj_set_chi(gl.h, chi.ctypes.data_as(C.c_void_p)) == 0
        assert lib.chdwf_traj_begin(gl.h) == 0
        it = C.c_int()
        assert lib.chdwf_traj_set_momenta(gl.h, np.zeros((3, L * L * Lt), np.float32)
                                          .ctypes.data_as(C.c_void_p)) == 0
        assert lib.chdwf_traj_heatbath(gl.h, ps.ctypes.data_as(C.c_void_p), 1e-5, 0.0, 0.0, 1,
                                       C.byref(it)) == 0
        out = np.zeros(16)
        assert lib.chdwf_traj_hamilton(gl.h, 1e-5, 0.0, 0.0, 1, out.ctypes.data_as(C.c_void_p),
                                       C.byref(it)) == 0
        gl.close()
        hs.append((out, it.value))
    assert hs[0][1] == hs[1][1]
    assert np.array_equal(hs[0][0], hs[1][0])
