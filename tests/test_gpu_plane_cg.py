"""Edges of the batched conjugate gradients (csrc/plane_cg.cuh): more systems
than one set of launches holds, more lattices than it holds, both mass terms
interleaved, odd Ls, and the smallest lattices.  A system's blocks and the
order of its sums depend on its lattice alone, so each system of a batch has
the bits of the same solve alone; the per-shift solver's corrections reach
the true residual that is asked for."""
import ctypes as C

import pytest

import chiralheisenberg_b200 as chb
from conftest import random_fields

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2), (3, 5, 3), (5, 4, 7), (6, 3, 5), (9, 7, 2), (4, 4, 4), (7, 6, 3), (13, 2, 3)]


def _alone(L, Lt, Ls, imass, hpin, Phi, chi):
    import torch
    gl = chb.Lattice(L, Lt, Ls)
    x, it = Phi.clone(), C.c_int()
    rc = gl.lib.chdwf_congrad_dev(gl.h, C.c_void_p(Phi.data_ptr()), 1e-7, C.byref(it), hpin,
                                  imass, C.c_void_p(chi.data_ptr()), C.c_void_p(x.data_ptr()))
    torch.cuda.synchronize()
    gl.close()
    assert rc in (0, 1)       # 1: 2^4 may meet congrad's cap of Ls*kvol iterations
    return x, it.value, rc


@pytest.mark.parametrize("nsys", [1, 7, 32, 33, 70])
def test_batch_has_the_bits_of_single_solves(nsys):
    import torch
    keep, systems = [], []
    for k in range(nsys):
        L, Lt, Ls = SIZES[k % len(SIZES)]
        imass = 3 if k % 3 == 1 else 1
        hpin = 0.25 * (k % 2) if imass == 1 else 0.0
        Phi, chi = (torch.from_numpy(a).cuda()
                    for a in random_fields(L, Lt, Ls, seed=900 + k, chi_scale=0.5))
        x = Phi.clone()
        keep.append((L, Lt, Ls, imass, hpin, Phi, chi, x))
        systems.append(chb.CgSystem(L, Lt, Ls, imass, hpin, 1.0, -1, Phi.data_ptr(),
                                    x.data_ptr(), chi.data_ptr()))
    host = chb.Lattice(4, 4, 4)
    its, sts = chb.congrad_batch(host, systems, 1e-7)
    torch.cuda.synchronize()
    host.close()
    for k, (L, Lt, Ls, imass, hpin, Phi, chi, x) in enumerate(keep):
        xr, it, rc = _alone(L, Lt, Ls, imass, hpin, Phi, chi)
        assert (its[k], sts[k]) == (it, rc), k
        assert torch.equal(x, xr), k


@pytest.mark.parametrize("L,Lt,Ls", [(2, 2, 2), (5, 4, 7), (6, 3, 5)])
@pytest.mark.parametrize("imass", [1, 3])
@pytest.mark.parametrize("n", [1, 32])
def test_multishift_corrections_reach_the_residual(L, Lt, Ls, imass, n):
    Phi, chi = random_fields(L, Lt, Ls, seed=77, chi_scale=0.4)
    gl = chb.Lattice(L, Lt, Ls, beta=0.475)
    sigma = [0.003 * 1.2 ** k for k in range(n)]
    out = gl.multishift(Phi, 1e-9, chi, sigma, imass=imass, prec="f32")
    gl.close()
    assert len(out[1]) == n
    assert max(out[1]) <= 1e-9
