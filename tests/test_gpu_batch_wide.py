"""Batches of many small systems (chdwf_congrad_batch, csrc/plane_cg.cuh): they
advance together however many lattices, mass terms, heights and pinnings are among
them and in whatever order they are listed, so a batch queues about as many kernels
as its longest solve alone; and each system has the bits of the same solve alone,
also where its blocks share blocks of the launch and beyond the systems that one
set of launches holds."""
import ctypes as C

import pytest

import chiralheisenberg_b200 as chb
from conftest import random_fields

pytestmark = pytest.mark.gpu


def _batch(specs, res=1e-6):
    """specs: (L, Lt, Ls, imass, hpin, am3, ibound).  The solutions, the iterations
    and the kernels launched, of the batch and of the solves alone."""
    import torch
    lib = chb.load_library()
    keep, systems = [], []
    for k, (L, Lt, Ls, imass, hpin, am3, ib) in enumerate(specs):
        Phi, chi = (torch.from_numpy(a).cuda()
                    for a in random_fields(L, Lt, Ls, seed=300 + k, chi_scale=0.5))
        x = Phi.clone()
        keep.append((Phi, chi, x))
        systems.append(chb.CgSystem(L, Lt, Ls, imass, hpin, am3, ib, Phi.data_ptr(),
                                    x.data_ptr(), chi.data_ptr()))
    host = chb.Lattice(4, 4, 4)
    n0 = lib.chdwf_kernel_launches()
    its, sts = chb.congrad_batch(host, systems, res)
    nbatch = lib.chdwf_kernel_launches() - n0
    torch.cuda.synchronize()
    host.close()
    nalone = 0
    for k, ((L, Lt, Ls, imass, hpin, am3, ib), (Phi, chi, x)) in enumerate(zip(specs, keep)):
        gl = chb.Lattice(L, Lt, Ls, am3=am3, ibound=ib)
        xr, it = Phi.clone(), C.c_int()
        n0 = lib.chdwf_kernel_launches()
        rc = gl.lib.chdwf_congrad_dev(gl.h, C.c_void_p(Phi.data_ptr()), res, C.byref(it), hpin,
                                      imass, C.c_void_p(chi.data_ptr()), C.c_void_p(xr.data_ptr()))
        torch.cuda.synchronize()
        nalone = max(nalone, lib.chdwf_kernel_launches() - n0)
        gl.close()
        assert rc in (0, 1)
        assert (its[k], sts[k]) == (it.value, rc), k
        assert torch.equal(x, xr), k
    return nbatch, nalone


def test_parameters_do_not_split_a_batch():
    """40 parameter sets on one lattice, as a scan has them.  One set of launches;
    a chunk of iterations may be queued beyond each solve's end."""
    specs = [(6, 4, 4, 1, 0.02 * k, 1.0 - 0.004 * k, -1 if k % 2 else 1) for k in range(40)]
    nbatch, nalone = _batch(specs)
    assert nbatch <= 1.5 * nalone, (nbatch, nalone)


def test_order_does_not_split_a_batch():
    """Eight lattices, four sources each, listed source by source."""
    sizes = [(4, 4, 4), (6, 6, 6), (4, 6, 8), (6, 4, 6), (6, 8, 4), (4, 8, 4), (8, 4, 4), (6, 6, 4)]
    nbatch, nalone = _batch([(*sizes[k % 8], 1, 0.0, 1.0, -1) for k in range(32)])
    assert nbatch <= 1.5 * nalone, (nbatch, nalone)


def test_more_systems_than_one_set_of_launches():
    """Over 256 systems of one mass term, some lattices with tiles of one warp, one
    of six, and both mass terms."""
    sizes = [(2, 2, 2), (3, 5, 3), (12, 12, 2), (4, 4, 4), (5, 4, 7)]
    _batch([(*sizes[k % 5], 3 if k % 41 == 1 else 1, 0.1 * (k % 3 if k % 41 != 1 else 0), 1.0, -1)
            for k in range(270)])
