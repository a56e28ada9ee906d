"""What congrad leaves behind when a call ends with an error (csrc/plane_cg.cuh).
The solver keeps x site-fastest in the caller's buffer while it runs; after an
error of the CUDA runtime, here one that an earlier call of the program left
standing, x is back in the ABI's layout, as it is after a success."""
import ctypes as C

import pytest

import chiralheisenberg_b200 as chb
from conftest import random_fields

pytestmark = pytest.mark.gpu


def _stale_error():
    rt = C.CDLL("libcudart.so.12")
    assert rt.cudaSetDevice(4096) != 0          # refused by the runtime; its code stays
    assert rt.cudaPeekAtLastError() != 0


def _clear():
    C.CDLL("libcudart.so.12").cudaGetLastError()


@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (5, 3, 7)])
@pytest.mark.parametrize("batch", [False, True])
def test_x_is_in_its_layout_after_an_error(L, Lt, Ls, batch):
    import torch
    Phi, chi = (torch.from_numpy(a).cuda()
                for a in random_fields(L, Lt, Ls, seed=9, chi_scale=0.4))
    gl = chb.Lattice(L, Lt, Ls)

    def solve():
        x, it = Phi.clone(), C.c_int()
        torch.cuda.synchronize()
        if batch:
            q = (chb.CgSystem * 1)(chb.CgSystem(L, Lt, Ls, 1, 0.0, 1.0, -1, Phi.data_ptr(),
                                                x.data_ptr(), chi.data_ptr()))
            st = C.c_int()
            run = lambda: gl.lib.chdwf_congrad_batch(gl.h, q, 1, 1e-7, C.byref(it), C.byref(st))
        else:
            run = lambda: gl.lib.chdwf_congrad_dev(gl.h, C.c_void_p(Phi.data_ptr()), 1e-7,
                                                   C.byref(it), 0.0, 1,
                                                   C.c_void_p(chi.data_ptr()),
                                                   C.c_void_p(x.data_ptr()))
        return x, run

    x, run = solve()
    assert run() == 0
    y, run = solve()
    _stale_error()
    rc = run()
    _clear()
    torch.cuda.synchronize()
    assert rc == chb.CHDWF_CUDA_ERROR
    assert torch.equal(y, x)
    z, run = solve()
    assert run() == 0
    torch.cuda.synchronize()
    assert torch.equal(z, x)
    gl.close()
