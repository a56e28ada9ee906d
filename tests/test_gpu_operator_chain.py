"""Operator calls one behind the other on a stream (csrc/dslash.cu): M^dagger is
scheduled while M still writes the vector that it reads, and M of the next pair
while M^dagger still reads it.  Pairs queued without a synchronisation between
the calls have the bits of the same calls with the GPU waited for after each."""
import ctypes as C

import pytest

import chiralheisenberg_b200 as chb
from conftest import random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (5, 3, 7), (8, 8, 8), (12, 10, 6)])
@pytest.mark.parametrize("prec", ["f64", "f32", "f16"])
def test_queued_calls_equal_synchronised_ones(L, Lt, Ls, prec):
    import torch
    R, chi_h = random_fields(L, Lt, Ls, seed=5, chi_scale=0.5)
    chi = torch.from_numpy(chi_h).cuda()
    z = torch.from_numpy(R).cuda()
    if prec == "f64":
        base = z
    elif prec == "f32":
        base = z.to(torch.complex64)
    else:
        base = torch.view_as_real(z).to(torch.float16).contiguous()
    n = 24
    src = [base * (0.01 + 0.002 * k) for k in range(n)]
    gl = chb.Lattice(L, Lt, Ls)

    def apply(out, x, dag):
        args = [gl.h, C.c_void_p(out.data_ptr()), C.c_void_p(x.data_ptr()),
                C.c_void_p(chi.data_ptr()), 0.0, 1, int(dag)]
        if prec == "f64":
            rc = gl.lib.chdwf_dslash_dev(*args, None)
        else:
            rc = gl.lib.chdwf_dslash_dev_lp(*args, 1 if prec == "f32" else 2, None)
        assert rc == 0

    t = torch.empty_like(base)             # one vector between, as a solver has it
    out = [torch.empty_like(base) for _ in src]
    ref = [torch.empty_like(base) for _ in src]
    torch.cuda.synchronize()
    for s, r in zip(src, ref):
        apply(t, s, False)
        torch.cuda.synchronize()
        apply(r, t, True)
        torch.cuda.synchronize()
    for _ in range(5):
        for o in out:
            o.zero_()
        torch.cuda.synchronize()
        for s, o in zip(src, out):
            apply(t, s, False)
            apply(o, t, True)
        torch.cuda.synchronize()
        for o, r in zip(out, ref):
            assert torch.equal(o, r)
    gl.close()
