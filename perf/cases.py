"""What a user of this framework has it do, as cases that can be timed.

The Dirac operator on device fields in each precision, the multi-shift solves
and forces of a trajectory (FP64 and mixed), the batched propagator solves,
the per-shift solver, and the solvers of the two sister programs (the HMC
predecessor and the bulk Thirring model), each through the public entry
points.  exact() evaluates the same quantities in 64 bits with plain torch.

A case is a dict of plain values:
  kind      operator | solve | force | propagators | multishift | hmc | thirring
  L, Lt, Ls lattice (propagators: the largest of its ensembles)
  imass     mass term, 1 or 3
and per kind the precision, the rational approximation, the residual.
Iteration counts are not returned: they follow from how the solvers group
their sums, the solutions and forces are what is computed.
"""
import ctypes as C
import math

import numpy as np
import torch

import chiralheisenberg_b200 as chb

BETA = 0.475        # the benchmark configuration's coupling
SETS = {            # rational approximations: file, poles, coefficient set
    "heatbath25": ("remez4", 25, "a"),        # (M^dag M)^(1/4), one pseudofermion
    "action25": ("remez2", 25, "b"),          # (M^dag M)^(-1/2)
    "guidance12": ("remez2g", 12, "b"),
    "force12": ("remez2g", 12, "a"),
    "heatbath20": ("remez8_20", 20, "a"),     # (M^dag M)^(1/8), two pseudofermions
    "action20": ("remez4_20", 20, "b"),       # (M^dag M)^(-1/4)
}


def listed():
    return [
        # one application on the smallest lattice that is run: launch latency
        {"name": "operator_f64_8x8", "kind": "operator", "L": 8, "Lt": 8, "Ls": 8, "prec": "f64",
         "dag": False, "imass": 1},
        # the drop-in operator at the production lattice
        {"name": "operator_f64_24x24", "kind": "operator", "L": 24, "Lt": 24, "Ls": 24,
         "prec": "f64", "dag": True, "imass": 1},
        # the operator sweep's largest lattice, complex64
        {"name": "operator_f32_48x32", "kind": "operator", "L": 48, "Lt": 48, "Ls": 32,
         "prec": "f32", "dag": False, "imass": 1},
        # FP16 storage, the other mass term
        {"name": "operator_f16_32x24", "kind": "operator", "L": 32, "Lt": 32, "Ls": 24,
         "prec": "f16", "dag": True, "imass": 3},
        # the reference's force evaluation (guidance and force solve, 12 poles)
        # at the size of its shipped input deck, FP64
        {"name": "force_f64_12x8", "kind": "force", "L": 12, "Lt": 12, "Ls": 8, "prec": "f64",
         "poles": 12, "imass": 1},
        # one force evaluation of the production trajectory: 20 poles, FP32
        # Krylov vectors; a trajectory makes 42 of them
        {"name": "force_mixed_24x24", "kind": "force", "L": 24, "Lt": 24, "Ls": 24,
         "prec": "f32", "poles": 20, "imass": 1},
        # the pseudofermion action of the Metropolis test, FP64
        {"name": "action_f64_20x20", "kind": "solve", "L": 20, "Lt": 20, "Ls": 20,
         "set": "action20", "res": 1e-9, "imass": 1},
        # a pseudofermion heatbath on a ragged lattice with an odd Ls
        {"name": "heatbath_f64_ragged", "kind": "solve", "L": 14, "Lt": 18, "Ls": 11,
         "set": "heatbath25", "res": 1e-9, "imass": 3},
        # propagators of ensembles of uneven size, four sources each, one batch
        {"name": "propagators_uneven", "kind": "propagators", "L": 16, "Lt": 16, "Ls": 24,
         "ensembles": 8, "sources": 4, "res": 1e-8, "imass": 1},
        # every shift's solution to 1e-10, FP32 inner solves with FP64 correction
        {"name": "multishift_f32_16x16", "kind": "multishift", "L": 16, "Lt": 16, "Ls": 16,
         "prec": "f32", "shifts": 20, "res": 1e-10, "imass": 1},
        # the HMC predecessor's force solve
        {"name": "hmc_congrad_16x16", "kind": "hmc", "L": 16, "Lt": 16, "Ls": 16, "res": 1e-6,
         "imass": 1},
        # the Thirring model's force solve (12 poles, link force of every pole)
        {"name": "thirring_force_12x12", "kind": "thirring", "L": 12, "Lt": 12, "Ls": 12,
         "set": "force12", "iflag": 2, "res": 1e-6, "imass": 1},
    ]


def _spread(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _lattice(rng, side, third, most):
    """A lattice of at most `most` points, its sides spread over their logarithm."""
    while True:
        L = _spread(rng, side[0], side[1])
        Lt = L if rng.random() < 0.5 else _spread(rng, side[0], side[1])
        Ls = _spread(rng, third[0], third[1])
        if L * L * Lt * Ls <= most:
            return {"L": L, "Lt": Lt, "Ls": Ls}


def draw(rng):
    kind = rng.choice(["operator", "operator", "solve", "force", "force", "propagators",
                       "multishift", "hmc", "thirring"])
    imass = rng.choice([1, 1, 3])
    if kind == "operator":
        return {"kind": kind, **_lattice(rng, (6, 48), (5, 32), 48 ** 3 * 32),
                "prec": rng.choice(["f64", "f32", "f16"]), "dag": rng.random() < 0.5,
                "imass": imass}
    if kind == "solve":
        return {"kind": kind, **_lattice(rng, (6, 20), (6, 20), 20 ** 3 * 20),
                "set": rng.choice(["heatbath25", "action25", "heatbath20", "action20"]),
                "res": 1e-9, "imass": imass}
    if kind == "force":
        return {"kind": kind, **_lattice(rng, (8, 24), (6, 24), 24 ** 3 * 24),
                "prec": rng.choice(["f64", "f32"]), "poles": rng.choice([12, 20]),
                "imass": imass}
    if kind == "propagators":
        return {"kind": kind, **_lattice(rng, (8, 16), (8, 24), 16 ** 3 * 24),
                "ensembles": rng.randint(1, 8), "sources": rng.randint(1, 4), "res": 1e-8,
                "imass": imass}
    if kind == "multishift":
        return {"kind": kind, **_lattice(rng, (6, 16), (6, 16), 16 ** 3 * 16),
                "prec": rng.choice(["f64", "f32"]), "shifts": rng.randint(4, 20), "res": 1e-10,
                "imass": imass}
    if kind == "hmc":
        return {"kind": kind, **_lattice(rng, (6, 24), (6, 24), 20 ** 3 * 20), "res": 1e-6,
                "imass": imass}
    name, iflag = rng.choice([("force12", 2), ("action25", 0)])
    return {"kind": kind, **_lattice(rng, (6, 16), (6, 16), 14 ** 3 * 14), "set": name,
            "iflag": iflag, "res": 1e-6, "imass": rng.choice([1, 3])}


# ---- inputs ------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _spinor_shape(c):
    return (2, 4, c["Lt"], c["L"], c["L"], c["Ls"])


def _gauss(g, shape, dtype=torch.complex128):
    return torch.randn(shape, dtype=dtype, device="cuda", generator=g)


def _chi(g, c):
    """chi(kvol, 3) with the width that thermalised configurations have, 1/sqrt(2 beta)."""
    return torch.randn((3, c["L"] ** 2 * c["Lt"]), dtype=torch.float64, device="cuda",
                       generator=g) / math.sqrt(2 * BETA)


def _set(name):
    fn, n, ab = SETS[name]
    r = chb.read_remez(fn, n)
    return (r["anum"], r["aden"]) if ab == "a" else (r["bnum"], r["bden"])


def _p(t):
    return C.c_void_p(t.data_ptr())


def _np(a):
    return a.ctypes.data_as(C.c_void_p)


def _ensembles(c, seed):
    """Lattice sizes of a batch: the case's own first, the others up to it (the
    same for every seed, so that a case is one batch layout)."""
    import random
    r = random.Random(c["L"] * 1000 + c["Ls"] * 10 + c["ensembles"])
    out = [(c["L"], c["Lt"], c["Ls"])]
    for _ in range(c["ensembles"] - 1):
        L = min(c["L"], r.choice([8, 12, 16]))
        out.append((L, L, min(c["Ls"], r.choice([8, 16, 24]))))
    return out


def _sources(c, seed):
    """Per ensemble: chi, and Phi = M^dag xi of its point sources on s = 1."""
    g = _gen(seed)
    out = []
    for L, Lt, Ls in _ensembles(c, seed):
        e = {"L": L, "Lt": Lt, "Ls": Ls}
        chi = _chi(g, e)
        kvol = L * L * Lt
        at = torch.randint(kvol, (1,), device="cuda", generator=g)
        xi = torch.zeros((c["sources"], 2, 4, kvol, Ls), dtype=torch.complex128, device="cuda")
        for k in range(c["sources"]):
            xi[k, k // 2, 2 + k % 2, at, 0] = 1.0
        xi = xi.view((c["sources"],) + _spinor_shape(e))
        out.append((e, chi, _apply(xi, e, chi, c["imass"], True)))
    return out


def _hmc_inputs(c, seed):
    g = _gen(seed)
    chi = _chi(g, c).float()
    Phi = _apply(_gauss(g, _spinor_shape(c)), c, chi.double(), c["imass"], True)
    return chi, Phi.to(torch.complex64)


def _thirring_inputs(c, seed):
    g = _gen(seed)
    kvol = c["L"] ** 2 * c["Lt"]
    theta = 0.3 * torch.randn((3, kvol), dtype=torch.float32, device="cuda", generator=g)
    Phi = _gauss(g, (4, c["Lt"], c["L"], c["L"], c["Ls"]))
    return theta, Phi


THIRRING_AM = 0.05


def _links(theta, c):
    u = torch.complex(torch.ones_like(theta, dtype=torch.float64), theta.double())
    u = u.view(3, c["Lt"], -1)
    u[2, c["Lt"] - 1] *= -1                      # antiperiodic in t
    return u.reshape(3, -1)


SIGMA = lambda n: 10.0 ** np.linspace(-5, 1, n)   # noqa: E731


# ---- the states and the passes -------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "operator":
        g = _gen(seed)
        lat = chb.Lattice(c["L"], c["Lt"], c["Ls"], beta=BETA)
        R = _gauss(g, _spinor_shape(c), torch.complex128 if c["prec"] == "f64" else torch.complex64)
        if c["prec"] == "f16":
            R = torch.view_as_real(R).half().contiguous()
        s.update(lat=lat, R=R, chi=_chi(g, c), out=torch.empty_like(R))
    elif kind == "solve":
        g = _gen(seed)
        lat = chb.Lattice(c["L"], c["Lt"], c["Ls"], beta=BETA)
        lat.set_basis_store(40e9)
        num, den = _set(c["set"])
        Phi = _gauss(g, _spinor_shape(c)) * math.sqrt(0.5)
        s.update(lat=lat, Phi=Phi, chi=_chi(g, c), x=torch.empty_like(Phi), num=num, den=den)
    elif kind == "force":
        s["lat"] = _resident(c, seed)
        s["dS"] = np.empty((3, c["L"] ** 2 * c["Lt"]), dtype=np.float32)
    elif kind == "propagators":
        systems, keep = [], []
        for e, chi, Phi in _sources(c, seed):
            x = torch.empty_like(Phi)
            keep.append((chi, Phi, x))
            for k in range(c["sources"]):
                systems.append(chb.CgSystem(e["L"], e["Lt"], e["Ls"], c["imass"], 0.0, 1.0, -1,
                                            Phi[k].data_ptr(), x[k].data_ptr(), chi.data_ptr()))
        s.update(lat=chb.Lattice(c["L"], c["Lt"], c["Ls"], beta=BETA), systems=systems, keep=keep)
    elif kind == "multishift":
        g = _gen(seed)
        lat = chb.Lattice(c["L"], c["Lt"], c["Ls"], beta=BETA)
        lat.set_basis_store(40e9)
        Phi = _gauss(g, _spinor_shape(c))
        s.update(lat=lat, Phi=Phi, chi=_chi(g, c),
                 x=torch.empty((c["shifts"],) + Phi.shape, dtype=Phi.dtype, device="cuda"))
    elif kind == "hmc":
        chi, Phi = _hmc_inputs(c, seed)
        h = chb.Hmc(c["L"], c["Lt"], c["Ls"], 0.1, BETA, 1.0, 0.0, c["imass"], 10)
        Phi = Phi.cpu().numpy()
        s.update(h=h, Phi=Phi, chi=chi.cpu().numpy(), x0=np.zeros_like(Phi))
    else:
        theta, Phi = _thirring_inputs(c, seed)
        num, den = _set(c["set"])
        h = chb.Thirring(c["L"], c["Lt"], c["Ls"], 0.1, 0.5, 1.0, THIRRING_AM, c["imass"], 10)
        s.update(h=h, Phi=Phi.cpu().numpy(), u=h.coef(theta.cpu().numpy()), num=num, den=den,
                 P0=np.zeros((len(den),) + tuple(Phi.shape), dtype=np.complex128))
    torch.cuda.synchronize()
    return s


def _force_inputs(c, seed):
    """chi and the heatbath's Gaussians (variance 1/2) of one pseudofermion field,
    in the order in which the trajectory's driver draws them."""
    g = _gen(seed)
    chi = _chi(g, c)
    kvol = c["L"] ** 2 * c["Lt"]
    ps = torch.randn((8 * c["Ls"], 2, kvol), device="cuda", generator=g) * math.sqrt(0.5)
    return chi, ps


def _resident(c, seed):
    """A lattice with chi and a pseudofermion field resident, as a trajectory has
    them when it asks for a force."""
    chi, ps = _force_inputs(c, seed)
    torch.cuda.synchronize()
    lat = chb.Lattice(c["L"], c["Lt"], c["Ls"], beta=BETA)
    lib, h, it = lat.lib, lat.h, C.c_int()
    lat.set_basis_store(30e9)
    lat._check(lib.chdwf_set_precision(h, 1 if c["prec"] == "f32" else 0, 0))
    lat._check(lib.chdwf_traj_set_chi(h, _np(chi.cpu().numpy())))
    lat._check(lib.chdwf_traj_begin(h))
    if c["poles"] == 12:        # the reference's algorithm
        for which, name, n in ((4, "remez4", 25), (22, "remez2g", 12)):
            r = chb.read_remez(name, n)
            lat._check(lib.chdwf_traj_set_remez(h, which, _np(r["anum"]), _np(r["aden"]),
                                                _np(r["bnum"]), _np(r["bden"]), n))
        lat._check(lib.chdwf_traj_heatbath_dev(h, _p(ps), 1e-9, 0.0, 0.0, c["imass"],
                                               C.byref(it)))
    else:                       # two pseudofermion fields, one force solve each
        for which, name in ((0, "heatbath20"), (1, "action20")):
            num, den = _set(name)
            lat._check(lib.chdwf_ext_set_remez(h, which, _np(num), _np(den), len(den)))
        lat._check(lib.chdwf_ext_heatbath_dev(h, _p(ps), 1e-9, 0.0, c["imass"], C.byref(it)))
    lat._check(lib.chdwf_traj_sync(h))
    return lat


def run(state):
    s, c = state, state["case"]
    kind, it, it2 = c["kind"], C.c_int(), C.c_int()
    if kind == "operator":
        lat = s["lat"]
        if c["prec"] == "f64":
            lat._check(lat.lib.chdwf_dslash_dev(lat.h, _p(s["out"]), _p(s["R"]), _p(s["chi"]), 0.0,
                                                c["imass"], int(c["dag"]), None))
        else:
            lat._check(lat.lib.chdwf_dslash_dev_lp(lat.h, _p(s["out"]), _p(s["R"]), _p(s["chi"]),
                                                   0.0, c["imass"], int(c["dag"]),
                                                   1 if c["prec"] == "f32" else 2, None))
        return s["out"]
    if kind == "solve":
        lat = s["lat"]
        lat._check(lat.lib.chdwf_qmrherm_dev(lat.h, _p(s["Phi"]), c["res"], C.byref(it), 0.0,
                                             c["imass"], _np(s["num"]), _np(s["den"]),
                                             len(s["den"]), 0, _p(s["chi"]), _p(s["x"]), None))
        return s["x"]
    if kind == "force":
        lat = s["lat"]
        if c["poles"] == 12:
            lat._check(lat.lib.chdwf_traj_force(lat.h, 1e-6, 0.0, 0.0, c["imass"], C.byref(it),
                                                C.byref(it2)))
        else:
            lat._check(lat.lib.chdwf_ext_force(lat.h, 1e-6, 0.0, c["imass"], 1, C.byref(it)))
        lat._check(lat.lib.chdwf_traj_get_force(lat.h, _np(s["dS"])))
        return s["dS"]
    if kind == "propagators":
        for _, Phi, x in s["keep"]:
            x.copy_(Phi)                          # x0 = Phi
        torch.cuda.current_stream().synchronize()   # the library works on a stream of its own
        _, status = chb.congrad_batch(s["lat"], s["systems"], c["res"])
        if status.any():
            raise RuntimeError("a propagator did not converge")
        return [x for _, _, x in s["keep"]]
    if kind == "multishift":
        lat, n = s["lat"], c["shifts"]
        sigma, tr = SIGMA(n), np.zeros(n)
        ptrs = (C.c_void_p * n)(*[s["x"][k].data_ptr() for k in range(n)])
        lat._check(lat.lib.chdwf_multishift_dev(lat.h, _p(s["Phi"]), c["res"], _p(s["chi"]), 0.0,
                                                c["imass"], n, _np(sigma), ptrs, _np(tr),
                                                1 if c["prec"] == "f32" else 0, C.byref(it),
                                                C.byref(it2)))
        return s["x"]
    if kind == "hmc":
        x, _, capped = s["h"].congrad(s["Phi"], s["chi"], s["x0"], c["res"])
        if capped:
            raise RuntimeError("congrad did not converge")
        return x
    dS = np.zeros((3, c["L"] ** 2 * c["Lt"]), dtype=np.float32)
    x, _, capped, _, dS = s["h"].qmrherm(s["Phi"], s["u"], c["res"], THIRRING_AM, c["imass"],
                                         s["num"], s["den"], iflag=c["iflag"], Phi0=s["P0"],
                                         dSdpi=dS)
    if capped:
        raise RuntimeError("qmrherm did not converge")
    return [x, dS] if c["iflag"] == 2 else [x]


# ---- work ------------------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass.  A Lanczos iteration applies M and
    M^dagger (each reads its input and writes its output) and reads the two
    previous vectors; a CG iteration also updates x, r and p.  Iterations as
    they are needed at these residuals and field strengths."""
    c, kind = case, case["kind"]
    n = 8 * c["L"] ** 2 * c["Lt"] * c["Ls"]        # complex numbers of a spinor
    size = {"f64": 16, "f32": 8, "f16": 4}.get(c.get("prec"), 16)
    op = 46                                        # operations per complex number and application
    if kind == "operator":
        return {"bytes": 2 * n * size + 24 * c["L"] ** 2 * c["Lt"], "flops": op * n}
    its = _iterations(c)
    if kind == "solve":
        return {"bytes": n * size * (6 * its + its + 2), "flops": n * its * (2 * op + 16)}
    if kind == "force":
        solves = 2 if c["poles"] == 12 else 1
        return {"bytes": solves * n * size * (6 * its + 2), "flops": solves * n * its * (2 * op + 12)}
    if kind == "propagators":
        n = sum(8 * L * L * Lt * Ls for L, Lt, Ls in _ensembles(c, 0)) * c["sources"]
        return {"bytes": n * 16 * its * 9, "flops": n * its * (2 * op + 20)}
    if kind == "multishift":
        b = n * size * 7 * its + c["shifts"] * n * 16
        if c["prec"] == "f32":                     # corrected once per shift at least
            b += c["shifts"] * n * (5 * 16 + 8 * 9)
        return {"bytes": b, "flops": n * its * (2 * op + 12 + 4 * c["shifts"])}
    if kind == "hmc":
        return {"bytes": n * 8 * its * 9, "flops": n * its * (2 * op + 20)}
    n //= 2                                        # one flavour
    return {"bytes": n * 16 * 7 * its, "flops": n * its * (2 * 80 + 16)}


def _iterations(c):
    """Iterations to the case's residual: proportional to the lattice's side
    (counted at 6 to 24 sites a side, to 15%; Ls hardly matters)."""
    per_site = {"solve": 54, "force": 40, "multishift": 46, "propagators": 25, "hmc": 28,
                "thirring": 14}[c["kind"]]
    return int(per_site * (c["L"] ** 2 * c["Lt"]) ** (1 / 3))


# ---- the same in 64 bits with plain torch -----------------------------------------
def _hop(acc, R, dim, mu, fwd, sig, wrap):
    """acc += one hop of the Wilson-Dirac operator (times two): R[..., d, t, y, x, s]
    from its forward (fwd) or backward neighbour in direction mu."""
    pa, pb = ((3, 2), (3, 2), (2, 3))[mu]
    i = 1j if mu != 1 else 1.0
    sb = sig if mu == 0 else -sig
    a = torch.add(R[0], R[pa], alpha=i * sig)
    b = torch.add(R[1], R[pb], alpha=i * sb)
    shift = -1 if fwd else 1
    a, b = a.roll(shift, dim), b.roll(shift, dim)
    if wrap:
        for v in (a, b):
            v.select(dim, -1 if fwd else 0).neg_()
    acc[0] -= a
    acc[1] -= b
    s3, s4 = sig, sig if mu == 0 else -sig
    acc[2].add_(a if mu == 2 else b, alpha=i * s3)
    acc[3].add_(b if mu == 2 else a, alpha=i * s4)


def _apply(R, c, chi, imass, dag):
    """M R or M^dagger R; R is [..., 2, 4, Lt, L, L, Ls], am3 = 1, antiperiodic in t."""
    Ls = c["Ls"]
    Rd = [R.select(-5, d) for d in range(4)]       # [..., 2, t, y, x, s]
    acc = [6.0 * v for v in Rd]
    sf = -1 if dag else 1
    for mu, dim in ((0, -2), (1, -3), (2, -4)):
        for fwd in (True, False):
            _hop(acc, Rd, dim, mu, fwd, sf if fwd else -sf, mu == 2)
    for v in acc:
        v *= 0.5
    up, dn = ((0, 1), (2, 3)) if dag else ((2, 3), (0, 1))
    for d in up:
        acc[d][..., :-1] -= Rd[d][..., 1:]
    for d in dn:
        acc[d][..., 1:] -= Rd[d][..., :-1]
    c1, c2, c3 = chi.float().double().view(3, c["Lt"], c["L"], c["L"])
    for pair, s, other in ((up, Ls - 1, 0), (dn, 0, Ls - 1)):
        for d in pair:
            o0, o1 = Rd[d][..., 0, :, :, :, other], Rd[d][..., 1, :, :, :, other]
            a0, a1 = acc[d][..., 0, :, :, :, s], acc[d][..., 1, :, :, :, s]
            if imass == 1:
                a0 += c3 * o0 + torch.complex(c1, -c2) * o1
                a1 += -c3 * o1 + torch.complex(c1, c2) * o0
            else:
                sg = -1.0 if (s == Ls - 1) != dag else 1.0
                z3 = torch.complex(torch.zeros_like(c3), -c3 if dag else c3)
                z = torch.complex(-c2, -c1) if dag else torch.complex(c2, c1)
                a0 += sg * (z3 * o0 + z * o1)
                a1 += -sg * (z3 * o1 + z.conj() * o0)
    return torch.stack(acc, -5)


def _apply_thirring(R, c, u, am, imass, dag):
    """The Thirring operator on R[4, t, y, x, s] with links u[3, kvol]."""
    Ls, shape = c["Ls"], (3, c["Lt"], c["L"], c["L"], 1)
    U = u.view(shape)
    acc = 3.0 * R
    for mu, dim in ((0, -2), (1, -3), (2, -4)):
        f = U[mu] * R.roll(-1, dim)
        b = (U[mu].conj() * R).roll(1, dim)
        acc = acc - 0.5 * (f + b)
        w = _gamma(mu, f - b)
        acc = acc - w if dag else acc + w
    up, dn = (slice(0, 2), slice(2, 4)) if dag else (slice(2, 4), slice(0, 2))
    acc[up, ..., :-1] -= R[up, ..., 1:]
    acc[dn, ..., 1:] -= R[dn, ..., :-1]
    zk = am if imass == 1 else 1j * (am if dag else -am)
    sa = 1 if imass == 1 else (-1 if not dag else 1)
    sb = 1 if imass == 1 else -sa
    acc[up, ..., Ls - 1] += sa * zk * R[up, ..., 0]
    acc[dn, ..., 0] += sb * zk * R[dn, ..., Ls - 1]
    return acc


_GI = ((3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1))
_GV = ((-0.5j, -0.5j, 0.5j, 0.5j), (-0.5, 0.5, 0.5, -0.5), (-0.5j, 0.5j, 0.5j, -0.5j))


def _gamma(mu, v):
    return torch.stack([_GV[mu][d] * v[_GI[mu][d]] for d in range(4)])


def _shifted_cg(A, b, sigma, tol, weights=None, most=20000):
    """x_k = (A + sigma_k)^-1 b for every k by shifted CG on the smallest shift
    (or, with weights, sum_k weights_k x_k only).  b is [n]."""
    sigma = torch.as_tensor(np.asarray(sigma), dtype=torch.float64, device=b.device)
    base = sigma.min()
    rel = sigma - base
    K = len(sigma)
    P = b.repeat(K, 1)
    X = torch.zeros_like(b) if weights is not None else torch.zeros_like(P)
    if weights is not None:
        weights = torch.as_tensor(np.asarray(weights), dtype=torch.float64, device=b.device)
    r, p = b.clone(), b.clone()
    rr = torch.vdot(r, r).real
    stop = tol * tol * float(rr)
    one = torch.ones(K, dtype=torch.float64, device=b.device)
    z, zm, am, bm = one.clone(), one.clone(), one[0].clone(), torch.zeros_like(one[0])
    for it in range(most):
        q = A(p) + base * p
        alpha = rr / torch.vdot(p, q).real
        zn = z * zm * am / (alpha * bm * (zm - z) + zm * am * (1.0 + rel * alpha))
        zn = torch.where(torch.isfinite(zn), zn, torch.zeros_like(zn))
        ak = torch.where(z != 0, alpha * zn / z, torch.zeros_like(z))
        if weights is None:
            X.addcmul_(ak.to(X.dtype)[:, None], P)
        else:
            X += (weights * ak).to(X.dtype) @ P
        r = r - alpha * q
        rn = torch.vdot(r, r).real
        beta = rn / rr
        bk = torch.where(z != 0, beta * (zn / z) ** 2, torch.zeros_like(z))
        P.mul_(bk.to(P.dtype)[:, None]).addr_(zn.to(P.dtype), r)
        p = r + beta * p
        z, zm, am, bm, rr = zn, z, alpha, beta, rn
        if it % 50 == 49 and float(rr) <= stop:
            break
    return X


def _cg(c, chi, imass, b, tol=1e-12, most=20000):
    """(M^dag M)^-1 b by CG for a stack of right-hand sides."""
    dot = lambda v, w: (v.conj() * w).real.sum((1, 2, 3, 4, 5, 6), keepdim=True)   # noqa: E731
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    rr = dot(r, r)
    stop = tol * tol * rr
    for it in range(most):
        q = _apply(_apply(p, c, chi, imass, False), c, chi, imass, True)
        alpha = rr / dot(p, q)
        x += alpha * p
        r -= alpha * q
        rn = dot(r, r)
        p = r + (rn / rr) * p
        rr = rn
        if it % 50 == 49 and bool((rr <= stop).all()):
            break
    return x


def _rational(A, b, num, den, tol=1e-13):
    x = _shifted_cg(A, b.reshape(-1), den, tol, weights=num[1:])
    return (num[0] * b.reshape(-1) + x).view(b.shape)


def _normal(c, chi, imass):
    sh = _spinor_shape(c)
    return lambda v: _apply(_apply(v.view(sh), c, chi, imass, False), c, chi, imass,
                            True).reshape(-1)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "operator":
        g = _gen(seed)
        R = _gauss(g, _spinor_shape(c), torch.complex128 if c["prec"] == "f64" else torch.complex64)
        if c["prec"] == "f16":
            R = torch.view_as_complex(torch.view_as_real(R).half().float())
        out = _apply(R.to(torch.complex128), c, _chi(g, c), c["imass"], c["dag"])
        return torch.view_as_real(out) if c["prec"] == "f16" else out
    if kind == "solve":
        g = _gen(seed)
        Phi = _gauss(g, _spinor_shape(c)) * math.sqrt(0.5)
        num, den = _set(c["set"])
        return _rational(_normal(c, _chi(g, c), c["imass"]), Phi, num, den)
    if kind == "force":
        chi, ps = _force_inputs(c, seed)
        R = torch.complex(ps[:, 0].double(), ps[:, 1].double())        # [call, site]
        R = R.view(2, 4, c["Ls"], c["Lt"], c["L"], c["L"]).permute(0, 1, 3, 4, 5, 2).contiguous()
        A = _normal(c, chi, c["imass"])
        if c["poles"] == 12:
            Phi = _rational(A, R, *_set("heatbath25"))
            Phi = _rational(A, Phi, *_set("guidance12"))
            num, den = _set("force12")
            sign = 1.0
        else:
            Phi = _rational(A, R, *_set("heatbath20"))
            num, den = _set("action20")
            sign = -1.0
        X = _shifted_cg(A, Phi.reshape(-1), den, 1e-12)
        dS = 2 * float(np.float32(BETA)) * chi
        for k in range(len(den)):
            x = X[k].view(_spinor_shape(c))
            y = _apply(x, c, chi, c["imass"], False)
            dS += _force_of(x, y, sign * num[k + 1], c["imass"])
        return dS
    if kind == "propagators":
        out = []
        for e, chi, Phi in _sources(c, seed):
            out.append(_cg(e, chi, c["imass"], Phi))
        return out
    if kind == "multishift":
        g = _gen(seed)
        Phi = _gauss(g, _spinor_shape(c))
        X = _shifted_cg(_normal(c, _chi(g, c), c["imass"]), Phi.reshape(-1), SIGMA(c["shifts"]),
                        1e-14)
        return X.view((c["shifts"],) + Phi.shape)
    if kind == "hmc":
        chi, Phi = _hmc_inputs(c, seed)
        x = _shifted_cg(_normal(c, chi.double(), c["imass"]),
                        Phi.to(torch.complex128).reshape(-1), [0.0], 1e-12)
        return x[0].view(Phi.shape)
    theta, Phi = _thirring_inputs(c, seed)
    u = _links(theta, c)
    num, den = _set(c["set"])

    def A(v):
        v = _apply_thirring(v.view(Phi.shape), c, u, THIRRING_AM, c["imass"], False)
        return _apply_thirring(v, c, u, THIRRING_AM, c["imass"], True).reshape(-1)
    if c["iflag"] == 0:
        return [_rational(A, Phi, num, den)]
    X = _shifted_cg(A, Phi.reshape(-1), den, 1e-13)
    dS = torch.zeros((3, c["L"] ** 2 * c["Lt"]), dtype=torch.float64, device="cuda")
    for k in range(len(den)):
        x = X[k].view(Phi.shape)
        y = _apply_thirring(x, c, u, THIRRING_AM, c["imass"], False)
        tz = 2j * num[k + 1]
        for mu, dim in ((0, -2), (1, -3), (2, -4)):
            xu, yu = x.roll(-1, dim), y.roll(-1, dim)
            f = -0.5 * (tz * (x.conj() * yu - xu.conj() * y)).real.sum((0, -1))
            gy, gyu = (torch.stack([_GV[mu][d] * v[_GI[mu][d]] for d in range(4)]) for v in (y, yu))
            f -= (tz * (x.conj() * gyu + xu.conj() * gy)).real.sum((0, -1))
            dS[mu] += f.reshape(-1)
    return [num[0] * Phi, dS]


def _force_of(x, y, a, imass):
    """One pole's term of dS/dchi: x_k and M x_k on the walls, weight a."""
    dS = 0.0
    for d in range(4):
        sr, sy = (-1, 0) if d < 2 else (0, -1)
        r1, r2 = x[0, d, ..., sr].conj(), x[1, d, ..., sr].conj()
        y1, y2 = y[0, d, ..., sy], y[1, d, ..., sy]
        c1, c2, c3 = r1 * y2 + r2 * y1, r1 * y2 - r2 * y1, r1 * y1 - r2 * y2
        if imass == 1:
            t = torch.stack([c1.real, c2.imag, c3.real])
        else:
            t = torch.stack([c1.imag, -c2.real, c3.imag]) * (1.0 if d < 2 else -1.0)
        dS = dS + 2.0 * a * t
    return dS.reshape(3, -1)
