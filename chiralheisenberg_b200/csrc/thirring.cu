// thirring.cu -- the bulk Thirring RHMC, bulk_rhmc.f, on the GPU: its link
// operator, multi-shift solver with the Phi0 register, link force, force and
// Hamiltonian with the Pauli-Villars terms, and main loop
// (include/chdwf_thirring.h).
//
// The operator is a chain of sweeps in the reference (diagonal, Wilson and
// Dirac hops through the links, s hops, wall mass term).  One thread per
// spinor element replays the chain for its element in FP64 with
// round-to-nearest intrinsics, so the result equals the sequential
// evaluation bit for bit.  derivs gives one thread to each link (site, mu)
// and adds its 8*kthird terms in the reference's order into a REAL*4
// register, also bit for bit.  The multi-shift solver and congrad run
// their scalar recurrences on the device with the reference's implicit
// REAL*4 / REAL*8 types; the sums are FP64 block partials added in one order,
// and the host polls a stop flag once a chunk of iterations instead of reading
// every scalar.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "chdwf_thirring.h"
#include "chunk_graph.h"
#include "common.cuh"
#include "internal.h"
#include "planes.cuh"
#include "rng.h"
#include "row_stage.cuh"

namespace chdwf {
namespace {

constexpr int kThrMaxPoles = 25;
constexpr int kRedBlocks = 592;           // 4 per SM, fixed: partials summed in block order

struct TGeom {
    int L, Lt, Ls, kvol;
    int64_t kferm;                        // 4*kvol*Ls
};

// gamval(mu,idirac)*akappa, gamin(mu,idirac) - 1 (bulk_rhmc.f:1646-1722)
__constant__ double2 c_tgv[3][4] = {{{0., -0.5}, {0., -0.5}, {0., 0.5}, {0., 0.5}},
                                    {{-0.5, 0.}, {0.5, 0.}, {0.5, 0.}, {-0.5, 0.}},
                                    {{0., -0.5}, {0., 0.5}, {0., 0.5}, {0., -0.5}}};
__constant__ int c_tgi[3][4] = {{3, 2, 1, 0}, {3, 2, 1, 0}, {2, 3, 0, 1}};

__device__ __forceinline__ int64_t tsite(int L, int x, int y, int t) {
    return x + (int64_t)L * (y + (int64_t)L * t);
}

// the periodic neighbours up/down of site (x, y, t) in direction mu (addrc, :1746-1797)
__device__ __forceinline__ void tnbr(const TGeom& g, int x, int y, int t, int mu, int64_t* up,
                                     int64_t* dn) {
    if (mu == 0) {
        *up = tsite(g.L, x + 1 == g.L ? 0 : x + 1, y, t);
        *dn = tsite(g.L, x == 0 ? g.L - 1 : x - 1, y, t);
    } else if (mu == 1) {
        *up = tsite(g.L, x, y + 1 == g.L ? 0 : y + 1, t);
        *dn = tsite(g.L, x, y == 0 ? g.L - 1 : y - 1, t);
    } else {
        *up = tsite(g.L, x, y, t + 1 == g.Lt ? 0 : t + 1);
        *dn = tsite(g.L, x, y, t == 0 ? g.Lt - 1 : t - 1);
    }
}

// Site coordinates (site < kvol < 2^31): 32-bit divisions.
__device__ __forceinline__ void tsite_xyt(int L, int64_t site, int* x, int* y, int* t) {
    const uint32_t uL = (uint32_t)L, st = (uint32_t)site, xy = st / uL;
    *x = (int)(st - xy * uL);
    const uint32_t tt = xy / uL;
    *y = (int)(xy - tt * uL);
    *t = (int)tt;
}

// One element (s, site, d) of Phi = M R (DAG false, :1946-2069) or
// Phi = M^dagger R (DAG true, :2071-2188).
template <bool DAG, int IMASS>
__device__ double2 thr_element(const double2* __restrict__ R, const double2* __restrict__ u,
                               const TGeom& g, int s, int64_t i, int d, double diag, double2 zk) {
    const int L = g.L, Ls = g.Ls;
    const int64_t kvol = g.kvol;
    auto at = [&](int ss, int64_t st, int dd) -> double2 {
        return __ldg(R + ss + (int64_t)Ls * (st + kvol * dd));
    };
    int x, y, t;
    tsite_xyt(L, i, &x, &y, &t);
    int64_t up[3], dn[3];
#pragma unroll
    for (int mu = 0; mu < 3; mu++) tnbr(g, x, y, t, mu, &up[mu], &dn[mu]);
    double2 phi = zscal(diag, at(s, i, d));                                 // :1967-1974
#pragma unroll
    for (int mu = 0; mu < 3; mu++) {                                         // Wilson, :1976-1987
        const double2 uu = __ldg(u + i + kvol * mu), ud = zconj(__ldg(u + dn[mu] + kvol * mu));
        const double2 w = zadd(zmul(uu, at(s, up[mu], d)), zmul(ud, at(s, dn[mu], d)));
        phi = zsub(phi, zscal(0.5, w));
    }
#pragma unroll
    for (int mu = 0; mu < 3; mu++) {                                         // Dirac, :1989-2002
        const int dg = c_tgi[mu][d];
        const double2 uu = __ldg(u + i + kvol * mu), ud = zconj(__ldg(u + dn[mu] + kvol * mu));
        const double2 tt = zmul(c_tgv[mu][d], zsub(zmul(uu, at(s, up[mu], dg)),
                                                   zmul(ud, at(s, dn[mu], dg))));
        phi = DAG ? zsub(phi, tt) : zadd(phi, tt);
    }
    // s hops (:2004-2020): M takes Dirac 3,4 from s+1, Dirac 1,2 from s-1;
    // M^dagger the reverse (:2129-2145)
    const bool from_up = DAG ? d < 2 : d >= 2;
    if (from_up) {
        if (s < Ls - 1) phi = zsub(phi, at(s + 1, i, d));
    } else if (s > 0) {
        phi = zsub(phi, at(s - 1, i, d));
    }
    // mass term (:2022-2067, :2147-2186): group A at s=kthird (the pair that
    // takes s+1), group B at s=1 (the other pair)
    const bool grpA = s == Ls - 1 && from_up, grpB = s == 0 && !from_up;
    if (grpA || grpB) {
        double2 src;
        int sg;
        if (IMASS == 5) {
            src = at(s, i, d >= 2 ? d - 2 : d + 2);
            sg = -1;
        } else {
            src = at(grpA ? 0 : Ls - 1, i, d);
            sg = IMASS == 1 ? 1 : (grpA == !DAG ? -1 : 1);
        }
        const double2 tt = zmul(zk, src);
        phi = sg > 0 ? zadd(phi, tt) : zsub(phi, tt);
    }
    return phi;
}

// Stop state of a solve whose scalar recurrences run on the device: once
// done is set at iteration iters, the kernels queued for later iterations
// return at once (the host polls the flag only every few iterations).
struct ThrRun {
    int done, iters;   // done: 0 running, 1 converged, 2 at the iteration cap
};
__device__ __forceinline__ bool thr_skip(const ThrRun* run, int it) {
    return run != nullptr && run->done && it > run->iters;
}

template <bool DAG, int IMASS>
__global__ void __launch_bounds__(kThreads) k_thr_dslash(double2* __restrict__ out,
                                                         const double2* __restrict__ in,
                                                         const double2* __restrict__ u, TGeom g,
                                                         double diag, double2 zk,
                                                         const ThrRun* run, int it) {
    if (thr_skip(run, it)) return;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= g.kferm) return;
    if (g.kferm <= (int64_t)0xffffffffLL) {   // 32-bit divisions when every index fits
        const uint32_t uj = (uint32_t)j, Ls = (uint32_t)g.Ls, kv = (uint32_t)g.kvol;
        const uint32_t r = uj / Ls, d = r / kv;
        out[j] = thr_element<DAG, IMASS>(in, u, g, (int)(uj - r * Ls), (int64_t)(r - d * kv),
                                         (int)d, diag, zk);
        return;
    }
    const int s = (int)(j % g.Ls);
    const int64_t r = j / g.Ls;
    out[j] = thr_element<DAG, IMASS>(in, u, g, s, r % g.kvol, (int)(r / g.kvol), diag, zk);
}

// derivs (:820-878), one thread per link (i, mu): for Dirac d and s in the
// reference's order, the Wilson term then the Dirac term, each rounded to
// REAL*4 as it is added.  The sum is a serial chain; the operands of the next
// kDerivS values of s are loaded while those before are added (12^3x12: 32 ->
// 15 us).
constexpr int kDerivS = 4;
struct DerivBatch {
    double2 ri[kDerivS], ru[kDerivS], xi[kDerivS], xu[kDerivS], yi[kDerivS], yu[kDerivS];
};
__global__ void __launch_bounds__(kThreads) k_thr_derivs(const double2* __restrict__ R,
                                                         const double2* __restrict__ X2, TGeom g,
                                                         double tz, int iflag,
                                                         float* __restrict__ dS) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= 3 * (int64_t)g.kvol) return;
    const int64_t kvol = g.kvol;
    const int mu = (int)((uint32_t)j / (uint32_t)kvol);    // j < 3 kvol < 2^32
    const int64_t i = j - (int64_t)mu * kvol;
    const int Ls = g.Ls;
    int x, y, t;
    tsite_xyt(g.L, i, &x, &y, &t);
    int64_t up, dn;
    tnbr(g, x, y, t, mu, &up, &dn);
    const double2 tzi = make_double2(0.0, tz);
    float f = dS[j];
    const int per = (Ls + kDerivS - 1) / kDerivS, nb = 4 * per;      // batches
    auto load = [&](DerivBatch& v, int b) {
        const int bb = b < nb ? b : nb - 1, d = bb / per, s0 = (bb - d * per) * kDerivS;
        const int64_t ei = Ls * (i + kvol * d), eu = Ls * (up + kvol * d);
        const int64_t gi = Ls * (i + kvol * c_tgi[mu][d]), gu = Ls * (up + kvol * c_tgi[mu][d]);
#pragma unroll
        for (int q = 0; q < kDerivS; q++) {
            const int s = s0 + q < Ls ? s0 + q : Ls - 1;
            v.ri[q] = zconj(R[ei + s]);
            v.ru[q] = zconj(R[eu + s]);
            v.xi[q] = X2[ei + s];
            v.xu[q] = X2[eu + s];
            v.yi[q] = X2[gi + s];
            v.yu[q] = X2[gu + s];
        }
    };
    auto add = [&](const DerivBatch& v, int b) {
        if (b >= nb) return;
        const int d = b / per, ns = Ls - (b - d * per) * kDerivS;
        const double2 tg = zmul(tzi, c_tgv[mu][d]);
#pragma unroll
        for (int q = 0; q < kDerivS; q++) {
            if (q >= ns) break;
            const double2 w = zmul(tzi, zsub(zmul(v.ri[q], v.xu[q]), zmul(v.ru[q], v.xi[q])));
            f = __double2float_rn(__dsub_rn((double)f, __dmul_rn(0.5, w.x)));     // :843-850
            const double2 w2 = zmul(tg, zadd(zmul(v.ri[q], v.yu[q]), zmul(v.ru[q], v.yi[q])));
            f = __double2float_rn(iflag == 0 ? __dsub_rn((double)f, w2.x)             // :851-868
                                             : __dadd_rn((double)f, w2.x));
        }
    };
    DerivBatch v0, v1;
    load(v0, 0);
    for (int b = 0; b < nb; b += 2) {
        load(v1, b + 1);
        add(v0, b);
        load(v0, b + 2);
        add(v1, b + 1);
    }
    dS[j] = f;
}

// coef (:1799-1827)
__global__ void k_thr_coef(const float* __restrict__ theta, double2* __restrict__ u, TGeom g) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= 3 * (int64_t)g.kvol) return;
    double2 v = make_double2(1.0, (double)theta[j]);
    const int64_t i = j % g.kvol;
    if (j / g.kvol == 2 && i >= (int64_t)(g.Lt - 1) * g.L * g.L) v = make_double2(-v.x, -v.y);
    u[j] = v;
}

// ---- multi-shift solver kernels (qmrherm, :630-818) ------------------------
struct PoleCoef {
    double rho[kThrMaxPoles], amu[kThrMaxPoles];
};

// One iteration is two kernels, one thread a point (s, site) with its four
// Dirac components, so a neighbour and a link serve all four:
//   k_thr_m    vt = M R, |vt|^2
//   k_thr_md   q = R/beta, R' = M^dagger vt/beta - alphatild q - beta q', |R'|^2
// with alphatild = q^dagger M^dagger M q = |vt|^2/beta^2, so that the vector
// enters M before beta = |R| is known and neither sum needs a kernel of its
// own: a block leaves its partial and k_thr_md's blocks add both sums' partials
// themselves.  One block more forms the pole recurrences with the reference's
// implicit types.  The q of a chunk of iterations are kept, and k_thr_poles
// takes p_k and x_k through all of them at once, so the 2*ndiag vectors are read
// and written once a chunk instead of once an iteration.
// At 12^3x12 with 12 poles (162 blocks: launches and latency) an iteration takes
// 9.8 us, k_thr_poles' share in it (28 us a chunk of 16); the call with 160
// iterations, its 12 link forces and its host copies 2.3 to 2.5 ms, against 9.9 to 10.4
// with seven kernels an iteration, two of which ended in a serial sum over 592
// partials, and p_k and x_k updated every time.
constexpr int kThrBlock = 128;
constexpr int kThrChunk = 16;                  // q kept, at most
// The q that a handle keeps: a longer chunk is an option, so it takes at most a
// quarter of the memory that is free beside everything else, and else the two that
// the solvers need (an even number of iterations).
inline int thr_chunk(size_t vector_bytes, size_t free_bytes) {
    int chunk = kThrChunk;
    while (chunk > 2 && vector_bytes * chunk > free_bytes / 4) chunk /= 2;
    return chunk;
}
struct ThrQCtl {
    ThrRun run[2];                             // by parity of the iteration
    int base, next;                            // iterations before this chunk, before the next
    int niterc, ndiag;
    float phimod, resid;
    double aden[kThrMaxPoles], d[kThrMaxPoles], rhom1[kThrMaxPoles];
    double rho[kThrChunk][kThrMaxPoles], amu[kThrChunk][kThrMaxPoles];
};
struct ThrQArgs {
    TGeom g;
    int nblk, chunk;                           // blocks, iterations a chunk (even)
    double2 *rr, *vt, *ring;                   // R, M R, the chunk's q
    const double2* u;
    double diag;
    double2 zk, zkd;
    double* part;                              // |vt|^2, |R|^2 of even and odd iterations
    double2 *p, *x1;
    ThrQCtl* c;
    int* hflag;
};

__device__ __forceinline__ double2 zfma(double2 a, double2 b, double2 c) {   // a b + c
    return make_double2(__fma_rn(a.x, b.x, __fma_rn(-a.y, b.y, c.x)),
                        __fma_rn(a.x, b.y, __fma_rn(a.y, b.x, c.y)));
}

// The four components of M R or M^dagger R at (s, site i): thr_element's terms,
// the two hops of a direction together.
template <bool DAG, int IMASS>
__device__ __forceinline__ void thr_point(double2 phi[4], const double2* R,
                                          const double2* __restrict__ u, const TGeom& g, int s,
                                          int i, double diag, double2 zk) {
    const int L = g.L, Ls = g.Ls;
    const int64_t kvol = g.kvol, cs = (int64_t)Ls * kvol;
    const double2* r0 = R + s + (int64_t)Ls * i;
    int x, y, t;
    tsite_xyt(L, i, &x, &y, &t);
#pragma unroll
    for (int d = 0; d < 4; d++) phi[d] = zscal(diag, r0[cs * d]);
#pragma unroll
    for (int mu = 0; mu < 3; mu++) {
        int64_t up, dn;
        tnbr(g, x, y, t, mu, &up, &dn);
        const double2 uu = __ldg(u + i + kvol * mu), ud = zconj(__ldg(u + dn + kvol * mu));
        const double2 *ru = R + s + Ls * up, *rd = R + s + Ls * dn;
        double2 a[4], b[4];
#pragma unroll
        for (int d = 0; d < 4; d++) {
            a[d] = ru[cs * d];
            b[d] = rd[cs * d];
        }
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const double2 z = make_double2(0.0, 0.0);
            a[d] = zfma(uu, a[d], z);
            b[d] = zfma(ud, b[d], z);
        }
        // gamval(mu, d) is +-1/2 (mu 1) or +-i/2 (mu 0, 2), gamin(mu, d): d' = 3-d, 3-d, d^2
        constexpr double sg[3][4] = {{-.5, -.5, .5, .5}, {-.5, .5, .5, -.5}, {-.5, .5, .5, -.5}};
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int dg = mu == 2 ? d ^ 2 : 3 - d;
            const double h = DAG ? -sg[mu][d] : sg[mu][d];
            const double2 w = zadd(a[d], b[d]), v = zsub(a[dg], b[dg]);
            phi[d].x = __fma_rn(-0.5, w.x, phi[d].x);
            phi[d].y = __fma_rn(-0.5, w.y, phi[d].y);
            phi[d].x = mu == 1 ? __fma_rn(h, v.x, phi[d].x) : __fma_rn(-h, v.y, phi[d].x);
            phi[d].y = mu == 1 ? __fma_rn(h, v.y, phi[d].y) : __fma_rn(h, v.x, phi[d].y);
        }
    }
    constexpr int UP = DAG ? 0 : 2, DN = DAG ? 2 : 0;   // pair that takes s+1, s-1
#pragma unroll
    for (int d = 0; d < 2; d++) {
        if (s < Ls - 1) phi[UP + d] = zsub(phi[UP + d], r0[cs * (UP + d) + 1]);
        if (s > 0) phi[DN + d] = zsub(phi[DN + d], r0[cs * (DN + d) - 1]);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const bool grpA = k < 2;
        if (grpA ? s != Ls - 1 : s != 0) continue;
        const int d = grpA ? UP + k : DN + k - 2;
        if (IMASS == 5) phi[d] = zsub(phi[d], zmul(zk, r0[cs * (d ^ 2)]));
        else {
            const double2 tt = zmul(zk, r0[cs * d + (grpA ? 1 - Ls : Ls - 1)]);
            phi[d] = IMASS == 3 && grpA == !DAG ? zsub(phi[d], tt) : zadd(phi[d], tt);
        }
    }
}
__device__ __forceinline__ double znorm2(double2 v) { return v.x * v.x + v.y * v.y; }

// Points of the block's threads: (s, site) = j, s fastest.
template <class F>
__device__ __forceinline__ void thr_points(const TGeom& g, F&& f) {
    const int64_t n = (int64_t)g.kvol * g.Ls, step = (int64_t)gridDim.x * kThrBlock;
    for (int64_t j = (int64_t)blockIdx.x * kThrBlock + threadIdx.x; j < n; j += step) {
        int64_t i;
        if (n <= (int64_t)0xffffffffLL) i = (uint32_t)j / (uint32_t)g.Ls;
        else i = j / g.Ls;
        f(j, (int)(j - i * g.Ls), (int)i);
    }
}

__global__ void k_thr_tick(ThrQCtl* c, int chunk) {
    c->base = c->next;
    c->next += chunk;
}

// R = Phi, partials of |R|^2
__global__ void __launch_bounds__(kThrBlock) k_thr_start(ThrQArgs a,
                                                         const double2* __restrict__ Phi) {
    __shared__ double sh[32];
    double loc = 0.0;
    for (int64_t j = (int64_t)blockIdx.x * kThrBlock + threadIdx.x; j < a.g.kferm;
         j += (int64_t)gridDim.x * kThrBlock) {
        const double2 v = Phi[j];
        a.rr[j] = v;
        loc += znorm2(v);
    }
    loc = block_sum_any(loc, sh);
    if (threadIdx.x == 0) a.part[a.nblk + blockIdx.x] = loc;
}

template <int IMASS>
__global__ void __launch_bounds__(kThrBlock, 4) k_thr_m(ThrQArgs a, int k) {
    __shared__ double sh[32];
    pdl_wait();
    if (a.c->run[k & 1].done) return;
    double loc = 0.0;
    thr_points(a.g, [&](int64_t j, int s, int i) {
        double2 phi[4];
        thr_point<false, IMASS>(phi, a.rr, a.u, a.g, s, i, a.diag, a.zk);
#pragma unroll
        for (int d = 0; d < 4; d++) {
            a.vt[j + (int64_t)a.g.Ls * a.g.kvol * d] = phi[d];
            loc += znorm2(phi[d]);
        }
    });
    loc = block_sum_any(loc, sh);
    if (threadIdx.x == 0) a.part[blockIdx.x] = loc;
}

// The pole recurrences of iteration it (:712-747) and the stopping test
// (:750-757), by the threads of a block of their own.
__device__ __forceinline__ void thr_scalars(const ThrQArgs& a, int k, int it, double beta,
                                            float alphat) {
    __shared__ float rm[kThrMaxPoles];
    ThrQCtl* c = a.c;
    const int nd = c->ndiag, p = threadIdx.x;
    const float beta0 = (float)beta;
    const float phimod = it == 1 ? beta0 : c->phimod;
    if (p < nd) {
        const double alpha = __dadd_rn((double)alphat, c->aden[p]);
        double rho, amu = 0.0;
        if (it == 1) {
            c->d[p] = alpha;
            rho = __ddiv_rn((double)beta0, alpha);
        } else {
            const double dm1 = c->d[p];
            amu = __ddiv_rn((double)beta0, dm1);
            const double dk = __dsub_rn(alpha, __dmul_rn((double)beta0, amu));
            rho = -__ddiv_rn(__dmul_rn(__dmul_rn(amu, dm1), c->rhom1[p]), dk);
            c->d[p] = dk;
            rm[p] = (float)fabs(__dmul_rn((double)phimod, rho));
        }
        c->rho[k][p] = rho;
        c->amu[k][p] = amu;
        c->rhom1[p] = rho;
    }
    __syncthreads();
    if (p != 0) return;
    if (it == 1) c->phimod = phimod;
    float rhomax = rm[0];
    for (int q = 1; q < nd; q++)
        if (rm[q] > rhomax) rhomax = rm[q];
    ThrRun r{0, 0};
    const float arelax = 2.0f;
    if (it > 1 && rhomax < __fmul_rn(arelax, c->resid)) r = ThrRun{1, it};
    else if (it >= c->niterc) r = ThrRun{2, it};
    c->run[(k + 1) & 1] = r;
    if (r.done && a.hflag) {
        *(volatile int*)a.hflag = r.done;
        __threadfence_system();
    }
}

// Sums of two runs of n <= kRedBlocks partials, the same in every block.
struct ThrSum2 {
    static constexpr int N = (kRedBlocks + kThrBlock - 1) / kThrBlock;
    double a[N], b[N];
    __device__ __forceinline__ void load(const double* pa, const double* pb, int n) {
#pragma unroll
        for (int q = 0; q < N; q++) {
            const int i = threadIdx.x + q * kThrBlock;
            a[q] = i < n ? __ldcg(pa + i) : 0.0;
            b[q] = i < n ? __ldcg(pb + i) : 0.0;
        }
    }
    __device__ __forceinline__ void sum(double* ta, double* tb) {
        __shared__ double sa[kThrBlock / 32], sb[kThrBlock / 32];
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int q = 0; q < N; q++) {
            x += a[q];
            y += b[q];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            x += __shfl_xor_sync(0xffffffffu, x, o);
            y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        if ((threadIdx.x & 31) == 0) {
            sa[threadIdx.x >> 5] = x;
            sb[threadIdx.x >> 5] = y;
        }
        __syncthreads();
        x = y = 0.0;
#pragma unroll
        for (int w = 0; w < kThrBlock / 32; w++) {
            x += sa[w];
            y += sb[w];
        }
        *ta = x;
        *tb = y;
    }
};

template <int IMASS>
__global__ void __launch_bounds__(kThrBlock, 4) k_thr_md(ThrQArgs a, int k) {
    __shared__ double sh[32];
    pdl_wait();
    const ThrRun run = a.c->run[k & 1];
    const bool scalars = blockIdx.x == (unsigned)a.nblk;      // the block behind the points'
    if (run.done) {
        if (scalars && threadIdx.x == 0) a.c->run[(k + 1) & 1] = run;
        return;
    }
    const int it = a.c->base + k + 1;
    ThrSum2 sums;
    sums.load(a.part, a.part + (size_t)a.nblk * (1 + (k & 1)), a.nblk);
    // the first point's hops while the partials are on their way
    const int64_t n = (int64_t)a.g.kvol * a.g.Ls, cs = n;
    int64_t j = (int64_t)blockIdx.x * kThrBlock + threadIdx.x;
    double2 phi[4];
    auto point = [&] {
        const int64_t i = n <= (int64_t)0xffffffffLL ? (uint32_t)j / (uint32_t)a.g.Ls : j / a.g.Ls;
        thr_point<true, IMASS>(phi, a.vt, a.u, a.g, (int)(j - i * a.g.Ls), (int)i, a.diag, a.zkd);
    };
    bool act = !scalars && j < n;
    if (act) point();
    double v2, b2;
    sums.sum(&v2, &b2);
    const double beta = __dsqrt_rn(b2), inv = 1.0 / beta;               // :684-694
    const float alphat = (float)(v2 / b2);
    if (scalars) {
        thr_scalars(a, k, it, beta, alphat);
        return;
    }
    const double2* qm1 = a.ring + a.g.kferm * (int64_t)(k > 0 ? k - 1 : a.chunk - 1);
    double2* q = a.ring + a.g.kferm * (int64_t)k;
    double loc = 0.0;
    while (act) {
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int64_t e = j + cs * d;
            const double2 qj = zscal(inv, a.rr[e]);
            double2 r = zsub(zscal(inv, phi[d]), zscal((double)alphat, qj));
            if (it > 1) r = zsub(r, zscal(beta, qm1[e]));
            q[e] = qj;
            a.rr[e] = r;
            loc += znorm2(r);
        }
        j += (int64_t)a.nblk * kThrBlock;
        act = j < n;
        if (act) point();
    }
    loc = block_sum_any(loc, sh);
    if (threadIdx.x == 0) a.part[(size_t)a.nblk * (2 - (k & 1)) + blockIdx.x] = loc;
}

// p_k = q - amu_k p_k, x_k += rho_k p_k for the chunk's iterations (first
// iteration of a solve: p_k = q, x_k = rho_k q; :712-747, pm1 equals p), four
// poles a thread: q is read ndiag/4 times.
constexpr int kThrPoles = 4;
__global__ void __launch_bounds__(kThreads) k_thr_poles(ThrQArgs a) {
    const ThrQCtl* c = a.c;
    const ThrRun run = c->run[0];              // a chunk is an even number of iterations
    const int base = c->base;
    const int nit = run.done ? run.iters - base : a.chunk;
    const int64_t n = a.g.kferm, j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (nit <= 0 || j >= n) return;
    const int k0 = (int)blockIdx.y * kThrPoles, nk = min(kThrPoles, c->ndiag - k0);
    double2 p[kThrPoles], x[kThrPoles];
#pragma unroll
    for (int k = 0; k < kThrPoles; k++) {
        p[k] = x[k] = make_double2(0.0, 0.0);
        if (k < nk && base > 0) {
            p[k] = a.p[j + n * (k0 + k)];
            x[k] = a.x1[j + n * (k0 + k)];
        }
    }
#pragma unroll 4
    for (int it = 0; it < nit; it++) {
        const double2 q = a.ring[j + n * it];
#pragma unroll
        for (int k = 0; k < kThrPoles; k++) {
            if (k >= nk) continue;
            const double rho = c->rho[it][k0 + k], amu = c->amu[it][k0 + k];
            p[k] = base + it == 0 ? q : zsub(q, zscal(amu, p[k]));
            x[k] = zadd(x[k], zscal(rho, p[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < kThrPoles; k++) {
        if (k >= nk) continue;
        a.p[j + n * (k0 + k)] = p[k];
        a.x1[j + n * (k0 + k)] = x[k];
    }
}

// Grid sum of one double per thread with the block partials added in block
// order by one thread (the order of a host loop over the partials).  The
// block that arrives last returns true with the total in *total (thread 0)
// and resets the counter.  NB is the fixed grid size of the reductions.
template <int NT, int NB>
__device__ __forceinline__ bool last_block_seq(double v, double* part, unsigned* count,
                                               double* total) {
    __shared__ double sh[NT / 32];
    __shared__ double all[NB];
    __shared__ bool is_last;
    v = block_sum<NT>(v, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = v;
        __threadfence();
        is_last = (atomicAdd(count, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    for (int i = threadIdx.x; i < NB; i += blockDim.x) all[i] = ((volatile double*)part)[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int b = 0; b < NB; b++) s = __dadd_rn(s, all[b]);
        *total = s;
        *count = 0;
    }
    return true;
}

// block partials of sum Re(conjg(a)*b); the host adds them in block order
__global__ void __launch_bounds__(kThreads) k_thr_dot(const double2* __restrict__ a,
                                                      const double2* __restrict__ b, int64_t n,
                                                      double* __restrict__ part) {
    __shared__ double sh[kThreads / 32];
    double loc = 0.0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x)
        loc += zmul(zconj(a[j]), b[j]).x;
    loc = block_sum<kThreads>(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = loc;
}

// x = anum0 Phi, then x += anum_k x_k in pole order (:666, :766-772)
__global__ void k_thr_combine(double2* __restrict__ x, const double2* __restrict__ Phi,
                              const double2* __restrict__ x1, PoleCoef c, double a0, int npole,
                              int64_t n) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    double2 v = zscal(a0, Phi[j]);
    for (int k = 0; k < npole; k++) v = zadd(v, zscal(c.rho[k], x1[j + n * k]));
    x[j] = v;
}

// R = x3 - ... helpers for the leapfrog: pp -= dS*d ; theta += d*pp
__global__ void k_thr_update_p(float* __restrict__ pp, const float* __restrict__ dS, float d,
                               int64_t n) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j < n) pp[j] = __fsub_rn(pp[j], __fmul_rn(dS[j], d));
}
__global__ void k_thr_update_theta(float* __restrict__ th, const float* __restrict__ pp,
                                   float d, int64_t n) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j < n) th[j] = __fadd_rn(th[j], __fmul_rn(d, pp[j]));
}

// end of force (:520-532): the antiperiodic sign on the t links of the last
// slice, then dSdpi + beta*Nf*theta
__global__ void k_thr_force_end(float* __restrict__ dS, const float* __restrict__ theta,
                                float b, TGeom g) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= 3 * (int64_t)g.kvol) return;
    float v = dS[j];
    if (j / g.kvol == 2 && j % g.kvol >= (int64_t)(g.Lt - 1) * g.L * g.L) v = -v;
    dS[j] = __fadd_rn(v, __fmul_rn(b, theta[j]));
}

// R(s, i, d) = cmplx(ps(i,1), ps(i,2)) of gauss0 call d*kthird + s (:213-222)
__global__ void k_thr_noise(double2* __restrict__ R, const float* __restrict__ gauss, TGeom g) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= g.kferm) return;
    const int s = (int)(j % g.Ls);
    const int64_t r = j / g.Ls;
    const int64_t site = r % g.kvol;
    const int64_t c = (r / g.kvol) * g.Ls + s;
    const float* ps = gauss + c * 2 * g.kvol;
    R[j] = make_double2((double)ps[site], (double)ps[g.kvol + site]);
}

// ---- congrad (:931-1025) and measure (:1027-1285) -------------------------
// The REAL*4 scalars of congrad, formed on the device like those of qmrherm.
struct ThrCgCtl {
    ThrRun run;
    int64_t niterc;
    float alpha, alphan, betad, beta, resid, pad_;
    unsigned count1, count2;
};

// alphad = |x1|^2 ; alpha = alphan/alphad (:970-977)
__global__ void __launch_bounds__(kThreads) k_thr_cg_alpha(const double2* __restrict__ x1,
                                                           int64_t n, double* __restrict__ part,
                                                           ThrCgCtl* __restrict__ c, int it) {
    if (thr_skip(&c->run, it)) return;
    double loc = 0.0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x)
        loc += zmul(zconj(x1[j]), x1[j]).x;
    double tot;
    if (!last_block_seq<kThreads, kRedBlocks>(loc, part, &c->count1, &tot)) return;
    if (threadIdx.x == 0) c->alpha = __fdiv_rn(c->alphan, (float)tot);
}

// x += alpha p (:979-983)
__global__ void k_thr_axpy(double2* __restrict__ x, const double2* __restrict__ p,
                           const ThrCgCtl* __restrict__ c, int it, int64_t n) {
    if (thr_skip(&c->run, it)) return;
    const double a = (double)c->alpha;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j < n) x[j] = zadd(x[j], zscal(a, p[j]));
}

// r -= alpha x2 ; betan = |r|^2, beta and the stopping test (:989-1001) in
// the last block
__global__ void __launch_bounds__(kThreads) k_thr_cg_r(double2* __restrict__ r,
                                                       const double2* __restrict__ x2, int64_t n,
                                                       double* __restrict__ part,
                                                       ThrCgCtl* __restrict__ c, int it,
                                                       int* hflag) {
    if (thr_skip(&c->run, it)) return;
    const double a = (double)c->alpha;
    double loc = 0.0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = zsub(r[j], zscal(a, x2[j]));
        r[j] = v;
        loc += zmul(zconj(v), v).x;
    }
    double bn;
    if (!last_block_seq<kThreads, kRedBlocks>(loc, part, &c->count2, &bn)) return;
    if (threadIdx.x != 0) return;
    const float betan = (float)bn;
    float beta = __fdiv_rn(betan, c->betad);
    c->betad = betan;
    c->alphan = betan;
    if (it == 1) beta = 0.0f;
    c->beta = beta;
    if (betan < c->resid) {
        c->run.iters = it;
        c->run.done = 1;
    } else if (it >= c->niterc) {
        c->run.iters = it;
        c->run.done = 2;
    }
    if (c->run.done && hflag) {
        *(volatile int*)hflag = c->run.done;
        __threadfence_system();
    }
}

// p = r + beta p (:1003-1005); runs in the iteration that stopped the solve
__global__ void k_thr_xpay(double2* __restrict__ p, const double2* __restrict__ r,
                           const ThrCgCtl* __restrict__ c, int it, int64_t n) {
    if (thr_skip(&c->run, it)) return;
    const double b = (double)c->beta;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j < n) p[j] = zadd(r[j], zscal(b, p[j]));
}

// xi = 0 except component d at wall s: sgn*cmplx(eta(i,1), eta(i,2))
__global__ void k_thr_wall_source(double2* __restrict__ xi, const float* __restrict__ eta,
                                  int s, int d, double sgn, TGeom g) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= g.kferm) return;
    const int sj = (int)(j % g.Ls);
    const int64_t r = j / g.Ls;
    const int64_t i = r % g.kvol;
    const int dj = (int)(r / g.kvol);
    double2 v = make_double2(0.0, 0.0);
    if (sj == s && dj == d) v = make_double2(sgn * (double)eta[i], sgn * (double)eta[g.kvol + i]);
    xi[j] = v;
}

// out[i] = x(s, i, d)
__global__ void k_thr_slice(const double2* __restrict__ x, int s, int d, TGeom g,
                            double2* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < g.kvol) out[i] = x[s + (int64_t)g.Ls * (i + (int64_t)g.kvol * d)];
}

unsigned tblk(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

}  // namespace
}  // namespace chdwf

using chdwf::TGeom;

struct ThrRemez {
    std::vector<double> anum, aden, bnum, bden;
    int n = 0;
};

struct chdwf_thr {
    int device = 0;
    TGeom g{};
    float dt = 0.1f, beta = 0.5f, am3 = 1.0f, am = 0.0f;
    int imass = 1, iterl = 1, iprint = 5;
    float rescga = 0.000000001f, rescgg = 0.000001f;                   // :39
    float respbp = 0.000001f;                                            // :39
    ThrRemez r2, r4, r2g, r4g;
    cudaStream_t st = nullptr;
    float *theta = nullptr, *thetat = nullptr, *pp = nullptr, *dS = nullptr, *gauss = nullptr;
    double2 *ut = nullptr, *uio = nullptr;
    double2 *Phi = nullptr, *X1 = nullptr, *R = nullptr, *X2 = nullptr, *Phi0 = nullptr;
    double2 *vt = nullptr, *rr = nullptr;
    double2* ring = nullptr;              // chunk vectors: the q of a chunk of iterations
    int chunk = 0;
    chdwf::ChunkGraphs graphs;
    double2 *p = nullptr, *x1 = nullptr;
    double* part = nullptr;
    std::vector<double> hpart;
    chdwf::ThrQCtl* qctl = nullptr;       // device scalars of qmrherm
    chdwf::ThrCgCtl* cgctl = nullptr;     // device scalars of congrad
    int* hflag_host = nullptr;            // stop flag, mapped pinned memory
    int* hflag_dev = nullptr;
    chdwf::Rng rng;
    int isweep = 0, itot = 0, naccp = 0;
    float action = 0.0f, gaction = 0.0f, paction = 0.0f;
    float actiona = 0.0f, vel2a = 0.0f, yav = 0.0f, yyav = 0.0f;
    std::string err;

    double diag() const { return (double)((3.0f - am3) + 1.0f); }       // :1967
    int fail(cudaError_t e, const char* where) {
        err = std::string(where) + ": " + cudaGetErrorString(e);
        return CHDWF_CUDA_ERROR;
    }
};

namespace {

thread_local std::string g_thr_create_err;

template <class T>
cudaError_t talloc(T** p, size_t n) { return cudaMalloc((void**)p, sizeof(T) * n); }

double2 thr_mass(float am, int imass, bool dag) {
    return imass == 1 ? make_double2((double)am, 0.0)
                      : make_double2(0.0, dag ? (double)am : (double)(-am));
}

// The launches of a chunk of qmrherm's iterations.
template <int IMASS>
void thr_launch_chunk(const chdwf::ThrQArgs& a, int ndiag, cudaStream_t st) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.blockDim = dim3(chdwf::kThrBlock);
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    chdwf::k_thr_tick<<<1, 1, 0, st>>>(a.c, a.chunk);
    for (int k = 0; k < a.chunk; k++) {
        c.gridDim = dim3((unsigned)a.nblk);
        cudaLaunchKernelEx(&c, chdwf::k_thr_m<IMASS>, a, k);
        c.gridDim = dim3((unsigned)a.nblk + 1);
        cudaLaunchKernelEx(&c, chdwf::k_thr_md<IMASS>, a, k);
    }
    const dim3 grid(chdwf::tblk(a.g.kferm), (unsigned)((ndiag + chdwf::kThrPoles - 1) / chdwf::kThrPoles));
    chdwf::k_thr_poles<<<grid, chdwf::kThreads, 0, st>>>(a);
}

void thr_dslash(chdwf_thr* h, bool dag, float am, int imass, double2* out, const double2* in,
                const double2* u, const chdwf::ThrRun* run = nullptr, int it = 0) {
    const unsigned nb = chdwf::tblk(h->g.kferm);
    const double2 zk = thr_mass(am, imass, dag);
    const double dg = h->diag();
#define THR_LAUNCH(D, I) chdwf::k_thr_dslash<D, I><<<nb, chdwf::kThreads, 0, h->st>>>(out, in, u, h->g, dg, zk, run, it)
    if (dag) {
        if (imass == 1) THR_LAUNCH(true, 1); else if (imass == 3) THR_LAUNCH(true, 3); else THR_LAUNCH(true, 5);
    } else {
        if (imass == 1) THR_LAUNCH(false, 1); else if (imass == 3) THR_LAUNCH(false, 3); else THR_LAUNCH(false, 5);
    }
#undef THR_LAUNCH
    chdwf::count_launches(1);
}

void thr_derivs(chdwf_thr* h, const double2* R, const double2* X2, double anum, int iflag) {
    const double tz = (double)(float)(2.0 * anum);                         // tzi, :839
    // small blocks: few links, each a long chain
    const unsigned nb = (unsigned)((3 * (int64_t)h->g.kvol + 31) / 32);
    chdwf::k_thr_derivs<<<nb, 32, 0, h->st>>>(
        R, X2, h->g, tz, iflag, h->dS);
    chdwf::count_launches(1);
}

// sum of the block partials in block order
cudaError_t thr_sum(chdwf_thr* h, double* out) {
    cudaMemcpyAsync(h->hpart.data(), h->part, sizeof(double) * chdwf::kRedBlocks,
                    cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    double s = 0.0;
    for (int b = 0; b < chdwf::kRedBlocks; b++) s = s + h->hpart[b];
    *out = s;
    return e;
}

// Launches a solve in chunks of iterations until the device raises the stop
// flag or cap iterations are queued: launch(first) queues the chunk that
// begins with iteration first.  The flag is read one chunk behind, so up to two
// chunks are in flight; the kernels of iterations past the stopping one return
// at once.
template <class F>
cudaError_t thr_run_chunks(chdwf_thr* h, int64_t cap, int chunk, F&& launch) {
    cudaEvent_t ev[2];
    cudaError_t e = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
    if (e) return e;
    if ((e = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming))) {
        cudaEventDestroy(ev[0]);
        return e;
    }
    int nchunk = 0;
    for (int64_t first = 1; first <= cap; first += chunk) {
        launch((int)first);
        if ((e = cudaGetLastError())) break;
        cudaEventRecord(ev[nchunk & 1], h->st);
        if (nchunk >= 1) {
            if ((e = cudaEventSynchronize(ev[(nchunk - 1) & 1]))) break;
            if (*(volatile int*)h->hflag_host) break;
        }
        nchunk++;
    }
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    return e;
}

// qmrherm on device vectors (:630-818): Phi in, x out, Phi0 and dS of the
// context; the scalars follow the reference's implicit typing.
int thr_qmrherm(chdwf_thr* h, const double2* Phi, float res, int* itercg, float am, int imass,
                const double* anum, const double* aden, int ndiag, int iflag, const double2* u,
                double2* x) {
    const int64_t n = h->g.kferm;
    const unsigned nb = chdwf::tblk(n);
    const int niterc = 7500;                                             // :635
    const float resid = std::sqrt((float)n * res * res);                // :660
    cudaError_t e;
    chdwf::ThrQCtl hc;
    memset(&hc, 0, sizeof(hc));
    hc.resid = resid;
    hc.niterc = niterc;
    hc.ndiag = ndiag;
    for (int k = 0; k < ndiag; k++) hc.aden[k] = aden[k];
    if ((e = cudaMemcpyAsync(h->qctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, h->st)))
        return h->fail(e, "thr_qmrherm");
    *h->hflag_host = 0;
    chdwf::ThrQArgs a;
    memset(&a, 0, sizeof(a));
    a.g = h->g;
    const int64_t pts = (int64_t)h->g.kvol * h->g.Ls;
    a.nblk = (int)std::min<int64_t>((pts + chdwf::kThrBlock - 1) / chdwf::kThrBlock,
                                    chdwf::kRedBlocks);
    a.chunk = h->chunk;
    a.rr = h->rr; a.vt = h->vt; a.ring = h->ring;
    a.u = u;
    a.diag = h->diag();
    a.zk = thr_mass(am, imass, false);
    a.zkd = thr_mass(am, imass, true);
    a.part = h->part;
    a.p = h->p; a.x1 = h->x1;
    a.c = h->qctl;
    a.hflag = h->hflag_dev;
    chdwf::k_thr_start<<<a.nblk, chdwf::kThrBlock, 0, h->st>>>(a, Phi);   // :662-667
    chdwf::count_launches(1);
    auto chunk = [&] {
        if (imass == 1) thr_launch_chunk<1>(a, ndiag, h->st);
        else if (imass == 3) thr_launch_chunk<3>(a, ndiag, h->st);
        else thr_launch_chunk<5>(a, ndiag, h->st);
    };
    const cudaGraphExec_t ge = h->graphs.get(a, imass + 8 * ndiag, h->st, chunk);
    e = thr_run_chunks(h, niterc, a.chunk, [&](int) {
        if (ge) cudaGraphLaunch(ge, h->st);
        else chunk();
        chdwf::count_launches(2 * a.chunk + 2);
    });
    if (e) return h->fail(e, "thr_qmrherm");
    chdwf::ThrRun hr;
    if ((e = cudaMemcpyAsync(&hr, &h->qctl->run[0], sizeof(hr), cudaMemcpyDeviceToHost, h->st)) ||
        (e = cudaStreamSynchronize(h->st)))
        return h->fail(e, "thr_qmrherm");
    *itercg = hr.iters;
    const int capped = hr.done != 1;
    chdwf::PoleCoef c0;
    memset(&c0, 0, sizeof(c0));
    if (iflag < 2) {                                                       // :766-780
        chdwf::PoleCoef a;
        for (int k = 0; k < ndiag; k++) a.rho[k] = anum[k + 1];
        chdwf::k_thr_combine<<<nb, chdwf::kThreads, 0, h->st>>>(x, Phi, h->x1, a, anum[0], ndiag, n);
        chdwf::count_launches(1);
        if (iflag == 1)
            cudaMemcpyAsync(h->Phi0, h->x1, sizeof(double2) * n * ndiag, cudaMemcpyDeviceToDevice,
                            h->st);
    } else {                                                               // :781-806
        chdwf::k_thr_combine<<<nb, chdwf::kThreads, 0, h->st>>>(x, Phi, h->x1, c0, anum[0], 0, n);
        chdwf::count_launches(1);
        for (int k = 0; k < ndiag; k++) {
            const double2* xk = h->x1 + n * k;
            thr_dslash(h, false, am, imass, h->X2, xk, u);
            if (iflag == 2) {
                thr_derivs(h, xk, h->X2, anum[k + 1], 0);
            } else {
                const double coeff = -anum[k + 1];
                const double2* p0 = h->Phi0 + n * k;
                thr_derivs(h, p0, h->X2, coeff, 0);
                thr_dslash(h, false, am, imass, h->X2, p0, u);
                thr_derivs(h, h->X2, xk, coeff, 1);
            }
        }
    }
    if ((e = cudaGetLastError())) return h->fail(e, "thr_qmrherm");
    return capped ? CHDWF_ITER_CAP : CHDWF_OK;
}

// force (:449-535) on thetat/ut; its[4] receives the four solves' iterations
int thr_force(chdwf_thr* h, float res1, int* its) {
    const int64_t n = h->g.kferm;
    cudaMemsetAsync(h->dS, 0, sizeof(float) * 3 * h->g.kvol, h->st);   // :477-481
    int rc;
    const ThrRemez& a4 = h->r4g;
    const ThrRemez& r2 = h->r2g;
    rc = thr_qmrherm(h, h->Phi, res1, &its[0], 1.0f, 1, a4.anum.data(), a4.aden.data(), a4.n, 1,
                     h->ut, h->X1);                                       // :493
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    cudaMemcpyAsync(h->R, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    rc = thr_qmrherm(h, h->R, res1, &its[1], h->am, h->imass, r2.bnum.data(), r2.bden.data(), r2.n,
                     0, h->ut, h->X1);                                    // :500
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    cudaMemcpyAsync(h->R, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    rc = thr_qmrherm(h, h->R, res1, &its[2], h->am, h->imass, r2.anum.data(), r2.aden.data(), r2.n,
                     2, h->ut, h->X1);                                    // :509
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    rc = thr_qmrherm(h, h->R, res1, &its[3], 1.0f, 1, a4.anum.data(), a4.aden.data(), a4.n, 3,
                     h->ut, h->X1);                                       // :514
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    const float b = h->beta * 1.0f;                                       // b = beta*Nf, :527
    chdwf::k_thr_force_end<<<chdwf::tblk(3 * (int64_t)h->g.kvol), chdwf::kThreads, 0, h->st>>>(
        h->dS, h->thetat, b, h->g);
    chdwf::count_launches(1);
    const cudaError_t e = cudaGetLastError();
    return e ? h->fail(e, "thr_force") : CHDWF_OK;
}

// hamilton (:539-628): out = h, hg, hp, s; its = {mass m, PV}
int thr_hamilton(chdwf_thr* h, float res2, double* out, int* its) {
    const int64_t n = h->g.kferm, n3 = 3 * (int64_t)h->g.kvol;
    std::vector<float> pp(n3), th(n3);
    cudaMemcpyAsync(pp.data(), h->pp, sizeof(float) * n3, cudaMemcpyDeviceToHost, h->st);
    cudaMemcpyAsync(th.data(), h->thetat, sizeof(float) * n3, cudaMemcpyDeviceToHost, h->st);
    int rc = thr_qmrherm(h, h->Phi, res2, &its[1], 1.0f, 1, h->r4.anum.data(), h->r4.aden.data(),
                         h->r4.n, 0, h->ut, h->X1);                       // :596
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    cudaMemcpyAsync(h->R, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    rc = thr_qmrherm(h, h->R, res2, &its[0], h->am, h->imass, h->r2.bnum.data(), h->r2.bden.data(),
                     h->r2.n, 0, h->ut, h->X1);                           // :603
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    chdwf::k_thr_dot<<<chdwf::kRedBlocks, chdwf::kThreads, 0, h->st>>>(h->R, h->X1, n, h->part);
    chdwf::count_launches(1);
    double hf;
    const cudaError_t e = thr_sum(h, &hf);                                 // :607-609
    if (e) return h->fail(e, "thr_hamilton");
    double hp = 0.0, hg = 0.0;
    for (int64_t j = 0; j < n3; j++) hp = hp + (double)(pp[j] * pp[j]);         // :571-575
    hp = hp * 0.5;
    for (int64_t j = 0; j < n3; j++) hg = hg + (double)(th[j] * th[j]);
    hg = (double)(0.5f * 1.0f * h->beta) * hg;                          // :581
    out[0] = hg + hp + hf;
    out[1] = hg;
    out[2] = hp;
    out[3] = hg + hf;
    return CHDWF_OK;
}

// congrad (:931-1025) on device vectors: x in = guess, out = solution;
// REAL*4 scalars, FP64 sums rounded once.  Returns CHDWF_ITER_CAP at the cap.
int thr_congrad(chdwf_thr* h, const double2* Phi, float res, int* itercg, float am, int imass,
                const double2* u, double2* x) {
    const int64_t n = h->g.kferm;
    const unsigned nb = chdwf::tblk(n);
    const int64_t niterc = h->g.Ls * (int64_t)h->g.kvol;                 // :934
    const float resid = (float)n * res * res;                            // :947
    double2 *p = h->ring, *r = h->rr, *x1 = h->vt, *x2 = h->ring + n;
    cudaMemcpyAsync(p, x, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);   // :956-959
    cudaMemcpyAsync(r, Phi, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    chdwf::ThrCgCtl hc;
    memset(&hc, 0, sizeof(hc));
    hc.betad = 1.0f;                                                      // :951-952
    hc.alpha = 1.0f;
    hc.alphan = 0.0f;
    hc.resid = resid;
    hc.niterc = niterc;
    cudaError_t e;
    if ((e = cudaMemcpyAsync(h->cgctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, h->st)))
        return h->fail(e, "thr_congrad");
    *h->hflag_host = 0;
    chdwf::ThrCgCtl* c = h->cgctl;
    const chdwf::ThrRun* run = &c->run;
    e = thr_run_chunks(h, niterc, 16, [&](int first) {
      for (int it = first; it < first + 16 && it <= niterc; it++) {
        thr_dslash(h, false, am, imass, x1, p, u, run, it);               // :966
        if (it != 1) {                                                    // :970-983
            chdwf::k_thr_cg_alpha<<<chdwf::kRedBlocks, chdwf::kThreads, 0, h->st>>>(x1, n, h->part,
                                                                                   c, it);
            chdwf::k_thr_axpy<<<nb, chdwf::kThreads, 0, h->st>>>(x, p, c, it, n);
            chdwf::count_launches(2);
        }
        thr_dslash(h, true, am, imass, x2, x1, u, run, it);               // :987
        chdwf::k_thr_cg_r<<<chdwf::kRedBlocks, chdwf::kThreads, 0, h->st>>>(r, x2, n, h->part, c,
                                                                          it, h->hflag_dev);
        chdwf::k_thr_xpay<<<nb, chdwf::kThreads, 0, h->st>>>(p, r, c, it, n);
        chdwf::count_launches(2);
      }
    });
    if (e) return h->fail(e, "thr_congrad");
    chdwf::ThrRun hr;
    if ((e = cudaMemcpyAsync(&hr, run, sizeof(hr), cudaMemcpyDeviceToHost, h->st)) ||
        (e = cudaStreamSynchronize(h->st)))
        return h->fail(e, "thr_congrad");
    *itercg = hr.iters;
    return hr.done == 1 ? CHDWF_OK : CHDWF_ITER_CAP;
}

// measure (:1027-1285) with links u: psibarpsi, susclsing, aviter and the
// unit-100 records (parts, 40 doubles, or NULL).  Noise from the context's
// generator (two gauss0 calls per noise vector); the overlaps are summed on
// the host in the reference's order.
int thr_measure(chdwf_thr* h, float res, float am, int imass, const double2* u, float* psibarpsi,
                float* susclsing, float* aviter, double* parts) {
    const TGeom& g = h->g;
    const int64_t kvol = g.kvol, n = g.kferm;
    const int Ls = g.Ls;
    constexpr int knoise = 10;
    std::vector<float> ps(2 * kvol), pt(2 * kvol);
    std::vector<double2> slice(kvol);
    double pbp[knoise];
    int iter = 0;
    double2* xi = h->X2;
    double2* Phi = h->R;
    for (int inoise = 0; inoise < knoise; inoise++) {
        h->rng.gauss0(kvol, ps.data());                                   // :1061
        h->rng.gauss0(kvol, pt.data());                                   // :1063
        double p1r = 0.0, p1i = 0.0, p2r = 0.0, p2i = 0.0;
        for (int idsource = 1; idsource <= 2; idsource++) {
            for (int w = 0; w < 2; w++) {
                const float* nz = w == 0 ? ps.data() : pt.data();
                int dn, dsrc;
                double sgn = 1.0;
                if (imass != 5) {
                    dn = w == 0 ? idsource : idsource + 2;
                    dsrc = dn;
                } else {
                    dn = w == 0 ? idsource + 2 : idsource;
                    dsrc = w == 0 ? dn - 2 : dn + 2;
                    sgn = -1.0;
                }
                const int s_src = w == 0 ? 0 : Ls - 1;
                cudaMemcpyAsync(h->gauss, nz, sizeof(float) * 2 * kvol, cudaMemcpyHostToDevice, h->st);
                chdwf::k_thr_wall_source<<<chdwf::tblk(n), chdwf::kThreads, 0, h->st>>>(
                    xi, h->gauss, s_src, dsrc - 1, sgn, g);
                chdwf::count_launches(1);
                thr_dslash(h, true, am, imass, Phi, xi, u);               // :1136, :1220
                int it = 0;
                const int rc = thr_congrad(h, Phi, res, &it, am, imass, u, xi);   // :1138, :1225
                if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
                iter += it;
                const int s_rd = imass != 5 ? (w == 0 ? Ls - 1 : 0) : s_src;
                chdwf::k_thr_slice<<<chdwf::tblk(kvol), chdwf::kThreads, 0, h->st>>>(xi, s_rd, dn - 1,
                                                                                 g, h->X1);
                chdwf::count_launches(1);
                cudaMemcpyAsync(slice.data(), h->X1, sizeof(double2) * kvol, cudaMemcpyDeviceToHost,
                                h->st);
                const cudaError_t e = cudaStreamSynchronize(h->st);
                if (e) return h->fail(e, "thr_measure");
                double ar = w == 0 ? p1r : p2r, ai = w == 0 ? p1i : p2i;
                for (int64_t i = 0; i < kvol; i++) {                      // conjg(x)*xi, in order
                    const double xr = (double)nz[i], xim = (double)nz[kvol + i];
                    const double yr = slice[i].x, yi = slice[i].y;
                    ar = ar + (xr * yr - (-xim) * yi);
                    ai = ai + (xr * yi + (-xim) * yr);
                }
                if (w == 0) { p1r = ar; p1i = ai; } else { p2r = ar; p2i = ai; }
            }
        }
        const double kv = (double)kvol;
        if (imass == 1) {                                                 // :1245-1257
            p1r = p1r / kv; p1i = p1i / kv; p2r = p2r / kv; p2i = p2i / kv;
        } else {
            // (0,-1)*p1 ; (0,+1)*p2 (imass 3) or (0,-1)*p2 (imass 5), as complex products
            const double s2 = imass == 3 ? 1.0 : -1.0;
            const double a1 = 0.0 * p1r - (-1.0) * p1i, b1 = 0.0 * p1i + (-1.0) * p1r;
            const double a2 = 0.0 * p2r - s2 * p2i, b2 = 0.0 * p2i + s2 * p2r;
            p1r = a1 / kv; p1i = b1 / kv; p2r = a2 / kv; p2i = b2 / kv;
        }
        pbp[inoise] = p1r + p2r;
        if (parts) {
            parts[4 * inoise] = p1r; parts[4 * inoise + 1] = p1i;
            parts[4 * inoise + 2] = p2r; parts[4 * inoise + 3] = p2i;
        }
    }
    float pb = 0.0f, sus = 0.0f;                                          // :1266-1276
    for (int i = 0; i < knoise; i++) {
        pb = (float)((double)pb + pbp[i]);
        for (int j = knoise - 1; j >= i + 1; j--) sus = (float)((double)sus + pbp[i] * pbp[j]);
    }
    *psibarpsi = pb / (float)knoise;
    *susclsing = (float)(2 * kvol) * sus / (float)(knoise * (knoise - 1));
    *aviter = (float)iter / (float)(4 * knoise);                          // :1278
    return CHDWF_OK;
}

chdwf_thr* thr_ok(chdwf_thr* h) {
    if (h) cudaSetDevice(h->device);
    return h;
}

int thr_apply(chdwf_thr* h, bool dag, double* Phi, const double* R, const double* u, float am,
              int imass) {
    if (!thr_ok(h) || !Phi || !R || !u || (imass != 1 && imass != 3 && imass != 5))
        return CHDWF_BAD_ARG;
    const int64_t n = h->g.kferm;
    cudaMemcpyAsync(h->R, R, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->uio, u, sizeof(double2) * 3 * h->g.kvol, cudaMemcpyHostToDevice, h->st);
    thr_dslash(h, dag, am, imass, h->X2, h->R, h->uio);
    cudaMemcpyAsync(Phi, h->X2, sizeof(double2) * n, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_dslash") : CHDWF_OK;
}

}  // namespace

extern "C" {

int chdwf_thr_create(chdwf_thr** out, int ksize, int ksizet, int kthird, float dt, float beta,
                     float am3, float am, int imass, int iterl, int device) {
    if (!out) return CHDWF_BAD_ARG;
    *out = nullptr;
    if (!chdwf::geom_ok(ksize, ksizet, kthird) || (imass != 1 && imass != 3 && imass != 5) ||
        iterl < 1) {
        g_thr_create_err = "chdwf_thr_create: bad lattice, imass or iterl";
        return CHDWF_BAD_ARG;
    }
    chdwf_thr* h = new chdwf_thr;
    h->device = device;
    h->g.L = ksize; h->g.Lt = ksizet; h->g.Ls = kthird;
    h->g.kvol = ksize * ksize * ksizet;
    h->g.kferm = 4 * (int64_t)h->g.kvol * kthird;
    h->dt = dt; h->beta = beta; h->am3 = am3; h->am = am; h->imass = imass; h->iterl = iterl;
    const int64_t n3 = 3 * (int64_t)h->g.kvol, n = h->g.kferm;
    const int np = chdwf::kThrMaxPoles;
    cudaError_t e = cudaSetDevice(device);
    if (!e) e = cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking);
    if (!e) e = talloc(&h->theta, n3);
    if (!e) e = talloc(&h->thetat, n3);
    if (!e) e = talloc(&h->pp, n3);
    if (!e) e = talloc(&h->dS, n3);
    if (!e) e = talloc(&h->gauss, 8 * (size_t)h->g.kvol * kthird);
    if (!e) e = talloc(&h->ut, n3);
    if (!e) e = talloc(&h->uio, n3);
    for (double2** v : {&h->Phi, &h->X1, &h->R, &h->X2, &h->vt, &h->rr})
        if (!e) e = talloc(v, n);
    if (!e) e = talloc(&h->Phi0, n * np);
    if (!e) e = talloc(&h->p, n * np);
    if (!e) e = talloc(&h->x1, n * np);
    if (!e) e = talloc(&h->part, 3 * chdwf::kRedBlocks);
    if (!e) e = talloc(&h->qctl, 1);
    if (!e) e = talloc(&h->cgctl, 1);
    if (!e) e = cudaHostAlloc((void**)&h->hflag_host, sizeof(int), cudaHostAllocMapped);
    if (!e) e = cudaHostGetDevicePointer((void**)&h->hflag_dev, h->hflag_host, 0);
    size_t fr = 0, tot = 0;
    if (!e) e = cudaMemGetInfo(&fr, &tot);
    if (!e) h->chunk = chdwf::thr_chunk(sizeof(double2) * n, fr);
    if (!e) e = talloc(&h->ring, n * h->chunk);
    if (!e) e = cudaMemsetAsync(h->theta, 0, sizeof(float) * n3, h->st);
    if (!e) e = cudaMemsetAsync(h->Phi0, 0, sizeof(double2) * n * np, h->st);
    if (!e) e = cudaStreamSynchronize(h->st);
    if (e) {
        g_thr_create_err = std::string("chdwf_thr_create: ") + cudaGetErrorString(e);
        chdwf_thr_destroy(h);
        return CHDWF_CUDA_ERROR;
    }
    h->hpart.resize(chdwf::kRedBlocks);
    h->rng.startup((double)693764523745.0f);
    *out = h;
    return CHDWF_OK;
}

void chdwf_thr_destroy(chdwf_thr* h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->st) cudaStreamSynchronize(h->st);
    for (float* v : {h->theta, h->thetat, h->pp, h->dS, h->gauss}) if (v) cudaFree(v);
    for (double2* v : {h->ut, h->uio, h->Phi, h->X1, h->R, h->X2, h->Phi0, h->ring, h->vt,
                       h->rr, h->p, h->x1})
        if (v) cudaFree(v);
    h->graphs.release();
    if (h->part) cudaFree(h->part);
    if (h->qctl) cudaFree(h->qctl);
    if (h->cgctl) cudaFree(h->cgctl);
    if (h->hflag_host) cudaFreeHost(h->hflag_host);
    if (h->st) cudaStreamDestroy(h->st);
    delete h;
}

const char* chdwf_thr_last_error(chdwf_thr* h) {
    return h ? h->err.c_str() : g_thr_create_err.c_str();
}

int chdwf_thr_set_remez(chdwf_thr* h, int which, const double* anum, const double* aden,
                        const double* bnum, const double* bden, int ndiag) {
    if (!h || !anum || !aden || !bnum || !bden || ndiag < 1 || ndiag > chdwf::kThrMaxPoles)
        return CHDWF_BAD_ARG;
    ThrRemez* r = which == 2 ? &h->r2 : which == 4 ? &h->r4 : which == 22 ? &h->r2g
                : which == 44 ? &h->r4g : nullptr;
    if (!r) return CHDWF_BAD_ARG;
    r->anum.assign(anum, anum + ndiag + 1);
    r->aden.assign(aden, aden + ndiag);
    r->bnum.assign(bnum, bnum + ndiag + 1);
    r->bden.assign(bden, bden + ndiag);
    r->n = ndiag;
    return CHDWF_OK;
}

int chdwf_thr_coef(chdwf_thr* h, const float* theta, double* u) {
    if (!thr_ok(h) || !theta || !u) return CHDWF_BAD_ARG;
    const int64_t n3 = 3 * (int64_t)h->g.kvol;
    cudaMemcpyAsync(h->dS, theta, sizeof(float) * n3, cudaMemcpyHostToDevice, h->st);
    chdwf::k_thr_coef<<<chdwf::tblk(n3), chdwf::kThreads, 0, h->st>>>(h->dS, h->uio, h->g);
    chdwf::count_launches(1);
    cudaMemcpyAsync(u, h->uio, sizeof(double2) * n3, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_coef") : CHDWF_OK;
}

int chdwf_thr_dslash(chdwf_thr* h, double* Phi, const double* R, const double* u, float am,
                     int imass) {
    return thr_apply(h, false, Phi, R, u, am, imass);
}

int chdwf_thr_dslashd(chdwf_thr* h, double* Phi, const double* R, const double* u, float am,
                      int imass) {
    return thr_apply(h, true, Phi, R, u, am, imass);
}

int chdwf_thr_derivs(chdwf_thr* h, const double* R, const double* X2, double anum, int iflag,
                     float* dSdpi) {
    if (!thr_ok(h) || !R || !X2 || !dSdpi || (iflag != 0 && iflag != 1)) return CHDWF_BAD_ARG;
    const int64_t n = h->g.kferm, n3 = 3 * (int64_t)h->g.kvol;
    cudaMemcpyAsync(h->R, R, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->X1, X2, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->dS, dSdpi, sizeof(float) * n3, cudaMemcpyHostToDevice, h->st);
    thr_derivs(h, h->R, h->X1, anum, iflag);
    cudaMemcpyAsync(dSdpi, h->dS, sizeof(float) * n3, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_derivs") : CHDWF_OK;
}

int chdwf_thr_qmrherm(chdwf_thr* h, const double* Phi, float res, int* itercg, float am,
                      int imass, const double* anum, const double* aden, int ndiag, int iflag,
                      const double* u, double* x, double* Phi0, float* dSdpi) {
    if (!thr_ok(h) || !Phi || !itercg || !anum || !aden || !u || !x ||
        ndiag < 1 || ndiag > chdwf::kThrMaxPoles || iflag < 0 || iflag > 3 ||
        (imass != 1 && imass != 3 && imass != 5) || (iflag >= 1 && !Phi0) ||
        (iflag >= 2 && !dSdpi))
        return CHDWF_BAD_ARG;
    const int64_t n = h->g.kferm, n3 = 3 * (int64_t)h->g.kvol;
    cudaMemcpyAsync(h->Phi, Phi, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->uio, u, sizeof(double2) * n3, cudaMemcpyHostToDevice, h->st);
    if (iflag == 3)
        cudaMemcpyAsync(h->Phi0, Phi0, sizeof(double2) * n * ndiag, cudaMemcpyHostToDevice, h->st);
    if (iflag >= 2) cudaMemcpyAsync(h->dS, dSdpi, sizeof(float) * n3, cudaMemcpyHostToDevice, h->st);
    const int rc = thr_qmrherm(h, h->Phi, res, itercg, am, imass, anum, aden, ndiag, iflag, h->uio,
                               h->X1);
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    cudaMemcpyAsync(x, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToHost, h->st);
    if (iflag == 1)
        cudaMemcpyAsync(Phi0, h->Phi0, sizeof(double2) * n * ndiag, cudaMemcpyDeviceToHost, h->st);
    if (iflag >= 2) cudaMemcpyAsync(dSdpi, h->dS, sizeof(float) * n3, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    if (e) return h->fail(e, "thr_qmrherm");
    return rc;
}

int chdwf_thr_congrad(chdwf_thr* h, const double* Phi, float res, int* itercg, float am,
                      int imass, const double* u, double* x) {
    if (!thr_ok(h) || !Phi || !itercg || !u || !x || (imass != 1 && imass != 3 && imass != 5))
        return CHDWF_BAD_ARG;
    const int64_t n = h->g.kferm;
    cudaMemcpyAsync(h->R, Phi, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->X2, x, sizeof(double2) * n, cudaMemcpyHostToDevice, h->st);
    cudaMemcpyAsync(h->uio, u, sizeof(double2) * 3 * h->g.kvol, cudaMemcpyHostToDevice, h->st);
    const int rc = thr_congrad(h, h->R, res, itercg, am, imass, h->uio, h->X2);
    if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc;
    cudaMemcpyAsync(x, h->X2, sizeof(double2) * n, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_congrad") : rc;
}

int chdwf_thr_measure(chdwf_thr* h, float res, const double* u, float* psibarpsi,
                      float* susclsing, float* aviter, double* parts) {
    if (!thr_ok(h) || !u || !psibarpsi || !susclsing || !aviter) return CHDWF_BAD_ARG;
    cudaMemcpyAsync(h->uio, u, sizeof(double2) * 3 * h->g.kvol, cudaMemcpyHostToDevice, h->st);
    return thr_measure(h, res, h->am, h->imass, h->uio, psibarpsi, susclsing, aviter, parts);
}

int chdwf_thr_set_measure(chdwf_thr* h, int iprint) {
    if (!h || iprint < 1) return CHDWF_BAD_ARG;
    h->iprint = iprint;
    return CHDWF_OK;
}

int chdwf_thr_set_theta(chdwf_thr* h, const float* theta) {
    if (!thr_ok(h) || !theta) return CHDWF_BAD_ARG;
    cudaMemcpyAsync(h->theta, theta, sizeof(float) * 3 * h->g.kvol, cudaMemcpyHostToDevice, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_set_theta") : CHDWF_OK;
}

int chdwf_thr_get_theta(chdwf_thr* h, float* theta) {
    if (!thr_ok(h) || !theta) return CHDWF_BAD_ARG;
    cudaMemcpyAsync(theta, h->theta, sizeof(float) * 3 * h->g.kvol, cudaMemcpyDeviceToHost, h->st);
    const cudaError_t e = cudaStreamSynchronize(h->st);
    return e ? h->fail(e, "thr_get_theta") : CHDWF_OK;
}

int chdwf_thr_startup(chdwf_thr* h, double seed) {
    if (!h) return CHDWF_BAD_ARG;
    h->rng.startup(seed);
    return CHDWF_OK;
}

double chdwf_thr_seed(chdwf_thr* h) { return h ? h->rng.seed() : 0.0; }

int chdwf_thr_sweep(chdwf_thr* h, chdwf_thr_record* rec) {
    if (!thr_ok(h) || !rec) return CHDWF_BAD_ARG;
    if (h->r2.n < 1 || h->r4.n < 1 || h->r2g.n < 1 || h->r4g.n < 1) {
        h->err = "thr_sweep: set remez2, remez4, remez2g and remez4g first";
        return CHDWF_BAD_ARG;
    }
    memset(rec, 0, sizeof(*rec));
    const TGeom& g = h->g;
    const int64_t kvol = g.kvol, n = g.kferm, n3 = 3 * kvol;
    const unsigned nb3 = chdwf::tblk(n3);
    int rc;
#define CK(x) do { rc = (x); if (rc != CHDWF_OK && rc != CHDWF_ITER_CAP) return rc; } while (0)
#define CKC(x, w) do { cudaError_t e_ = (x); if (e_) return h->fail(e_, w); } while (0)
    h->isweep++;
    cudaMemcpyAsync(h->thetat, h->theta, sizeof(float) * n3, cudaMemcpyDeviceToDevice, h->st);  // :203-208
    chdwf::k_thr_coef<<<nb3, chdwf::kThreads, 0, h->st>>>(h->thetat, h->ut, g);
    chdwf::count_launches(1);
    std::vector<float> gauss(8 * (size_t)kvol * g.Ls);                    // :213-222
    for (int c = 0; c < 4 * g.Ls; c++) h->rng.gauss0(kvol, gauss.data() + (size_t)c * 2 * kvol);
    CKC(cudaMemcpyAsync(h->gauss, gauss.data(), sizeof(float) * gauss.size(),
                        cudaMemcpyHostToDevice, h->st), "thr_sweep");
    chdwf::k_thr_noise<<<chdwf::tblk(n), chdwf::kThreads, 0, h->st>>>(h->R, h->gauss, g);
    chdwf::count_launches(1);
    CK(thr_qmrherm(h, h->R, h->rescga, &rec->it_pf, h->am, h->imass, h->r4.anum.data(),
                   h->r4.aden.data(), h->r4.n, 0, h->ut, h->X1));          // :226
    cudaMemcpyAsync(h->R, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    CK(thr_qmrherm(h, h->R, h->rescga, &rec->it_pfpv, 1.0f, 1, h->r4.bnum.data(),
                   h->r4.bden.data(), h->r4.n, 0, h->ut, h->X1));          // :236
    cudaMemcpyAsync(h->Phi, h->X1, sizeof(double2) * n, cudaMemcpyDeviceToDevice, h->st);
    std::vector<float> ps(2 * kvol), pp(n3);                               // :255-260
    for (int mu = 0; mu < 3; mu++) {
        h->rng.gaussp(kvol, ps.data());
        memcpy(pp.data() + kvol * mu, ps.data(), sizeof(float) * kvol);
    }
    CKC(cudaMemcpyAsync(h->pp, pp.data(), sizeof(float) * n3, cudaMemcpyHostToDevice, h->st),
        "thr_sweep");
    double hh[4];
    int ih[2];
    CK(thr_hamilton(h, h->rescga, hh, ih));                               // :265
    rec->it_h0 = ih[0];
    rec->it_h0pv = ih[1];
    rec->H0 = hh[0];
    rec->S0 = hh[3];
    if (h->isweep == 1) {                                                  // :267-271
        h->action = (float)(hh[3] / (double)kvol);
        h->gaction = (float)(hh[1] / (double)kvol);
        h->paction = (float)(hh[2] / (double)kvol);
    }
    int fi[4];
    CK(thr_force(h, h->rescgg, fi));                                      // :276
    for (int k = 0; k < 4; k++) rec->it_force[k] += fi[k];
    rec->nforce++;
    float d = h->dt * 0.5f;
    chdwf::k_thr_update_p<<<nb3, chdwf::kThreads, 0, h->st>>>(h->pp, h->dS, d, n3);
    chdwf::count_launches(1);
    const float proby = 1.0f / (float)h->iterl;                           // :151
    for (int iter = 1; iter <= 1000; iter++) {                            // :285-320
        d = h->dt;
        chdwf::k_thr_update_theta<<<nb3, chdwf::kThreads, 0, h->st>>>(h->thetat, h->pp, d, n3);
        chdwf::k_thr_coef<<<nb3, chdwf::kThreads, 0, h->st>>>(h->thetat, h->ut, g);
        chdwf::count_launches(2);
        CK(thr_force(h, h->rescgg, fi));
        for (int k = 0; k < 4; k++) rec->it_force[k] += fi[k];
        rec->nforce++;
        rec->nsteps = iter;
        const float ytest = h->rng.rano_yran();                            // :302
        if (ytest < proby) {
            d = h->dt * 0.5f;
            chdwf::k_thr_update_p<<<nb3, chdwf::kThreads, 0, h->st>>>(h->pp, h->dS, d, n3);
            chdwf::count_launches(1);
            h->itot = h->itot + iter;
            break;
        }
        d = h->dt;
        chdwf::k_thr_update_p<<<nb3, chdwf::kThreads, 0, h->st>>>(h->pp, h->dS, d, n3);
        chdwf::count_launches(1);
    }
    CK(thr_hamilton(h, h->rescga, hh, ih));                               // :325
    rec->it_h1 = ih[0];
    rec->it_h1pv = ih[1];
    rec->H1 = hh[0];
    rec->S1 = hh[3];
    rec->hg = hh[1];
    rec->hp = hh[2];
    rec->dH = rec->H0 - rec->H1;
    rec->dS = rec->S0 - rec->S1;
    rec->y = (float)std::exp(rec->dH);                                    // :330
    h->yav = h->yav + rec->y;
    h->yyav = h->yyav + rec->y * rec->y;
    int accept = 1;
    if (rec->dH < 0.0) {                                                  // :333-336
        rec->x = h->rng.rano_yran();
        rec->drew_x = 1;
        if (rec->x > rec->y) accept = 0;
    }
    if (accept) {                                                         // :338-348
        cudaMemcpyAsync(h->theta, h->thetat, sizeof(float) * n3, cudaMemcpyDeviceToDevice, h->st);
        h->naccp = h->naccp + 1;
        h->action = (float)(rec->S1 / (double)kvol);
        h->gaction = (float)(rec->hg / (double)kvol);
        h->paction = (float)(rec->hp / (double)kvol);
    }
    rec->accepted = accept;
    rec->action = h->action;
    rec->gaction = h->gaction;
    rec->paction = h->paction;
    h->actiona = h->actiona + h->action;                                  // :350
    CKC(cudaMemcpyAsync(pp.data(), h->pp, sizeof(float) * n3, cudaMemcpyDeviceToHost, h->st),
        "thr_sweep");
    CKC(cudaStreamSynchronize(h->st), "thr_sweep");
    float vel2 = 0.0f;                                                    // :351-357
    for (int64_t j = 0; j < n3; j++) vel2 = vel2 + pp[j] * pp[j];
    rec->vel2 = vel2 / (float)(3 * kvol);
    h->vel2a = h->vel2a + rec->vel2;
    if ((h->isweep / h->iprint) * h->iprint == h->isweep) {               // :361-371
        cudaMemcpyAsync(h->thetat, h->theta, sizeof(float) * n3, cudaMemcpyDeviceToDevice, h->st);
        chdwf::k_thr_coef<<<nb3, chdwf::kThreads, 0, h->st>>>(h->thetat, h->ut, g);
        chdwf::count_launches(1);
        float sus = 0.0f;
        CK(thr_measure(h, h->respbp, h->am, h->imass, h->ut, &rec->pbp, &sus, &rec->ancgm,
                       nullptr));
        rec->measured = 1;
    }
    CKC(cudaGetLastError(), "thr_sweep");
#undef CK
#undef CKC
    return CHDWF_OK;
}

}  // extern "C"
