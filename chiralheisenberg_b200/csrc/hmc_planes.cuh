// hmc_planes.cuh -- the operator of the HMC predecessor (mh/cheisdwf_hmc.f:
// 1334-2028) on planes (planes.cuh), for its conjugate gradients.  Included by
// hmc.cu behind its REAL*4 arithmetic and wall coupling.
//
// A unit is one element (8 bytes); a thread forms all four Dirac components,
// so a neighbour is loaded once for the Wilson and the Dirac terms
// (hmc_element, one element a thread, loads 20 elements for each).  Every
// element still receives its updates in the order of the reference's sweeps:
// diagonal, three Wilson terms, their antiperiodic correction, three Dirac
// terms, their correction, the s hop, the walls.  The differences of the x and
// y neighbours wait in registers for the Wilson terms to end; the t neighbours
// come last, so their corrections take them from registers too.  (With two s a
// thread, as the other FP32 solvers have them, the waiting values do not fit:
// 340-440 bytes of spills at 128 registers.)
//
// The couplings are +-1/2 and +-1 (times i): such a product is exact, so the
// fused multiply-adds here round once, where the reference's product and sum
// do.
#pragma once
#include "planes.cuh"

namespace chdwf {

struct hmc32 {};                                       // kind of system, plane_cg.cuh
template <> struct unit_of<hmc32> { typedef float2 type; };
template <> struct real_of<hmc32> { typedef float type; };

__device__ __forceinline__ float2 ld_unit(const float2* p) { return *p; }
__device__ __forceinline__ void st_unit(float2* p, float2 v) { *p = v; }

namespace {

// a +- 0.5 * (i b if IM, else b)
template <bool IM>
__device__ __forceinline__ void hmc_half(float2& a, float2 b, int sign) {
    const float p = 0.5f * sign;
    a = IM ? make_float2(__fmaf_rn(-p, b.y, a.x), __fmaf_rn(p, b.x, a.y))
           : make_float2(__fmaf_rn(p, b.x, a.x), __fmaf_rn(p, b.y, a.y));
}
// a +- i b
__device__ __forceinline__ void hmc_unit(float2& a, float2 b, int sign) {
    const float2 r = make_float2(-b.y, b.x);
    a = sign > 0 ? fc_add(a, r) : fc_sub(a, r);
}

// Walls of the Dirac pair D0, D0+1 (group A: s = kthird, B: s = 1); o: the
// other wall's units of this site.
template <bool DAG, int IMASS, int D0, bool A>
__device__ __forceinline__ void hmc_plane_wall(float2 acc[4], const float2* o, int64_t cst, int f,
                                               float c1, float c2, float c3) {
#pragma unroll
    for (int d = D0; d < D0 + 2; d++) {
        const float2 r1 = ld_unit(o + cst * d), r2 = ld_unit(o + cst * (d + 4));
        acc[d] = hmc_wall<DAG, IMASS>(acc[d], A, f, f ? r2 : r1, f ? r1 : r2, c1, c2, c3);
    }
}

// As plane_item (planes.cuh), warps without a site skipped.
template <bool DAG, int IMASS, class Epi>
__device__ __forceinline__ void hmc_plane_item(const float2* in, const PlanePlan& pl,
                                               const PlaneThread& th, uint32_t item,
                                               const float* chif, float diag, bool apbc,
                                               Epi& epi) {
    typedef float2 V;
    constexpr int UP = DAG ? 0 : 2, DN = DAG ? 2 : 0;
    // signs of gamval(mu, d), negated for M^dagger
    constexpr int SG = DAG ? -1 : 1;
    constexpr int g0[4] = {-SG, -SG, SG, SG}, g12[4] = {-SG, SG, SG, -SG};
    const PlanePlace w = plane_place<true, sizeof(V)>(pl, th, item);
    if (w.none) return;
    const uint32_t kv = pl.kvol;
    const int U = pl.U;
    const int64_t cst = (int64_t)U * kv;
    int64_t e = 4 * w.f * cst + (int64_t)w.u0 * kv;
    const V *p0 = in + e, *p1 = p0 + cst, *p2 = p1 + cst, *p3 = p2 + cst;
#pragma unroll 1
    for (int u = w.u0; u < w.u1; u++, e += kv) {
        auto load = [&](V r[4], uint32_t o) {
            r[0] = ld_unit(unit_at(p0, o));
            r[1] = ld_unit(unit_at(p1, o));
            r[2] = ld_unit(unit_at(p2, o));
            r[3] = ld_unit(unit_at(p3, o));
        };
        V phi[4], up[4], dn[4], dx[4], dy[4];
        auto wilson = [&] {
#pragma unroll
            for (int d = 0; d < 4; d++) hmc_half<false>(phi[d], fc_add(up[d], dn[d]), -1);
        };
        load(phi, w.o_0);
#pragma unroll
        for (int d = 0; d < 4; d++) phi[d] = fc_scal(diag, phi[d]);          // :1351-1365
        load(up, w.o_xp);                                                   // :1367-1411
        load(dn, w.o_xm);
        wilson();
#pragma unroll
        for (int d = 0; d < 4; d++) dx[d] = fc_sub(up[d], dn[d]);
        load(up, w.o_yp);
        load(dn, w.o_ym);
        wilson();
#pragma unroll
        for (int d = 0; d < 4; d++) dy[d] = fc_sub(up[d], dn[d]);
        load(up, w.o_tp);
        load(dn, w.o_tm);
        wilson();
        if (apbc) {                                                         // :1412-1437
#pragma unroll
            for (int d = 0; d < 4; d++) {
                if (w.t == pl.Lt - 1) phi[d] = fc_add(phi[d], up[d]);
                if (w.t == 0) phi[d] = fc_add(phi[d], dn[d]);
            }
        }
#pragma unroll
        for (int d = 0; d < 4; d++) {                                       // :1438-1490
            hmc_half<true>(phi[d], dx[3 - d], g0[d]);
            hmc_half<false>(phi[d], dy[3 - d], g12[d]);
            hmc_half<true>(phi[d], fc_sub(up[d ^ 2], dn[d ^ 2]), g12[d]);
            if (apbc) {                                                     // :1491-1516
                if (w.t == pl.Lt - 1) hmc_unit(phi[d], up[d ^ 2], -g12[d]);
                if (w.t == 0) hmc_unit(phi[d], dn[d ^ 2], g12[d]);
            }
        }
        // s hops (:1518-1546, :1867-1895)
        if (u + 1 < U) {
            phi[UP] = fc_sub(phi[UP], ld_unit(unit_at((DAG ? p0 : p2) + kv, w.o_0)));
            phi[UP + 1] = fc_sub(phi[UP + 1], ld_unit(unit_at((DAG ? p1 : p3) + kv, w.o_0)));
        }
        if (u > 0) {
            phi[DN] = fc_sub(phi[DN], ld_unit(unit_at((DAG ? p2 : p0) - kv, w.o_0)));
            phi[DN + 1] = fc_sub(phi[DN + 1], ld_unit(unit_at((DAG ? p3 : p1) - kv, w.o_0)));
        }
        if (u == 0 || u == U - 1) {                                         // :1549-1679
            const float c1 = chif[w.site], c2 = chif[kv + w.site], c3 = chif[2 * kv + w.site];
            if (u == U - 1)
                hmc_plane_wall<DAG, IMASS, UP, true>(phi, in + w.site, cst, w.f, c1, c2, c3);
            if (u == 0)
                hmc_plane_wall<DAG, IMASS, DN, false>(phi, in + (int64_t)(U - 1) * kv + w.site, cst,
                                                      w.f, c1, c2, c3);
        }
        epi(phi, e, cst, w.o_0, w.act, u, w.site);
        p0 += kv; p1 += kv; p2 += kv; p3 += kv;
    }
}

}  // namespace
}  // namespace chdwf
