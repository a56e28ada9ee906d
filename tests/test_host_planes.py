"""CPU check of the site-fastest stencil (csrc/planes.cuh) against the
point-wise operator, without a GPU.

plane_item is compiled for the host with stand-ins for the device intrinsics
and run for every work item and thread of several launch plans:
  * every unit of the output is produced exactly once;
  * FP64: the same bits as dwf_apply_flavour, both directions, both mass
    terms, both time boundaries, with the pinning term;
  * FP32 pairs: an element is a sum of at most 16 rounded terms of magnitude
    at most 4 max|R| (hops, projections, diagonal 3 R, walls |chi| <= 4), so
    it lies within 16 * 2^-24 * 32 max|R| of the FP64 value of the same
    inputs; the unused half of the last unit of an odd Ls is zero.
"""
import subprocess

import pytest

from test_host_kernels import CSRC, RHMC_PROGRAM, _build

PLANES_PROGRAM = RHMC_PROGRAM.split('#include "dwf_stencil.cuh"')[0] + r"""
#include <cmath>
#include <algorithm>
static inline int __any_sync(unsigned, int p) { return p; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
#include "planes.cuh"
using namespace chdwf;
static bool skip;
static int block;
struct Ld { const double2* p; double2 operator()(int64_t j) const { return p[j]; } };
template <class V> struct Store {
    V* out; int* hits;
    bool operator()(V* acc, int64_t e, int64_t cst, uint32_t o, bool act, int, uint32_t) {
        if (!act) return true;
        for (int d = 0; d < 4; d++) {
            V* p = unit_at(out + e + d * cst, o);
            *p = acc[d];
            hits[p - out]++;
        }
        return true;
    }
};
template <bool DAG, int IMASS, class V, class Real>
void sweep(const std::vector<V>& in, std::vector<V>& out, std::vector<int>& hits, const PlanePlan& pl,
           const float* chif, Real diag, Real hpin, bool apbc) {
    Store<V> st{out.data(), hits.data()};
    for (uint32_t it = 0; it < pl.nitem; it++)
        for (int t = 0; t < pl.threads; t++) {
            threadIdx.x = t;
            if (skip) plane_item<DAG, IMASS, true, true>(in.data(), pl, plane_thread(pl), it, chif, diag, hpin, apbc, st);
            else plane_item<DAG, IMASS>(in.data(), pl, plane_thread(pl), it, chif, diag, hpin, apbc, st);
        }
}
template <class V, class Real, class F>
void all(const std::vector<V>& in, const PlanePlan& pl, const float* chif, Real diag, Real hpin, F&& check) {
    for (int apbc = 0; apbc < 2; apbc++)
        for (int dag = 0; dag < 2; dag++)
            for (int imass = 1; imass <= 3; imass += 2) {
                std::vector<V> out(in.size());
                std::vector<int> hits(in.size(), 0);
                if (dag) { if (imass == 1) sweep<true, 1>(in, out, hits, pl, chif, diag, hpin, apbc); else sweep<true, 3>(in, out, hits, pl, chif, diag, hpin, apbc); }
                else { if (imass == 1) sweep<false, 1>(in, out, hits, pl, chif, diag, hpin, apbc); else sweep<false, 3>(in, out, hits, pl, chif, diag, hpin, apbc); }
                for (int h : hits) if (h != 1) { printf("hits %d\n", h); exit(0); }
                check(out, dag, imass, apbc);
            }
}
int main(int argc, char** argv) {
    const int L = atoi(argv[1]), Lt = atoi(argv[2]), Ls = atoi(argv[3]), nsm = atoi(argv[4]);
    block = atoi(argv[5]);
    skip = block != 256;
    const Geom g = make_geom(L, Lt, Ls);
    std::vector<double2> R(g.kferm), ref(g.kferm);
    std::vector<float> chif(3 * g.kvol);
    srand(7);
    auto rnd = [] { return (double)(float)(2.0 * rand() / RAND_MAX - 1.0); };
    for (auto& v : R) v = make_double2(rnd(), rnd());
    for (auto& v : chif) v = (float)(4.0 * rnd());
    const double diag = 6.0, hpin = (double)0.3f;
    auto reference = [&](int dag, int imass, int apbc) {
        const Ld ld{R.data()};
        for (int64_t p = 0; p < g.npts; p++) {
            const PointIdx q = point_of(g, p);
            for (int fl = 0; fl < 2; fl++) {
                double2 acc[4];
                if (dag) { if (imass == 1) dwf_apply_flavour<true, 1>(acc, ld, g, q, fl, chif.data(), diag, hpin, apbc); else dwf_apply_flavour<true, 3>(acc, ld, g, q, fl, chif.data(), diag, hpin, apbc); }
                else { if (imass == 1) dwf_apply_flavour<false, 1>(acc, ld, g, q, fl, chif.data(), diag, hpin, apbc); else dwf_apply_flavour<false, 3>(acc, ld, g, q, fl, chif.data(), diag, hpin, apbc); }
                for (int d = 0; d < 4; d++) ref[p + g.cs * (d + 4 * fl)] = acc[d];
            }
        }
    };
    long long bad = 0;
    double worst = 0.0;
    {
        const PlanePlan pl = plane_plan(g, false, nsm, block);
        std::vector<double2> in(plane_elems<double2>(g));
        auto at = [&](int c, int s, int site) { return ((int64_t)c * pl.U + s) * g.kvol + site; };
        for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < Ls; s++)
            in[at(c, s, i)] = R[s + (int64_t)Ls * i + g.cs * c];
        all<double2, double>(in, pl, chif.data(), diag, hpin, [&](std::vector<double2>& out, int dag, int imass, int apbc) {
            reference(dag, imass, apbc);
            for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < Ls; s++) {
                const double2 a = out[at(c, s, i)], b = ref[s + (int64_t)Ls * i + g.cs * c];
                if (a.x != b.x || a.y != b.y) bad++;
            }
        });
    }
    {
        const PlanePlan pl = plane_plan(g, true, nsm, block);
        std::vector<cpair> in(plane_elems<float2>(g) / 2);
        auto half = [&](std::vector<cpair>& v, int c, int s, int site, bool im) -> float& {
            cpair& p = v[((int64_t)c * pl.U + s / 2) * g.kvol + site];
            float2& h = im ? p.im : p.re;
            return s & 1 ? h.y : h.x;
        };
        for (auto& p : in) p = cpair{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < Ls; s++) {
            const double2 v = R[s + (int64_t)Ls * i + g.cs * c];
            half(in, c, s, i, false) = (float)v.x;
            half(in, c, s, i, true) = (float)v.y;
        }
        all<cpair, float>(in, pl, chif.data(), (float)diag, (float)hpin, [&](std::vector<cpair>& out, int dag, int imass, int apbc) {
            reference(dag, imass, apbc);
            for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < Ls; s++) {
                const double2 b = ref[s + (int64_t)Ls * i + g.cs * c];
                worst = std::max(worst, std::max(fabs(half(out, c, s, i, false) - b.x), fabs(half(out, c, s, i, true) - b.y)));
            }
            if (Ls & 1) for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++)
                if (half(out, c, Ls, i, false) != 0.f || half(out, c, Ls, i, true) != 0.f) bad++;
        });
    }
    printf("%lld %.9g\n", bad, worst);
    return 0;
}
"""


@pytest.fixture(scope="module")
def planes_exe(tmp_path_factory):
    return _build(str(tmp_path_factory.mktemp("planes")), "planes", PLANES_PROGRAM,
                  extra=["-I", CSRC])


# nsm steers the plan: many SMs give small tiles and short runs, one SM large ones
@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (2, 2, 2), (3, 5, 3), (5, 4, 7), (6, 3, 5),
                                     (67, 2, 2), (9, 7, 2)])
# block: 256 threads, the multi-shift solver's, and 192, the conjugate gradients',
# whose warps without a site leave at once
@pytest.mark.parametrize("nsm", [1, 148])
@pytest.mark.parametrize("block", [256, 192])
def test_plane_stencil_matches_point_operator(planes_exe, L, Lt, Ls, nsm, block):
    out = subprocess.run([planes_exe, *map(str, (L, Lt, Ls, nsm, block))], check=True,
                         capture_output=True, text=True).stdout
    bad, worst = out.split()
    assert int(bad) == 0, out
    assert float(worst) <= 16 * 2.0 ** -24 * 32, out
