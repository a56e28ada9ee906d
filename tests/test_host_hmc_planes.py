"""CPU check of the HMC predecessor's operator on planes
(csrc/hmc_planes.cuh) against its element-wise form, without a GPU: both are
compiled for the host with stand-ins for the device intrinsics; every unit of
the output is formed exactly once and has the value of the element-wise form
bit for bit (zeros may differ in sign), both directions and mass terms, with
and without the antiperiodic correction."""
import os
import subprocess

import pytest

from test_host_kernels import CSRC, RHMC_PROGRAM, _build, _hostify, _section

MAIN = r"""
struct Store {
    float2* out; int* hits;
    bool operator()(float2* acc, int64_t e, int64_t cst, uint32_t o, bool act, int, uint32_t) {
        if (!act) return true;
        for (int d = 0; d < 4; d++) {
            float2* p = unit_at(out + e + d * cst, o);
            *p = acc[d];
            hits[p - out]++;
        }
        return true;
    }
};
template <bool DAG, int IMASS>
long long check(const Geom& g, const std::vector<float2>& R, const std::vector<float2>& in,
                const std::vector<float>& chi, int nsm, int block) {
    const PlanePlan pl = plane_plan(g, false, nsm, block);
    long long bad = 0;
    for (int apbc = 0; apbc < 2; apbc++) {
        std::vector<float2> out(in.size());
        std::vector<int> hits(in.size(), 0);
        Store st{out.data(), hits.data()};
        for (uint32_t it = 0; it < pl.nitem; it++)
            for (int t = 0; t < pl.threads; t++) {
                threadIdx.x = t;
                hmc_plane_item<DAG, IMASS>(in.data(), pl, plane_thread(pl), it, chi.data(), 3.0f,
                                           apbc != 0, st);
            }
        for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < g.Ls; s++) {
            const int x = i % g.L, y = i / g.L % g.L, t = i / (g.L * g.L);
            const float2 a = hmc_element<DAG, IMASS>(R.data(), g, s, x, y, t, c & 3, c >> 2,
                                                     chi.data(), 3.0f, apbc != 0);
            const int64_t u = ((int64_t)c * g.Ls + s) * g.kvol + i;
            if (hits[u] != 1 || !(out[u].x == a.x) || !(out[u].y == a.y)) bad++;
        }
    }
    return bad;
}
int main(int argc, char** argv) {
    const int L = atoi(argv[1]), Lt = atoi(argv[2]), Ls = atoi(argv[3]), nsm = atoi(argv[4]);
    const Geom g = make_geom(L, Lt, Ls);
    std::vector<float2> R(g.kferm), in(g.kferm);
    std::vector<float> chi(3 * g.kvol);
    srand(11);
    auto rnd = [] { return (float)(2.0 * rand() / RAND_MAX - 1.0); };
    for (auto& v : R) v = make_float2(rnd(), rnd());
    for (auto& v : chi) v = rnd();
    for (int c = 0; c < 8; c++) for (int i = 0; i < g.kvol; i++) for (int s = 0; s < Ls; s++)
        in[((int64_t)c * Ls + s) * g.kvol + i] = R[s + (int64_t)Ls * i + g.cs * c];
    printf("%lld\n", check<false, 1>(g, R, in, chi, nsm, 192) + check<true, 1>(g, R, in, chi, nsm, 192) +
                     check<false, 3>(g, R, in, chi, nsm, 192) + check<true, 3>(g, R, in, chi, nsm, 192));
    return 0;
}
"""


@pytest.fixture(scope="module")
def hmc_planes_exe(tmp_path_factory):
    src = open(os.path.join(CSRC, "hmc.cu")).read()
    body = _section(src, "// ---- REAL*4 complex arithmetic",
                    "template <bool DAG, int IMASS>\n__global__ void __launch_bounds__(kThreads) k_hmc_dslash")
    code = RHMC_PROGRAM.split('#include "dwf_stencil.cuh"')[0] + r"""
#include <cmath>
static inline int __any_sync(unsigned, int p) { return p; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
#include "planes.cuh"
namespace chdwf {
""" + _hostify(body) + '}\n#include "hmc_planes.cuh"\nusing namespace chdwf;\n' + MAIN
    return _build(str(tmp_path_factory.mktemp("hmcp")), "hmcp", code, extra=["-I", CSRC])


@pytest.mark.parametrize("L,Lt,Ls", [(4, 4, 4), (2, 2, 2), (3, 5, 3), (5, 4, 7), (67, 2, 2)])
@pytest.mark.parametrize("nsm", [1, 148])
def test_hmc_plane_operator_matches_elements(hmc_planes_exe, L, Lt, Ls, nsm):
    out = subprocess.run([hmc_planes_exe, *map(str, (L, Lt, Ls, nsm))], check=True,
                         capture_output=True, text=True).stdout
    assert int(out) == 0, out
