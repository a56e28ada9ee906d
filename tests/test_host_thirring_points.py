"""CPU check of the bulk Thirring solver's operator, which forms the four Dirac
components of a point together (thr_point of csrc/thirring.cu), against the
element-wise operator, compiled for the host with stand-ins for the device
intrinsics.  The two add the same at most 16 terms of an element in a different
order and with fused multiply-adds; with |R|, |u| <= 1.5 each partial sum is
below 40, so they differ by at most 3 roundings a term: 48 * 2^-53 * 40."""
import os
import subprocess

import pytest

from test_host_kernels import CSRC, PRELUDE, ZOPS, _build, _hostify, _section

MAIN = r"""
template <bool DAG, int IMASS>
double check(const TGeom& g, const std::vector<double2>& R, const std::vector<double2>& u) {
    double worst = 0.0;
    const double2 zk = IMASS == 1 ? make_double2(0.3, 0.0) : make_double2(0.0, DAG ? 0.3 : -0.3);
    for (int i = 0; i < g.kvol; i++) for (int s = 0; s < g.Ls; s++) {
        double2 phi[4];
        thr_point<DAG, IMASS>(phi, R.data(), u.data(), g, s, i, 3.0, zk);
        for (int d = 0; d < 4; d++) {
            const double2 v = thr_element<DAG, IMASS>(R.data(), u.data(), g, s, i, d, 3.0, zk);
            worst = std::max(worst, std::max(fabs(phi[d].x - v.x), fabs(phi[d].y - v.y)));
        }
    }
    return worst;
}
int main(int argc, char** argv) {
    TGeom g;
    g.L = atoi(argv[1]); g.Lt = atoi(argv[2]); g.Ls = atoi(argv[3]);
    g.kvol = g.L * g.L * g.Lt;
    g.kferm = 4 * (int64_t)g.kvol * g.Ls;
    std::vector<double2> R(g.kferm), u(3 * g.kvol);
    srand(5);
    auto rnd = [] { return 2.0 * rand() / RAND_MAX - 1.0; };
    for (auto& v : R) v = make_double2(rnd(), rnd());
    for (auto& v : u) v = make_double2(1.0, rnd());
    double w = std::max(check<false, 1>(g, R, u), check<true, 1>(g, R, u));
    w = std::max(w, std::max(check<false, 3>(g, R, u), check<true, 3>(g, R, u)));
    w = std::max(w, std::max(check<false, 5>(g, R, u), check<true, 5>(g, R, u)));
    printf("%.6e\n", w);
    return 0;
}
"""


@pytest.fixture(scope="module")
def points_exe(tmp_path_factory):
    src = open(os.path.join(CSRC, "thirring.cu")).read()
    body = _section(src, "struct TGeom {", "// ---- multi-shift solver kernels")
    body += _section(src, "__device__ __forceinline__ double2 zfma", "__device__ __forceinline__ double znorm2")
    code = PRELUDE + "#include <cmath>\n#include <algorithm>\n" + ZOPS + \
        "static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }\n" + \
        "namespace X {\n" + _hostify(body) + "}\nusing namespace X;\n" + MAIN
    return _build(str(tmp_path_factory.mktemp("thrp")), "thrp", code)


@pytest.mark.parametrize("shape", [(2, 2, 2), (4, 4, 4), (3, 2, 5), (2, 6, 3)])
def test_thirring_point_matches_elements(points_exe, shape):
    out = subprocess.run([points_exe, *map(str, shape)], check=True, capture_output=True,
                         text=True).stdout
    assert float(out) <= 48 * 2.0 ** -53 * 40, out
