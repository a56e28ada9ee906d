"""CPU check of how the operator kernels on the ABI's spinors (csrc/dslash.cu)
read memory, without a GPU.

They are launched with programmatic serialisation: a kernel may be resident
while the one before it, M in front of M^dagger say, still writes the vector
that it will read.  Non-coherent loads (__ldg, or const __restrict__ parameters)
need data that nobody writes for as long as the kernel runs, and the compiler
may move them in front of the wait.  So every kernel that launch_op launches
takes plain pointers, and none of its loads goes through __ldg: the kernels are
compiled for the host with an __ldg that counts, and run for every block and
thread.  Their output shows that they ran: FP64 has the oracle's bits; FP32 lies
within 16 * 2^-24 * 32 max|R| of it (as many rounded terms of that size an
element, |chi| <= 4), and FP16 storage, inputs exact in FP16, within that and
the rounding of a result of at most 32 max|R| to 11 bits."""
import os
import re
import subprocess

import numpy as np
import pytest

import pyoracle as po
from test_host_kernels import CSRC, RHMC_PROGRAM, _build, _section

MAIN = r"""
template <class F> void grid(unsigned nb, unsigned nt, F&& f) {
    for (unsigned b = 0; b < nb; b++)
        for (unsigned t = 0; t < nt; t++) { blockIdx.x = b; threadIdx.x = t; f(); }
}
int main(int argc, char** argv) {
    const int L = atoi(argv[1]), Lt = atoi(argv[2]), Ls = atoi(argv[3]);
    const Geom g = make_geom(L, Lt, Ls);
    std::vector<double2> R(g.kferm), o64(g.kferm);
    std::vector<float2> R32(g.kferm), o32(g.kferm);
    std::vector<__half2> R16(g.kferm), o16(g.kferm);
    std::vector<double> chi(3 * g.kvol);
    FILE* f = fopen(argv[4], "rb");
    if (fread(R.data(), 16, g.kferm, f) != (size_t)g.kferm) return 1;
    if (fread(chi.data(), 8, 3 * g.kvol, f) != (size_t)(3 * g.kvol)) return 1;
    fclose(f);
    for (int64_t i = 0; i < g.kferm; i++) {
        R32[i] = make_float2((float)R[i].x, (float)R[i].y);
        R16[i] = __float22half2_rn(R32[i]);
    }
    f = fopen(argv[5], "wb");
    constexpr unsigned kThreads = 256;
    blockDim.x = kThreads;
    const unsigned nl = (unsigned)((g.npts + kThreads - 1) / kThreads);
#define RUN(D, I)                                                                              \
    {                                                                                          \
        grid(op_blocks(g.npts, 1), kOpThreads, [&] {                                           \
            k_dslash64<D, I, 6>(o64.data(), R.data(), chi.data(), g, 6.0, 0.25, 1); });        \
        fwrite(o64.data(), 16, g.kferm, f);                                                    \
        grid(nl, kThreads, [&] {                                                               \
            k_dslash_lp<D, I, 0>(o32.data(), R32.data(), chi.data(), g, 6.0f, 0.25f, 1); });   \
        fwrite(o32.data(), 8, g.kferm, f);                                                     \
        if (Ls % 2 == 0)                                                                       \
            grid(op_blocks(g.npts, 2), kOpThreads, [&] {                                       \
                k_dslash_f32_pair<D, I, 6>(o32.data(), R32.data(), chi.data(), g, 6.0f, 0.25f, 1); }); \
        fwrite(o32.data(), 8, g.kferm, f);                                                     \
        grid(nl, kThreads, [&] {                                                               \
            k_dslash_lp<D, I, 1>(o16.data(), R16.data(), chi.data(), g, 6.0f, 0.25f, 1); });   \
        fwrite(o16.data(), 4, g.kferm, f);                                                     \
        if (Ls % 4 == 0)                                                                       \
            grid(op_blocks(g.npts, 4), kOpThreads, [&] {                                       \
                k_dslash_quad<D, I, __half2>(o16.data(), R16.data(), chi.data(), g, 6.0f, 0.25f, 1); }); \
        fwrite(o16.data(), 4, g.kferm, f);                                                     \
    }
    RUN(false, 1) RUN(true, 1) RUN(false, 3) RUN(true, 3)
    fclose(f);
    printf("%lld\n", n_ldg);
    return 0;
}
"""


def _source():
    return open(os.path.join(CSRC, "dslash.cu")).read()


@pytest.fixture(scope="module")
def op_exe(tmp_path_factory):
    src = _source()
    body = _section(src, "struct LdF64 {", "template <class... P, class... A>")
    body += _section(src, "struct LdF32 {", "void launch_dslash_lp(")
    body = re.sub(r"__global__ void __launch_bounds__\([^)]*\)", "void", body)
    body = re.sub(r"asm volatile\([^;]*;\"[^;]*;", ";", body)          # prefetches
    head = RHMC_PROGRAM.split("int main")[0].replace(
        "template <class T> static inline T __ldg(const T* p) { return *p; }",
        "static long long n_ldg;\n"
        "template <class T> static inline T __ldg(const T* p) { n_ldg++; return *p; }")
    head = head.replace("#include <cuda_runtime.h>", "#include <cuda_runtime.h>\n#include <cuda_fp16.h>")
    code = head + "static void pdl_wait() {}\nnamespace chdwf {\n" + body + "}\n" + MAIN
    return _build(str(tmp_path_factory.mktemp("op")), "op", code, extra=["-I", CSRC])


def test_programmatic_kernels_take_plain_pointers():
    src = _source()
    launched = set(re.findall(r"\b(k_dslash\w+)<D, I", src))
    assert {"k_dslash64", "k_dslash_lp", "k_dslash_f32_pair", "k_dslash_quad"} <= launched
    for k in launched:
        head = re.search(r"\b%s\(([^)]*)\)\s*\{\s*(\S+)" % k, src)
        assert "__restrict__" not in head.group(1), k
        assert head.group(2) == "pdl_wait();", k


@pytest.mark.parametrize("shape", [(4, 4, 4), (3, 2, 5), (2, 5, 2), (5, 3, 8)])
def test_operator_kernels_load_coherently(op_exe, tmp_path, shape):
    L, Lt, Ls = shape
    lat = po.make_lat(L, Lt, Ls, am3=1.0)
    rng = np.random.default_rng(L * 100 + Lt * 10 + Ls)
    sh = po.spinor_shape(lat)
    R = (rng.standard_normal(sh).astype(np.float16).astype(np.float64)
         + 1j * rng.standard_normal(sh).astype(np.float16).astype(np.float64))
    chi = np.clip(rng.standard_normal((3, L * L * Lt)), -4, 4)
    fin, fout = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    with open(fin, "wb") as f:
        f.write(R.tobytes())
        f.write(chi.tobytes())
    out = subprocess.run([op_exe, str(L), str(Lt), str(Ls), fin, fout], check=True,
                         capture_output=True, text=True).stdout
    raw, off = open(fout, "rb").read(), 0

    def take(dt):
        nonlocal off
        v = np.frombuffer(raw, dtype=dt, count=2 * R.size, offset=off).astype(np.float64)
        off += v.size * np.dtype(dt).itemsize
        return v.view(np.complex128).reshape(sh)

    big = 32 * np.abs(R).max()
    for imass in (1, 3):
        for dag in (False, True):
            ref = po.dslash(lat, R, chi, hpin=0.25, imass=imass, dag=dag)
            assert np.array_equal(take(np.float64), ref)
            for _ in range(2):
                assert np.abs(take(np.float32) - ref).max() <= 16 * 2.0 ** -24 * big
            for _ in range(2):
                assert np.abs(take(np.float16) - ref).max() <= (16 * 2.0 ** -24 + 2.0 ** -11) * big
    assert off == len(raw)
    assert int(out) == 0, "loads through the non-coherent path"
