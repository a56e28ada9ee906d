"""How many iterations' vectors a Thirring handle keeps (thr_chunk of
csrc/thirring.cu): up to 16, an even number, at least the two that the solvers need,
and beyond those never more than a quarter of the free memory, so that a program's
other handles and buffers keep their place."""
import os
import subprocess

from test_host_kernels import CSRC, _build, _section

MAIN = r"""
int main() {
    int bad = 0;
    for (size_t v = 1024; v < (size_t)1 << 36; v = v * 3 / 2)
        for (size_t f = 0; f < (size_t)1 << 38; f = f * 5 / 4 + 4096) {
            const int c = thr_chunk(v, f);
            if (c < 2 || c > 16 || c % 2) bad++;
            if (c > 2 && v * c > f / 4) bad++;
            if (c < 16 && 2 * v * c <= f / 4) bad++;
        }
    printf("%d\n", bad);
    return 0;
}
"""


def test_chunk_leaves_memory(tmp_path):
    src = open(os.path.join(CSRC, "thirring.cu")).read()
    body = _section(src, "constexpr int kThrChunk", "struct ThrQCtl {")
    exe = _build(str(tmp_path), "chunk", "#include <cstddef>\n#include <cstdio>\n" + body + MAIN)
    assert int(subprocess.run([exe], check=True, capture_output=True, text=True).stdout) == 0
    # taken last, when everything else has its memory
    create = src[src.index("int chdwf_thr_create("):]
    create = create[:create.index("*out = h;")]
    assert create.rindex("talloc(") == create.index("talloc(&h->ring")
