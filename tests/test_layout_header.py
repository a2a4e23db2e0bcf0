"""The layouts that test_xwarp_layout.py checks are those of the header: their positions as the CUDA compiler
evaluates them (a host program, no GPU)."""
import subprocess

from mpc_gb300 import build
from test_xwarp_layout import CFG

SRC = r"""
#include <cstdio>
#include "mpc_kernels.cuh"
template <int NX> void row() {
    using C = mpc::XWarp<NX>;
    printf("x %d %d", NX, C::RS);
    for (int p = 0; p < NX; p++) printf(" %d", C::idx(p));
    printf("\n");
}
int main() {
    row<128>(); row<256>(); row<512>();
    printf("plane %d", mpc::PlaneS::SIZE);
    for (int y = 0; y < mpc::PlaneS::N; y++) printf(" %d %d", mpc::PlaneS::at(y), mpc::PlaneS::idx(y));
    printf("\n");
}
"""


def test_positions_of_the_header(tmp_path):
    src, exe = tmp_path / "layout.cu", tmp_path / "layout"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-diag-suppress", "177", "-I", build.CSRC, str(src), "-o", str(exe)], check=True,
                   capture_output=True)
    lines = [ln.split() for ln in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert {int(ln[1]) for ln in lines[:3]} == set(CFG)
    for ln in lines[:3]:
        nx, rs, idx = int(ln[1]), int(ln[2]), [int(v) for v in ln[3:]]
        sh, pad, stride = CFG[nx]
        assert rs == stride and idx == [p + (p >> sh) * pad for p in range(nx)]
    v = [int(x) for x in lines[3][1:]]
    n, rstr = 64, 88
    assert v[0] == n * rstr + 4 * ((n - 1) >> 1) and len(v) == 1 + 2 * n
    for y in range(n):
        assert v[1 + 2 * y] == y * rstr + 4 * (y >> 1) and v[2 + 2 * y] == y + (y >> 2)
