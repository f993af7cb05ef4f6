"""Launch shapes of the rebuild kernels up to the largest particle count that a context accepts (2^30), and of
the k-space tables up to theirs."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mfa_brush_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "mfa_grid.h"
int main() {
  for (long long n : {1ll, 16ll, 17ll, 6400ll, 1ll << 20, (1ll << 28) - 1, 1ll << 28, 1ll << 29, 1ll << 30})
    std::printf("%lld %d %d\n", n, mfa::sort_blocks(n, 152), mfa::list_blocks(n, 152));
}
"""


def test_blocks_cover_the_particles_or_fill_the_gpu(tmp_path):
    src = tmp_path / "grid.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "grid")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    for line in out.splitlines():
        n, sort, lists = map(int, line.split())
        assert sort == min(-(-n // 512), 2 * 152)
        assert lists == min(-(-8 * n // 128), 8 * 152)


TABLES = r"""
#include <cstdio>
#include "mfa_grid.h"
int main() {
  for (long long nq : {1ll, 257ll, 13760ll, 16600000ll, 25000000ll, 33000000ll, 40000000ll})
    std::printf("%lld %d\n", nq, mfa::table_blocks(nq, 130));
}
"""


def test_blocks_cover_the_tables(tmp_path):
    src = tmp_path / "tables.cpp"
    src.write_text(TABLES)
    exe = str(tmp_path / "tables")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    for line in out.splitlines():
        nq, blocks = map(int, line.split())
        assert blocks == (-(-130 * nq // 256) if 130 * nq < 2 ** 32 - 256 else -1)
