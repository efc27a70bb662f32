"""The launch of the g(r) histogram (csrc/gofr_shape.h), compiled alone on the host: a block counts in 32-bit bins, so
the pairs of its items may not pass 2^32 - 1 (all of them can fall in one bin), and the blocks' shares are the items."""
import shutil
import subprocess

import pytest

from helpers import ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "gofr_shape.h"
int main(int, char **argv) {
  const long long n = atoll(argv[1]), slices = atoll(argv[2]);
  const pimc::GofrShape g = pimc::gofr_shape(n, slices, 148);
  long long most = 0, at = 0;
  bool whole = true;
  const long long step = g.blocks > 5000 ? g.blocks / 5000 : 1;
  for (long long b = 0; b < g.blocks; b += step) {
    const long long f = pimc::gofr_first(g.items, g.blocks, b), e = pimc::gofr_first(g.items, g.blocks, b + 1);
    whole = whole && (step > 1 || f == at) && e > f;
    at = e;
    most = e - f > most ? e - f : most;
  }
  whole = whole && pimc::gofr_first(g.items, g.blocks, 0) == 0 && pimc::gofr_first(g.items, g.blocks, g.blocks) == g.items;
  printf("%d %lld %d %lld %d\n", g.tile, g.items, g.blocks, most, whole ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("gofr")
    (d / "shape.cc").write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", f"{ROOT}/pimcplusplus_b200/csrc",
                    str(d / "shape.cc"), "-o", str(d / "shape")], check=True)

    def run(n, slices):
        out = subprocess.run([str(d / "shape"), str(n), str(slices)], capture_output=True, text=True, check=True)
        return [int(x) for x in out.stdout.split()]

    return run


@pytest.mark.parametrize("n,slices", [(1, 1), (2, 1), (33, 3), (64, 40), (512, 128), (4096, 256), (100000, 60),
                                      (262144, 75), (262144, 10000), (1 << 20, 3000), (1700000000, 1)])
def test_bins_hold_a_blocks_pairs(shape, n, slices):
    tile, items, blocks, most, whole = shape(n, slices)
    nt = (n + tile - 1) // tile
    assert items == nt * (nt + 1) // 2 * slices
    assert whole and 1 <= blocks < 2 ** 31
    assert most * tile * tile < 2 ** 32
    if items // (4 * 148) * tile * tile < 2 ** 31:  # ordinary sizes: one resident wave
        assert blocks == min(items, 4 * 148)
