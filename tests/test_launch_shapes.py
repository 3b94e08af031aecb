"""Default launch shapes over the whole range of sizes, from the library's own rule
compiled for the host: the force pass's item list stays within about a million
items (its count is an int), and sizes below that keep the chunk their costs give."""
import subprocess

import pytest

import build as engine_build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "kernels.h"
int main(int argc, char **argv) {  // slots, atoms, points per atom
    const long long slots = atoll(argv[1]), n = atoll(argv[2]), P = n * atoll(argv[3]);
    auto items = [&](long long C) { return (n + 127) / 128 * ((P + C - 1) / C); };
    const int C = isspa::default_chunk(slots, items);
    std::printf("%d %lld\n", C, items(C));
}
"""

SLOTS = 152 * 8  # resident force blocks of the chip


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("shapes")
    src, exe = d / "shapes.cu", d / "shapes"
    src.write_text(PROGRAM)
    subprocess.run([engine_build.nvcc()] + engine_build._flags() + [str(src), "-o", str(exe)], check=True)
    return lambda *a: tuple(map(int, subprocess.run([str(exe)] + [str(x) for x in a], check=True, capture_output=True,
                                                    text=True).stdout.split()))


@pytest.mark.parametrize("atoms, n_mc, chunk", [(1, 1, 32), (44, 20, 32), (264, 50, 32), (741, 50, 48), (1100, 50, 64),
                                                (4400, 50, 256), (8800, 100, 256), (16384, 100, 256)])
def test_chunk_by_cost(rule, atoms, n_mc, chunk):
    assert rule(SLOTS, atoms, n_mc)[0] == chunk


@pytest.mark.parametrize("atoms, n_mc", [(18542, 100), (66000, 100), (264000, 50), (1000000, 100), (2000000, 1000)])
def test_list_is_bounded(rule, atoms, n_mc):
    chunk, items = rule(SLOTS, atoms, n_mc)
    assert chunk >= 256 and items <= 1 << 20
