"""The FP64 product's choice of tile and K split, on the host compiler: the partial products of a split
stay within the workspace that a stream may keep for them, small deep products are still split, and
every shape gets a tile whose modelled time is finite."""
from __future__ import annotations

import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "remora_b200" / "csrc"

PROGRAM = r"""
#include "gemm_plan.cuh"
#include <cstdio>
int main() {
    long long m, n, k;
    while (std::scanf("%lld %lld %lld", &m, &n, &k) == 3) {
        const rc::Problem p{m, n, k, false};
        rc::TileId id;
        int nz;
        rc::pick_tile(p, false, false, k >= 2048, 148, &id, &nz);
        const double cycles = id == rc::kTileM ? rc::tile_cycles<rc::TileM>(p, nz, 148)
                              : id == rc::kTileS ? rc::tile_cycles<rc::TileS>(p, nz, 148)
                                                 : rc::tile_cycles<rc::TileT>(p, nz, 148);
        std::printf("%d %d %.0f %.0f\n", (int)id, nz, rc::split_bytes(p, nz), cycles);
    }
}
"""


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "a.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(d / "a.cpp"), "-o",
                    str(d / "a.out")], check=True)

    def run(shapes):
        text = "".join("%d %d %d\n" % s for s in shapes)
        out = subprocess.run([str(d / "a.out")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


def test_split_workspace_is_bounded(pick):
    rng = random.Random(1)
    size = lambda lo, hi: int(lo * (hi / lo) ** rng.random())  # noqa: E731
    shapes = [(5000, 5000, 20000), (20000, 4000, 40000), (12246, 9876, 61089), (60000, 60000, 150000),
              (1, 1, 1 << 30), (1 << 24, 1, 4096)]
    shapes += [(size(1, 40000), size(1, 40000), size(2048, 200000)) for _ in range(3000)]
    got = pick(shapes)
    assert max(b for _, _, b, _ in got) <= 256 << 20
    assert all(1 <= nz <= 8 and cycles < 10 ** 15 for _, nz, _, cycles in got)


def test_small_deep_products_are_split_and_tall_ones_have_a_tile(pick):
    assert all(nz > 1 for _, nz, _, _ in pick([(64, 64, 8192), (130, 200, 4096), (1024, 64, 16384), (512, 512, 32768)]))
    assert all(nz == 1 and cycles < 10 ** 9
               for _, nz, _, cycles in pick([(4_200_001, 8, 8), (8_000_000, 16, 16), (100_000_000, 1, 1)]))
