"""Which f32 products run on the tensor cores (csrc/gemm_plan.h is host arithmetic)."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_f32_split_gpu import SHAPES

SMS = 148


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    """ask(b, m, n, k, rows_contiguous) -> (rows of a tile, CTAs along k); (0, 1): the FFMA kernel"""
    d = tmp_path_factory.mktemp("split")
    (d / "plan.cpp").write_text("""
#include "gemm_plan.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **v) {
  const ugb_f32_split_plan p = ugb_f32_gemm_split_plan(%d, strtoull(v[1], 0, 10), strtoull(v[2], 0, 10), strtoull(v[3], 0, 10), strtoull(v[4], 0, 10), v[5][0] == '1');
  printf("%%d %%d", p.bn, p.split);
}
""" % SMS)
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "ug_b200", "csrc"), str(d / "plan.cpp"), "-o", exe], check=True)
    return lambda *q: tuple(int(x) for x in subprocess.run([exe] + [str(int(x)) for x in q], check=True, capture_output=True, text=True).stdout.split())


@pytest.mark.parametrize("case", list(SHAPES))
def test_tested_sizes_reach_their_tiles(ask, case):
    assert ask(*case, 0) == SHAPES[case]
    bn, split = ask(*case, 1)
    assert bn in (0, 64, 128) and split in (1, 2, 4, 8)


def test_every_tile_and_cluster_is_reached():
    assert {s[0] for s in SHAPES.values()} == {32, 64, 96, 128} and {s[1] for s in SHAPES.values()} == {1, 2, 4, 8}


def test_short_k_and_next_to_nothing_stay_where_they_were(ask):
    assert ask(1, 4096, 4096, 63, 0)[0] == 0 and ask(1, 4096, 4096, 16, 1)[0] == 0
    assert ask(1, 0, 5, 100, 0)[0] == 0 and ask(5, 3922, 8, 88, 0)[0] == 0 and ask(5, 3922, 33, 88, 0)[0] != 0
