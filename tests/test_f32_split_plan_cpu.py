"""Which f32 products run on the tensor cores (csrc/gemm_plan.h is host arithmetic)."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_f32_split_gpu import CHAINS, SHAPES
from test_f32_tile_gpu import FFMA, FFMA_KM

SMS = 148


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    """plan(b, m, n, k, rows_contiguous) -> (rows of a tile, CTAs along k; 0, 1: the FFMA kernel), (wm, wk, split, turned) of that kernel"""
    d = tmp_path_factory.mktemp("split")
    (d / "plan.cpp").write_text("""
#include "gemm_plan.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **v) {
  const size_t b = strtoull(v[1], 0, 10), m = strtoull(v[2], 0, 10), n = strtoull(v[3], 0, 10), k = strtoull(v[4], 0, 10);
  const ugb_f32_split_plan p = ugb_f32_gemm_split_plan(%d, b, m, n, k, v[5][0] == '1');
  const ugb_f32_shape s = ugb_f32_gemm_shape(%d, b, m, n, k);
  printf("%%d %%d %%d %%d %%d %%d", p.bn, p.split, s.wm, s.wk, s.split, s.turned ? 1 : 0);
}
""" % (SMS, SMS))
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "ug_b200", "csrc"), str(d / "plan.cpp"), "-o", exe], check=True)

    def f(*q):
        x = tuple(int(x) for x in subprocess.run([exe] + [str(int(x)) for x in q], check=True, capture_output=True, text=True).stdout.split())
        return x[:2], x[2:]
    return f


@pytest.fixture
def ask(plan):
    return lambda *q: plan(*q)[0]


@pytest.mark.parametrize("case", list(SHAPES))
def test_tested_sizes_reach_their_tiles(ask, case):
    assert ask(*case, 0) == SHAPES[case]
    bn, split = ask(*case, 1)
    assert bn in (0, 64) and split in (1, 2, 4, 8)


@pytest.mark.parametrize("case", [(1, 257, 5632, 2048), (1, 128, 2048, 2048)])
def test_single_values_with_contiguous_rows_reach_the_tensor_cores(ask, case):
    assert ask(*case, 1)[0] != 0


@pytest.mark.parametrize("case", list(FFMA) + list(FFMA_KM))
def test_what_stays_on_the_ffma_kernel(plan, case):
    """The sizes of test_f32_tile_gpu.py reach the instances of the FFMA kernel that f32 products still run on."""
    for rows_contiguous in (0, 1) if case in FFMA else (1,):
        assert plan(*case, rows_contiguous) == ((0, 1), (FFMA | FFMA_KM)[case])


def test_every_instance_of_the_ffma_kernel_is_reached():
    shapes, whole = FFMA | FFMA_KM, lambda c: c[1] % 4 == c[2] % 4 == c[3] % 4 == 0
    for vec in (True, False):              # operands in 16-byte pieces, or value by value
        assert {(s[0], s[1], s[3]) for c, s in shapes.items() if whole(c) == vec} == {(4, 1, 0), (2, 2, 0), (1, 4, 0), (2, 2, 1), (1, 4, 1)}


def test_every_tile_and_cluster_is_reached():
    assert {s[0] for s in SHAPES.values()} == {32, 64, 96} and {s[1] for s in SHAPES.values()} == {1, 2, 4, 8}


def test_short_k_and_next_to_nothing_stay_where_they_were(ask):
    assert ask(1, 4932, 132, 99, 0)[0] == 0 and ask(1, 4096, 4096, 16, 1)[0] == 0 and ask(1, 4932, 132, 100, 0)[0] != 0
    assert ask(1, 0, 5, 100, 0)[0] == 0 and ask(5, 3922, 8, 408, 0)[0] == 0 and ask(5, 3922, 33, 408, 0)[0] != 0


@pytest.mark.parametrize("case", list(CHAINS))
def test_chains_beside_which_errors_are_held(plan, case):
    (bn, split), (wm, wk, cluster, _) = plan(*case, 0)
    assert CHAINS[case] == wk * cluster and case[3] >= 100 * wk * cluster


def test_short_chains_stay_with_ffma(plan):
    for case in ((1, 128, 2048, 760), (1, 17, 5632, 2048), (1, 70, 3000, 300)):
        (bn, _), (_, wk, cluster, _) = plan(*case, 0)
        assert bn == 0, case
