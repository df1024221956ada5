"""Which shape a product runs on (csrc/gemm_plan.h is host arithmetic): the sizes of the GPU tests reach the shapes they are there for."""
import os
import subprocess

import pytest

from conftest import ROOT
from test_f32_tile_gpu import TURNED
from test_llama_prefill_gpu import SPLIT_PROMPT
from test_tc_shapes_gpu import SHAPES

SMS = 148


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    """ask("tc", m, n, k, kn, pairs, max_splits) -> (bn, pair, splits); ask("f32", b, m, n, k) -> (wm, wk, split, turned)"""
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text("""
#include "gemm_plan.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
int main(int argc, char **argv) {
  size_t a[6];
  for (int i = 0; i < 6; ++i) a[i] = i + 2 < argc ? strtoull(argv[i + 2], nullptr, 10) : 0;
  if (!strcmp(argv[1], "tc")) {
    const ugb_tc_plan p = ugb_tc_gemm_plan(%d, 1, a[0], a[1], a[2], !a[3], a[4] != 0, (int)a[5]);
    printf("%%d %%d %%d", p.bn, p.pair ? 1 : 0, p.splits);
  } else {
    const ugb_f32_shape s = ugb_f32_gemm_shape(%d, a[0], a[1], a[2], a[3]);
    printf("%%d %%d %%d %%d", s.wm, s.wk, s.split, s.turned ? 1 : 0);
  }
}
""" % (SMS, SMS))
    exe = str(d / "plan")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "ug_b200", "csrc"), str(d / "plan.cpp"), "-o", exe], check=True)
    return lambda *q: tuple(int(x) for x in subprocess.run([exe] + [str(int(x) if not isinstance(x, str) else x) for x in q], check=True, capture_output=True,
                                                           text=True).stdout.split())


@pytest.mark.parametrize("case", list(SHAPES))
def test_tensor_core_shapes(ask, case):
    m, n, k, kn = case
    assert ask("tc", m, n, k, kn, 1, 1)[:2] == (SHAPES[case][0], int(SHAPES[case][1]))
    assert ask("tc", m, n, k, kn, 0, 1)[1] == 0


def test_every_shape_is_reached():
    assert set(SHAPES.values()) == {(64, False), (128, False), (192, False), (256, False), (128, True), (192, True), (256, True)}


def test_prompt_that_splits_k(ask):
    cfg, rows, splits = SPLIT_PROMPT
    h, f = cfg["hidden_size"], cfg["intermediate_size"]
    for cap, (o, down) in splits.items():
        assert (ask("tc", rows, h, h, 0, 1, cap)[2], ask("tc", rows, h, f, 0, 1, cap)[2]) == (o, down)
    # with or without pairs decides over a split only where the planner is asked without them
    assert ask("tc", 2310, 2048, 5632, 0, 1, 3)[2] == 1 and ask("tc", 2310, 2048, 5632, 0, 0, 3)[2] == 2


@pytest.mark.parametrize("m,n,k", TURNED)
def test_few_columns_are_turned(ask, m, n, k):
    assert ask("f32", 1, m, n, k)[3] == 1


def test_turned_in_both_tile_heights(ask):
    assert {ask("f32", 1, *c)[0] for c in TURNED} == {1, 2}
