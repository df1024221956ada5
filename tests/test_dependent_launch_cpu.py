"""Dependent launches: what a kernel reads that another kernel of the stream may still be writing when it starts."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "ug_b200", "csrc")
# written once, by calls whose kernels are no dependent launches: weights, rotation tables
FIXED = {"embed", "alpha", "cos_", "sin_", "bz", "bu", "q_gain", "c_gain", "table"}


def _kernels():
    """(file, name, parameters, body) of every kernel that waits for its predecessor itself."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for k in re.finditer(r"__global__[^;{]*?(\w+)\(([^(){};]*)\)\s*\{", src, re.S):
            depth, end = 1, k.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            if "ugb_pdl_wait" in src[k.end():end]:
                yield f, k.group(1), k.group(2), src[k.end():end]


KERNELS = list(_kernels())


def test_all_kinds_are_seen():
    names = {k[1] for k in KERNELS}
    assert {"f32_tile_kernel", "f32_skinny_kernel", "f32_skinny_n_kernel", "short_k_kernel", "skinny_gemm_kernel", "tc_gemm_kernel", "row_reg_kernel", "row_general_kernel",
            "row_update_kernel", "reduce_rmsnorm_kernel", "argmax_rows_kernel", "expert_rows_kernel"} <= names


@pytest.mark.parametrize("f,name,params,body", KERNELS, ids=[k[1] for k in KERNELS])
def test_no_noncoherent_reads_of_what_a_predecessor_writes(f, name, params, body):
    """const __restrict__ parameters and __ldg are ld.global.nc, which is defined for memory that nothing writes as long as the
    kernel lives; a dependent launch lives while its predecessor still writes."""
    loose = {p.split()[-1].lstrip("*") for p in params.split(",") if "__restrict__" in p and p.strip().startswith("const")} - FIXED
    assert not loose, f"{f}: {name} reads {sorted(loose)} without coherence"
    if f in ("matmul.cu", "rowops.cu"):           # operands of public calls: nothing is fixed
        assert "__ldg" not in body and "ld.global.nc" not in body


def test_matrix_that_a_kernel_may_write_is_read_coherently():
    src = open(os.path.join(CSRC, "gemm_skinny.cu")).read()
    load = src[src.index("ld_stream(const void *p)"):]
    fixed, ordinary = load[:load.index("return v;")].split("else", 1)
    assert "if constexpr (FIXED)" in fixed and ".nc" in fixed and ".nc" not in ordinary
    for launch in re.findall(r"skinny_gemm_kernel<([^>]*)>", src):
        if launch.split(",")[1].strip() == "true":        # f16: public calls only
            assert launch.split(",")[2].strip() == "false"


def test_few_rows_read_ahead_on_late_triggers_only():
    """A decode step of few rows lets kernels read ahead of their wait whatever its projections run on: no path of gemm_rows may
    take the late trigger back."""
    src = open(os.path.join(CSRC, "llama_engine.cu")).read()
    body = src[src.index("int32_t gemm_rows("):src.index("int32_t gemm(ugb_llama")]
    assert "late_trigger = true" in body and "late_trigger = false" not in body


def test_f32_products_of_an_engine_follow_its_option():
    """pdl = 0 means ordinary launches for the f32 products of a layer-list model too."""
    engine, products = (open(os.path.join(CSRC, f)).read() for f in ("hybrid_engine.cu", "matmul.cu"))
    call = engine[engine.index("ugb_f32_gemm("):]
    assert "m->pdl != 0" in call[:call.index(";")]
    gemm = products[products.index("int32_t ugb_f32_gemm("):products.index('extern "C" {')]
    assert gemm.count("pdl") >= 3 and "true)" not in re.sub(r"R\{[^}]*\}", "", gemm)
    launches = re.findall(r"ugb_launch(?:_cluster)?\(([^;]*?)\)[;\n]", products)
    assert len(launches) >= 4 and all("dev->stream, pdl," in l for l in launches)
