"""16-bit products of more than 64 rows at sizes for which each tile shape of the tensor-core kernel is chosen (128- and 256-row
tiles, 64 to 256 columns), ragged in every direction; few rows, few results and sizes that no tensor-core kernel takes."""
import numpy as np
import pytest

from ug_b200 import synth

pytestmark = pytest.mark.gpu


# (m, n, k, kn): the shape that a device of 148 SMs runs the product on, columns and whether on pairs of CTAs
# (test_gemm_plan_cpu.py holds the rule to this)
SHAPES = {
    (100, 2040, 200, False): (64, False), (129, 2056, 520, True): (64, False), (300, 2048, 2048, False): (64, False),
    (65, 72, 64, False): (128, False), (100, 11256, 2040, False): (128, False), (777, 2056, 2040, False): (128, False), (500, 2560, 1000, True): (128, False),
    (2040, 2056, 264, False): (128, False),
    (777, 11256, 520, False): (192, False), (200, 11264, 2056, True): (192, False), (1023, 2552, 2048, False): (192, False),
    (300, 11264, 2040, False): (256, False),
    (1023, 2040, 5640, False): (128, True), (511, 11256, 2040, False): (192, True), (1500, 2040, 5632, False): (192, True), (2047, 2048, 2048, True): (256, True)}


@pytest.mark.parametrize("m,n,k,kn", list(SHAPES))
def test_shapes(dev, m, n, k, kn):
    ab, wb = synth.to_bf16_bits(synth.normal(m, (m, k), 0.5)), synth.to_bf16_bits(synth.normal(n, (k, n) if kn else (n, k), 0.5))
    guard = 64
    out = dev.slice_from_values(synth.to_bf16_bits(np.full(m * n + guard, 3.0, np.float32)), bf16=True)
    dev.matmul(out, dev.slice_from_values(ab.ravel(), bf16=True), dev.slice_from_values(wb.ravel(), bf16=True), (1, m, n, k),
               ([1, m, k], [m * k, k, 1], 0), ([1, k, n], [n * k, n, 1] if kn else [n * k, 1, k], 0))
    got = synth.bf16_bits_to_f32(out.to_vec())
    assert np.all(got[m * n:] == 3.0)
    rows = np.unique(np.r_[np.arange(0, m, 37), m - 1, min(m - 1, 127), min(m - 1, 128), min(m - 1, 255), min(m - 1, 256)])
    a = synth.bf16_bits_to_f32(ab)[rows].astype(np.float64)
    w = synth.bf16_bits_to_f32(wb).astype(np.float64)
    w = w if kn else w.T
    # one rounding of the result (to nearest: at most 2^-8 of it) plus f32 sums of k products
    assert np.all(np.abs(got[:m * n].reshape(m, n)[rows] - a @ w) <= np.abs(a @ w) * 2.0 ** -8 + np.abs(a) @ np.abs(w) * k * 2.0 ** -24 + 1e-6)


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("b,m,n,k,kn", [(1, 14, 520, 2048, False), (3, 9, 136, 264, True), (2, 4, 128, 880, True), (1, 1, 9, 7, True), (1, 15, 4096, 520, True),   # few rows
                                        (1, 1, 8, 8, True), (1, 9, 8, 8, False), (2, 24, 64, 192, False), (3, 65, 8, 16, True), (64, 20, 24, 40, False), (1, 8, 8192, 16, False),  # few results
                                        (1, 37, 333, 777, True), (2, 100, 255, 129, False), (1, 130, 129, 1001, False), (1, 3, 8, 2, True),
                                        (3, 65, 67, 1, True), (1, 200, 129, 15, False), (2, 63, 64, 13, True), (1, 8, 20000, 16, False),   # one slice of k
                                        (1, 20001, 17, 67, True), (2, 1500, 3, 999, False), (1, 2601, 36, 1001, True)])                   # no 16-byte rows
def test_few_rows_and_odd_sizes(dev, b, m, n, k, kn, f16):
    def bits(x):
        return x.astype(np.float16) if f16 else synth.to_bf16_bits(x)

    def wide(x):
        return x.astype(np.float64) if f16 else synth.bf16_bits_to_f32(x).astype(np.float64)
    ab, wb = bits(synth.normal(m, (b, m, k), 0.5)), bits(synth.normal(n, (b, k, n) if kn else (b, n, k), 0.5))
    out = dev.slice_from_values(bits(np.full(b * m * n + 64, 3.0, np.float32)), bf16=not f16)
    dev.matmul(out, dev.slice_from_values(ab.ravel(), bf16=not f16), dev.slice_from_values(wb.ravel(), bf16=not f16), (b, m, n, k),
               ([b, m, k], [m * k, k, 1], 0), ([b, k, n], [n * k, n, 1] if kn else [n * k, 1, k], 0))
    got = wide(out.to_vec())
    assert np.all(got[b * m * n:] == 3.0)
    a, w = wide(ab), wide(wb) if kn else wide(wb).transpose(0, 2, 1)
    # one rounding of the result (to nearest: at most 2^-11 of it in f16, 2^-8 in bf16) plus f32 sums of k products
    assert np.all(np.abs(got[:b * m * n].reshape(b, m, n) - a @ w) <= np.abs(a @ w) * 2.0 ** (-11 if f16 else -8) + np.abs(a) @ np.abs(w) * k * 2.0 ** -24 + 1e-6)
