"""f32 products on the tensor cores: edges of their tiles (128 columns of the result x 32 to 128 rows), of the 32-k stages, the pairs of
stages and the shares of a cluster, every layout of both operands, and values that three bf16 parts do not hold, against float64."""
import numpy as np
import pytest

from ug_b200 import DType, synth

pytestmark = pytest.mark.gpu
# (b, m, n, k) -> (rows of a tile, CTAs along k) on 148 SMs; test_f32_split_plan_cpu.py holds the rule to these
SHAPES = {(1, 257, 5632, 2048): (96, 1), (1, 128, 2048, 2048): (64, 4), (1, 120, 1352, 7144): (128, 8), (2, 526, 1080, 216): (96, 1), (1, 31, 8000, 128): (32, 1),
          (32, 128, 64, 64): (32, 1), (16, 300, 777, 400): (128, 1), (1, 33, 4000, 512): (64, 4), (1, 500, 1001, 999): (128, 4), (1, 19, 1031, 65): (32, 1),
          (1, 65, 129, 97): (32, 1), (1, 97, 127, 4095): (32, 8), (1, 128, 5000, 500): (64, 1), (1, 60, 5000, 500): (64, 2), (1, 250, 3000, 500): (96, 2)}


def _product(dev, a, w, a_km, b_kn, guard=64):
    """a [b, m, k] stored [m, k], or [k, m] with a_km; w [b, k, n] stored [n, k], or [k, n] with b_kn."""
    b, m, k = a.shape
    n = w.shape[2]
    sa = dev.slice_from_values(np.ascontiguousarray(a.transpose(0, 2, 1) if a_km else a).ravel())
    sw = dev.slice_from_values(np.ascontiguousarray(w if b_kn else w.transpose(0, 2, 1)).ravel())
    out = dev.slice_from_values(np.full(b * m * n + guard, 3.0, np.float32))
    dev.matmul(out, sa, sw, (b, m, n, k), ([b, m, k], [m * k, 1, m] if a_km else [m * k, k, 1], 0), ([b, k, n], [n * k, n, 1] if b_kn else [n * k, 1, k], 0))
    got = out.to_vec()
    assert np.all(got[b * m * n:] == 3.0)
    return got[:b * m * n].reshape(b, m, n)


def _bound(a, w):
    """k products and sums in f32, each rounding at most 2^-24 of the sum of magnitudes; the parts that are left out are 2^-26 of it."""
    return np.abs(a).astype(np.float64) @ np.abs(w).astype(np.float64) * (a.shape[2] + 16) * 2.0 ** -24 + 1e-44


@pytest.mark.parametrize("a_km", [False, True])
@pytest.mark.parametrize("b_kn", [False, True])
@pytest.mark.parametrize("b,m,n,k", list(SHAPES))
def test_layouts(dev, b, m, n, k, a_km, b_kn):
    a, w = synth.normal(31 + m, (b, m, k), 0.5), synth.normal(32 + n, (b, k, n), 0.5)
    got = _product(dev, a, w, a_km, b_kn)
    assert np.all(np.abs(got - a.astype(np.float64) @ w.astype(np.float64)) <= _bound(a, w))


def test_error_is_that_of_one_rounding_not_of_k(dev):
    """The sums are drained every 64 k and added in f32: over long k the error stays far below that of 4096 f32 additions."""
    a, w = synth.normal(1, (1, 200, 4096), 0.5), synth.normal(2, (1, 4096, 640), 0.5)
    want = a.astype(np.float64) @ w.astype(np.float64)
    assert np.linalg.norm(_product(dev, a, w, False, False) - want) < 3e-7 * np.linalg.norm(want)


@pytest.mark.parametrize("scale_a,scale_w", [(2.0 ** -100, 1.0), (2.0 ** -110, 2.0 ** 100), (2.0 ** -60, 2.0 ** -60), (2.0 ** -70, 2.0 ** -75), (2.0 ** 100, 2.0 ** -100),
                                             (2.0 ** -135, 2.0 ** 120), (2.0 ** 63, 2.0 ** 60)])
def test_ends_of_the_range(dev, scale_a, scale_w):
    """Parts or products of parts that would not be normal numbers, subnormal inputs, large ones."""
    a, w = synth.normal(3, (1, 70, 200), 0.5) * np.float32(scale_a), synth.normal(4, (1, 200, 300), 0.5) * np.float32(scale_w)
    got, want = _product(dev, a, w, False, False), a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.isfinite(got))
    # a result below the normal range is rounded to its spacing, and so is every product on the way
    assert np.all(np.abs(got - want) <= _bound(a, w) + 200 * 2.0 ** -149)


def test_one_tiny_value_in_a_tile(dev):
    """A value that only FFMA holds: its own tiles are computed again, and it counts where everything else is zero."""
    a, w = synth.normal(5, (1, 130, 128), 0.5), synth.normal(6, (1, 128, 260), 0.5)
    a[0, 5] = 0.0
    a[0, 5, 77] = np.float32(1e-41)
    w[0, 77] *= np.float32(1e30)
    got, want = _product(dev, a, w, False, True), a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.abs(got - want) <= _bound(a, w)) and np.any(got[0, 5] != 0.0)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
def test_what_is_not_finite_stays_in_its_row(dev, value):
    a, w = synth.normal(7, (1, 70, 300), 0.5), synth.normal(8, (1, 300, 260), 0.5)
    a[0, 69, 299] = value
    w[0, :, 100] = 0.0
    w[0, 299, 100] = 0.25
    with np.errstate(all="ignore"):
        want = (a[0].astype(np.float64) @ w[0].astype(np.float64)).astype(np.float32)
    got = _product(dev, a, w, False, False)[0]
    assert np.all(np.isfinite(got[:69]))
    assert np.array_equal(np.isnan(got[69]), np.isnan(want[69])) and np.array_equal(np.isinf(got[69]), np.isinf(want[69]))
    assert got[69, 100] == want[69, 100] or np.isnan(value)


def test_whole_numbers_are_exact(dev):
    rng = np.random.default_rng(9)
    a, w = rng.integers(-200, 200, (1, 150, 256)).astype(np.float32), rng.integers(-200, 200, (1, 256, 300)).astype(np.float32)
    assert np.array_equal(_product(dev, a, w, False, False), a @ w)


def test_shared_matrix_and_strided_result(dev):
    """One matrix for every batch step, as a linear layer of the graph has it."""
    b, m, n, k = 3, 45, 200, 320
    a, w = synth.normal(10, (b, m, k), 0.5), synth.normal(11, (k, n), 0.5)
    out = dev.allocate_uninit(DType.F32, b * m * n)
    dev.matmul(out, dev.slice_from_values(a.ravel()), dev.slice_from_values(np.ascontiguousarray(w.T).ravel()), (b, m, n, k), ([b, m, k], [m * k, k, 1], 0), ([b, k, n], [0, 1, k], 0))
    got = out.to_vec().reshape(b, m, n)
    assert np.all(np.abs(got - a.astype(np.float64) @ w.astype(np.float64)) <= _bound(a, np.broadcast_to(w, (b, k, n))))
