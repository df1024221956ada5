"""f32 products on the tensor cores: edges of their tiles (128 columns of the result x 32 to 96 rows), of the 32-k stages and the shares of a
cluster, every layout of both operands, and values that three bf16 parts do not hold, against float64; and their error beside the FFMA kernel's."""
import numpy as np
import pytest

from ug_b200 import DType, synth

pytestmark = pytest.mark.gpu
# (b, m, n, k) -> (rows of a tile, CTAs along k) on 148 SMs; test_f32_split_plan_cpu.py holds the rule to these.  Four stages of k, 32 and 33 of them, several
# groups of stages and transfers of the small products; and the tests of single values, of long k and of shared matrices
SHAPES = {(1, 4932, 132, 100): (96, 1), (1, 2000, 1500, 101): (96, 1), (1, 600, 3000, 1024): (64, 1), (1, 600, 3000, 1025): (64, 1), (1, 257, 5632, 2048): (96, 1),
          (1, 922, 523, 420): (32, 1), (16, 300, 777, 400): (64, 1), (1, 128, 5000, 500): (64, 1), (2, 526, 1080, 216): (96, 1),
          (1, 31, 8000, 999): (32, 2), (1, 500, 1001, 999): (64, 2), (1, 60, 5000, 500): (64, 2), (1, 33, 8001, 1031): (64, 2), (1, 250, 3000, 500): (96, 2),
          (3, 257, 1024, 512): (96, 2), (1, 64, 2048, 2048): (32, 4), (1, 128, 2048, 2048): (64, 4), (1, 97, 1027, 4095): (64, 4), (1, 770, 269, 412): (96, 4),
          (1, 97, 127, 4095): (32, 8), (1, 129, 300, 4097): (64, 8), (1, 386, 131, 1628): (96, 8)}
# chains of f32 additions that the FFMA kernel has for these, which are the shortest that leave it
CHAINS = {(1, 4932, 132, 100): 1, (16, 300, 777, 400): 2, (1, 250, 3000, 500): 4, (1, 500, 1001, 999): 8, (1, 64, 2048, 2048): 16, (1, 97, 127, 4095): 32}


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
    """k products and sums in f32, each rounding at most 2^-24 of the sum of magnitudes; the product of parts that is left out is 2^-33 of it."""
    return np.abs(a).astype(np.float64) @ np.abs(w).astype(np.float64) * (a.shape[2] + 16) * 2.0 ** -24 + 1e-44


@pytest.mark.parametrize("a_km", [False, True])
@pytest.mark.parametrize("b_kn", [False, True])
@pytest.mark.parametrize("b,m,n,k", list(SHAPES))
def test_layouts(dev, b, m, n, k, a_km, b_kn):
    a, w = synth.normal(31 + m, (b, m, k), 0.5), synth.normal(32 + n, (b, k, n), 0.5)
    got = _product(dev, a, w, a_km, b_kn)
    want = a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.abs(got - want) <= _bound(a, w))
    # A few times the spacing of f32 at 1 (1.2e-7): sums of 16 products that are cut off once, then rounded additions.  A part that is missing
    # or taken from the wrong k is 2e-6 and more of such a result, which the bound above does not see.
    assert np.linalg.norm(got - want) <= 3e-7 * np.linalg.norm(want)


@pytest.mark.parametrize("a_km", [False, True])
@pytest.mark.parametrize("b_kn", [False, True])
@pytest.mark.parametrize("b,m,n,k", list(SHAPES))
def test_every_part_counts(dev, b, m, n, k, a_km, b_kn):
    """Values whose last seven bits are in the third part alone, times a matrix that picks one of them for every result: each comes out
    exact, through either operand."""
    rng = np.random.default_rng(m + n)
    full = lambda *shape: (1 + 129 * 2.0 ** -16 + rng.integers(-63, 64, shape) * 2.0 ** -23).astype(np.float32)
    a, pick = full(b, m, k), rng.integers(0, k, n)
    pick[:min(n, k)] = np.arange(k)[::-1][:min(n, k)]
    w = np.zeros((b, k, n), np.float32)
    w[:, pick, np.arange(n)] = 1.0
    assert np.array_equal(_product(dev, a, w, a_km, b_kn), a[:, :, pick])
    w, pick = full(b, k, n), rng.integers(0, k, m)
    pick[:min(m, k)] = np.arange(k)[:min(m, k)]
    a = np.zeros((b, m, k), np.float32)
    a[:, np.arange(m), pick] = 1.0
    assert np.array_equal(_product(dev, a, w, a_km, b_kn), w[:, pick])


def _content(kind, b, m, n, k):
    rng = np.random.default_rng(m)
    probs = lambda d: (lambda e: e / e.sum(-1, keepdims=True))(np.exp(d * rng.standard_normal((b, m, k))))
    a, w = {"normal": lambda: (rng.standard_normal((b, m, k)), rng.standard_normal((b, k, n))), "uniform": lambda: (rng.random((b, m, k)), rng.random((b, k, n))),
            "probabilities": lambda: (probs(3), rng.random((b, k, n))), "one large probability": lambda: (probs(8), rng.random((b, k, n))),
            "one value": lambda: (np.full((b, m, k), 1 + 255 * 2.0 ** -16 + 63 * 2.0 ** -23), np.full((b, k, n), 1 + 255 * 2.0 ** -16 + 63 * 2.0 ** -23))}[kind]()
    return a.astype(np.float32), w.astype(np.float32)


def _ffma(a, w, chains):
    """Dot products of rows in f32 as the FFMA kernel has them: `chains` sums of every so many products, then the sum of those."""
    sums = []
    for c in range(chains):
        acc = np.zeros(len(a), np.float32)
        for i in range(c, a.shape[1], chains):
            acc = (a[:, i].astype(np.float64) * w[:, i] + acc).astype(np.float32)
        sums.append(acc)
    out = sums[0]
    for x in sums[1:]:
        out = out + x
    return out


@pytest.mark.parametrize("kind", ["normal", "uniform", "probabilities", "one large probability", "one value"])
@pytest.mark.parametrize("b,m,n,k", list(CHAINS))
def test_error_beside_the_ffma_kernel(dev, b, m, n, k, kind):
    """Sums of one sign too, where what a sum is cut off by adds up: 4000 results against those of FFMAs, whose error may be the smaller one by
    what a sample of it varies (5 %) and no more."""
    a, w = _content(kind, b, m, n, k)
    got, rng = _product(dev, a, w, False, False), np.random.default_rng(1)
    bi, i, j = rng.integers(0, b, 4000), rng.integers(0, m, 4000), rng.integers(0, n, 4000)
    x, y = a[bi, i], w[bi, :, j]
    want = np.einsum("rk,rk->r", x.astype(np.float64), y.astype(np.float64))
    err = lambda v: np.linalg.norm(v - want) / np.linalg.norm(want)
    assert err(got[bi, i, j]) <= 1.1 * max(err(_ffma(x, y, CHAINS[b, m, n, k])), 2.0 ** -25)


@pytest.mark.parametrize("scale_a,scale_w", [(2.0 ** -100, 1.0), (2.0 ** -110, 2.0 ** 100), (2.0 ** -60, 2.0 ** -60), (2.0 ** -70, 2.0 ** -75), (2.0 ** 100, 2.0 ** -100),
                                             (2.0 ** -135, 2.0 ** 120), (2.0 ** 63, 2.0 ** 60)])
def test_ends_of_the_range(dev, scale_a, scale_w):
    """Parts or products of parts that would not be normal numbers, subnormal inputs, large ones."""
    a, w = synth.normal(3, (1, 250, 500), 0.5) * np.float32(scale_a), synth.normal(4, (1, 500, 3000), 0.5) * np.float32(scale_w)
    got, want = _product(dev, a, w, False, False), a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.isfinite(got))
    # a result below the normal range is rounded to its spacing, and so is every product on the way
    assert np.all(np.abs(got - want) <= _bound(a, w) + 500 * 2.0 ** -149)


def test_one_tiny_value_in_a_tile(dev):
    """A value that only FFMA holds: its own tiles are computed again, and it counts where everything else is zero."""
    a, w = synth.normal(5, (1, 2000, 101), 0.5), synth.normal(6, (1, 101, 1500), 0.5)
    a[0, 5] = 0.0
    a[0, 5, 77] = np.float32(1e-41)
    w[0, 77] *= np.float32(1e30)
    got, want = _product(dev, a, w, False, True), a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.abs(got - want) <= _bound(a, w)) and np.any(got[0, 5] != 0.0)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("m,n,k", [(257, 5632, 2048), (128, 2048, 2048), (922, 523, 420), (60, 5000, 500)])
def test_what_is_not_finite_stays_in_its_row(dev, m, n, k, last, value):
    """In the last row, at either end of k (with k over a cluster, one CTA sees it), against columns of which the last is zero elsewhere.  The
    results beside it in its tile are the bits that they are without it."""
    a, w = synth.normal(7, (1, m, k), 0.5), synth.normal(8, (1, k, n), 0.5)
    at = k - 1 if last else 3
    w[0, :, n - 1] = 0.0
    w[0, at, n - 1] = 0.25
    plain = _product(dev, a, w, False, False)[0]
    a[0, m - 1, at] = value
    with np.errstate(all="ignore"):
        want = (a[0, m - 1].astype(np.float64) @ w[0].astype(np.float64)).astype(np.float32)
    got = _product(dev, a, w, False, False)[0]
    assert np.array_equal(got[:m - 1], plain[:m - 1]) and np.all(np.isfinite(plain))
    assert np.array_equal(np.isnan(got[m - 1]), np.isnan(want)) and np.array_equal(np.isinf(got[m - 1]), np.isinf(want))
    on = np.isfinite(want)
    assert np.all(np.abs(got[m - 1, on] - want[on]) <= 2.0 ** -20 * np.abs(want[on])) and np.array_equal(got[m - 1][np.isinf(want)], want[np.isinf(want)])


@pytest.mark.parametrize("a_km,b_kn", [(False, True), (True, False), (True, True)])
def test_a_column_that_is_not_finite(dev, a_km, b_kn):
    a, w = synth.normal(12, (1, 257, 2048), 0.5), synth.normal(13, (1, 2048, 5632), 0.5)
    plain = _product(dev, a, w, a_km, b_kn)[0]
    w[0, 2047, 5631] = np.nan
    got = _product(dev, a, w, a_km, b_kn)[0]
    assert np.array_equal(got[:, :5631], plain[:, :5631]) and np.all(np.isnan(got[:, 5631]))


def test_whole_numbers_are_exact(dev):
    rng = np.random.default_rng(9)
    a, w = rng.integers(-200, 200, (1, 922, 420)).astype(np.float32), rng.integers(-200, 200, (1, 420, 523)).astype(np.float32)
    assert np.array_equal(_product(dev, a, w, False, False), a @ w)


@pytest.mark.parametrize("which", ["left", "right"])
def test_shared_matrix(dev, which):
    """One matrix for every batch step, as a linear layer of the graph has it, on either side."""
    b, m, n, k = 3, 257, 1024, 512
    a, w = synth.normal(10, (b if which == "right" else 1, m, k), 0.5), synth.normal(11, (b if which == "left" else 1, n, k), 0.5)
    out = dev.allocate_uninit(DType.F32, b * m * n)
    dev.matmul(out, dev.slice_from_values(a.ravel()), dev.slice_from_values(w.ravel()), (b, m, n, k),
               ([b, m, k], [m * k if which == "right" else 0, k, 1], 0), ([b, k, n], [n * k if which == "left" else 0, 1, k], 0))
    a, w = np.broadcast_to(a, (b, m, k)), np.broadcast_to(w.transpose(0, 2, 1), (b, k, n))
    got, want = out.to_vec().reshape(b, m, n), a.astype(np.float64) @ w.astype(np.float64)
    assert np.all(np.abs(got - want) <= _bound(a, w)) and np.linalg.norm(got - want) <= 3e-7 * np.linalg.norm(want)
