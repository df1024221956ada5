"""f32 products of many rows or few columns: edges of the 32- to 128-row tiles, of the 128-column tiles and 16-deep slices, products so small
that k is split inside a CTA and over a cluster, and every layout of both operands, against float64.  Sizes that run on the tensor cores on
148 SMs (test_f32_split_gpu.py has their edges) are here beside those that do not: FFMA and FFMA_KM."""
import numpy as np
import pytest

from ug_b200 import DType, synth

pytestmark = pytest.mark.gpu
TURNED = [(20000, 17, 64), (8193, 8, 512), (3000, 5, 1999), (2600, 36, 1000), (5000, 64, 300), (1301, 33, 597)]   # few columns: the rows of the tile

# (b, m, n, k) -> (warps over rows, over a slice's k, CTAs along k, turned) on 148 SMs, what stays on the FFMA kernel: whatever the left layout, and
# with the left operand stored [k, m]; test_f32_split_plan_cpu.py holds the rules to these
FFMA = {(1, 33, 132, 20): (1, 4, 1, 0), (1, 20, 4, 128): (1, 4, 2, 0), (1, 70, 260, 300): (1, 4, 4, 0), (1, 101, 511, 1030): (1, 4, 8, 0),
        (38, 100, 4, 88): (1, 4, 1, 1), (1, 8192, 8, 512): (1, 4, 2, 1), (1, 3000, 5, 1999): (1, 4, 4, 1), (11, 36, 4, 524): (1, 4, 8, 1),
        (1, 779, 667, 36): (2, 2, 1, 0), (1, 1212, 544, 40): (2, 2, 1, 0), (1, 371, 270, 582): (2, 2, 8, 0), (1, 356, 284, 584): (2, 2, 8, 0),
        (1, 2179, 35, 589): (2, 2, 8, 1), (1, 2200, 36, 584): (2, 2, 8, 1), (38, 100, 4, 20): (4, 1, 1, 0), (1, 1001, 3001, 21): (4, 1, 1, 0)}
FFMA_KM = {(1, 583, 131, 258): (2, 2, 4, 0), (1, 584, 132, 272): (2, 2, 4, 0), (1, 3876, 45, 289): (2, 2, 4, 1), (1, 3900, 36, 292): (2, 2, 4, 1),
           (1, 736, 261, 535): (4, 1, 8, 0), (1, 720, 280, 532): (4, 1, 8, 0)}


def _check(dev, b, m, n, k, a_km, b_kn, shared=False):
    """a stored [m, k], or [k, m] with a_km; b stored [n, k], or [k, n] with b_kn."""
    a, w = synth.normal(21 + m, (b, m, k), 0.5), synth.normal(22 + n, (1 if shared else b, k, n), 0.5)
    sa = dev.slice_from_values(np.ascontiguousarray(a.transpose(0, 2, 1) if a_km else a).ravel())
    sw = dev.slice_from_values(np.ascontiguousarray(w if b_kn else w.transpose(0, 2, 1)).ravel())
    out = dev.slice_from_values(np.full(b * m * n + 64, 3.0, np.float32))
    dev.matmul(out, sa, sw, (b, m, n, k), ([b, m, k], [m * k, 1, m] if a_km else [m * k, k, 1], 0),
               ([b, k, n], [0 if shared else n * k, n, 1] if b_kn else [0 if shared else n * k, 1, k], 0))
    got = out.to_vec()
    assert np.all(got[b * m * n:] == 3.0)
    a, w = a.astype(np.float64), np.broadcast_to(w, (b, k, n)).astype(np.float64)
    # k products and sums in f32: each rounding is at most 2^-24 of the sum of magnitudes
    assert np.all(np.abs(got[:b * m * n].reshape(b, m, n) - a @ w) <= np.abs(a) @ np.abs(w) * (k + 16) * 2.0 ** -24 + 1e-30)


@pytest.mark.parametrize("a_km", [False, True])
@pytest.mark.parametrize("b_kn", [False, True])
@pytest.mark.parametrize("m,n,k", [(17, 4, 4), (32, 128, 16), (33, 132, 20), (64, 260, 128), (100, 512, 1030), (129, 127, 129), (257, 640, 2048),
                                   (31, 33, 35), (1, 338, 6045), (600, 1280, 96),
                                   # one slice of k or less: 64 x 64 tiles; and far more results than those are taken for
                                   (65, 63, 1), (130, 129, 15), (64, 65, 16), (63, 200, 17), (5000, 4000, 6)] + TURNED)
def test_layouts(dev, m, n, k, a_km, b_kn):
    _check(dev, 1, m, n, k, a_km, b_kn)


@pytest.mark.parametrize("b_kn", [False, True])
@pytest.mark.parametrize("b,m,n,k", list(FFMA) + list(FFMA_KM))
def test_every_instance(dev, b, m, n, k, b_kn):
    for a_km in (False, True) if (b, m, n, k) in FFMA else (True,):
        _check(dev, b, m, n, k, a_km, b_kn)


@pytest.mark.parametrize("b,m,n,k,shared", [(5, 40, 96, 512, False), (3, 130, 36, 61, False), (16, 20, 200, 256, True), (40, 65, 132, 72, False)])
def test_batches(dev, b, m, n, k, shared):
    _check(dev, b, m, n, k, False, False, shared)
    _check(dev, b, m, n, k, False, True, shared)


def test_infinities_stay_in_their_row(dev):
    """Rows behind the edge of a tile are filled with zeros: they must not meet an infinity of another row or column."""
    m, n, k = 70, 132, 300
    a, w = synth.normal(1, (m, k), 0.5), synth.normal(2, (n, k), 0.5)
    a[69, 299] = np.inf
    w[131, 7] = -np.inf
    out = dev.allocate_uninit(DType.F32, m * n)
    dev.matmul(out, dev.slice_from_values(a.ravel()), dev.slice_from_values(w.ravel()), (1, m, n, k), ([1, m, k], [m * k, k, 1], 0), ([1, k, n], [n * k, 1, k], 0))
    got = out.to_vec().reshape(m, n)
    assert np.all(np.isfinite(got[:69, :131])) and not np.any(np.isfinite(got[69])) and not np.any(np.isfinite(got[:, 131]))
