"""Products of few rows against [n, k] rows (the kernel of a decode step's projections): every number of rows it takes, and
the edges of its 16-column tiles, 64-wide k chunks, warps and pieces, against float64 on the same 16-bit values."""
import numpy as np
import pytest

from ug_b200 import synth

pytestmark = pytest.mark.gpu


def _bits(x, f16):
    return x.astype(np.float16) if f16 else synth.to_bf16_bits(x)


def _wide(b, f16):
    return b.astype(np.float64) if f16 else synth.bf16_bits_to_f32(b).astype(np.float64)


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("m", [1, 2, 7, 8, 9])
@pytest.mark.parametrize("n,k", [(1, 8), (15, 64), (16, 72), (17, 520), (33, 2048), (200, 2056), (3000, 512), (48, 5632), (40, 8200),
                                 # more than a piece for every CTA of a 148-SM device: by k and alignment on three kernels
                                 (3152, 64), (3168, 64), (3168, 1016), (3168, 1024), (3161, 72), (3161, 136), (8191, 8)])
def test_rows_against_nk(dev, m, n, k, f16):
    a, w = synth.normal(11 + m, (m, k), 0.5), synth.normal(12 + n, (n, k), 0.5)
    ab, wb = _bits(a, f16), _bits(w, f16)
    from ug_b200 import DType
    sa, sw = dev.slice_from_values(ab.ravel(), bf16=not f16), dev.slice_from_values(wb.ravel(), bf16=not f16)
    guard = 64
    out = dev.slice_from_values(_bits(np.full(m * n + guard, 3.0, np.float32), f16), bf16=not f16)
    dev.matmul(out, sa, sw, (1, m, n, k), ([1, m, k], [m * k, k, 1], 0), ([1, k, n], [n * k, 1, k], 0))
    got = _wide(out.to_vec(), f16)
    assert np.all(got[m * n:] == 3.0)
    wa, ww = _wide(ab, f16), _wide(wb, f16)
    want = wa @ ww.T
    # one rounding of the result (to nearest: at most 2^-8 of it in bf16, 2^-11 in f16) plus f32 sums of k products: k 2^-24 of the sum of magnitudes
    bound = np.abs(want) * 2.0 ** (-11 if f16 else -8) + (np.abs(wa) @ np.abs(ww).T) * k * 2.0 ** -24 + 1e-6
    assert np.all(np.abs(got[:m * n].reshape(m, n) - want) <= bound)


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("m", [1, 8])
@pytest.mark.parametrize("n,k", [(4720, 1024), (4736, 2056), (4737, 1032), (9489, 1024)])
def test_pieces_around_two_ctas_per_sm(dev, m, n, k, f16):
    """295 to 594 pieces: one for every CTA of two per SM (148 SMs), and one and two more than that."""
    test_rows_against_nk(dev, m, n, k, f16)


@pytest.mark.parametrize("b,m,shared", [(3, 4, False), (2, 8, False), (2, 4, True), (3, 3, True)])
@pytest.mark.parametrize("n,k", [(72, 328), (1600, 64), (1601, 136)])
def test_batches(dev, b, m, shared, n, k):
    a, w = synth.to_bf16_bits(synth.normal(3, (b, m, k), 0.5)), synth.to_bf16_bits(synth.normal(4, (1 if shared else b, n, k), 0.5))
    from ug_b200 import DType
    out = dev.allocate_uninit(DType.BF16, b * m * n)
    dev.matmul(out, dev.slice_from_values(a.ravel(), bf16=True), dev.slice_from_values(w.ravel(), bf16=True), (b, m, n, k),
               ([b, m, k], [m * k, k, 1], 0), ([b, k, n], [0 if shared else n * k, 1, k], 0))
    wa, ww = (synth.bf16_bits_to_f32(x).astype(np.float64) for x in (a, w))
    want = np.einsum("bmk,bnk->bmn", wa, np.broadcast_to(ww, (b, n, k)))
    got = synth.bf16_bits_to_f32(out.to_vec()).reshape(b, m, n)
    assert np.all(np.abs(got - want) <= np.abs(want) * 2.0 ** -8 + np.einsum("bmk,bnk->bmn", np.abs(wa), np.broadcast_to(np.abs(ww), (b, n, k))) * k * 2.0 ** -24 + 1e-6)
