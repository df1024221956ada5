"""Chains of operators that read and overwrite the same few buffers without a host synchronisation between two of them.  Every
kernel is a dependent launch, so several are resident at once: the bits have to be those of the same chain with the host waiting
after every call."""
import numpy as np
import pytest

from ug_b200 import DType, synth

pytestmark = pytest.mark.gpu


def _both(dev, chain):
    want = chain(dev.synchronize)
    for _ in range(3):
        got = chain(lambda: None)
        assert len(got) == len(want)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)


def _nk(b, n, k):
    return [b, k, n], [n * k, 1, k], 0


def _kn(b, n, k):
    return [b, k, n], [n * k, n, 1], 0


def _rows(b, m, k):
    return [b, m, k], [m * k, k, 1], 0


@pytest.mark.parametrize("m", [1, 4, 24, 130])           # streamed columns; the same; 32- and 128-row tiles
@pytest.mark.parametrize("n", [256, 255])                # 255: no 16-byte rows
def test_f32_rows_and_products(dev, m, n):
    p0, w0, v0 = synth.normal(1, (m, n)), synth.normal(2, (n, n), n ** -0.5), synth.normal(3, (n, n), n ** -0.5)

    def chain(wait):
        p, w, w2, v = (dev.slice_from_values(x.ravel()) for x in (p0, w0, w0, v0))
        q = dev.allocate_uninit(DType.F32, m * n)
        dev.synchronize()
        for i in range(24):
            dev.matmul(q, p, w, (1, m, n, n), _rows(1, m, n), _nk(1, n, n)); wait()
            dev.custom_softmax(q, p, m, n); wait()
            dev.matmul(q, p, w, (1, m, n, n), _rows(1, m, n), _kn(1, n, n)); wait()          # p again, w by its other direction
            dev.rms_norm(q, p, p, m, n, 1e-5) if m == 1 else dev.rms_norm(q, w2, p, m, n, 1e-5); wait()
            dev.matmul(w2, w, v, (1, n, n, n), _rows(1, n, n), _kn(1, n, n)); wait()         # the next w
            dev.rms_norm_silu_gate(w2, p, v, w, n, n, 1e-5); wait()                          # gain: the first row of p
        return [p.to_vec(), q.to_vec(), w.to_vec(), w2.to_vec()]
    _both(dev, chain)


@pytest.mark.parametrize("m", [1, 8, 40])                # streamed matrix, the most of it, tensor-core tiles
@pytest.mark.parametrize("n,f16", [(256, False), (256, True), (2048, False), (250, False)])
def test_16_bit_products(dev, m, n, f16):
    def bits(seed, shape, std):
        x = synth.normal(seed, shape, std)
        return x.astype(np.float16) if f16 else synth.to_bf16_bits(x)
    a0, w0, v0 = bits(4, (m, n), 1.0), bits(5, (n, n), n ** -0.5), bits(6, (n, n), n ** -0.5)
    steps = 12 if n < 1000 else 6

    def chain(wait):
        a, c, w, w2, v = (dev.slice_from_values(x.ravel(), bf16=not f16) for x in (a0, a0, w0, w0, v0))
        dev.synchronize()
        for i in range(steps):
            dev.matmul(c, a, w, (1, m, n, n), _rows(1, m, n), _nk(1, n, n)); wait()
            dev.matmul(w2, w, v, (1, n, n, n), _rows(1, n, n), _nk(1, n, n)); wait()
            dev.matmul(a, c, w2, (1, m, n, n), _rows(1, m, n), _nk(1, n, n)); wait()         # w2 straight behind its writer
            dev.matmul(w, w2, v, (1, n, n, n), _rows(1, n, n), _nk(1, n, n)); wait()
        return [a.to_vec(), c.to_vec(), w.to_vec(), w2.to_vec()]
    _both(dev, chain)
