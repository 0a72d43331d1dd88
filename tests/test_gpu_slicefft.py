"""The bit-sliced product transform (csrc/slicefft.cu) against the oracle's
products: one-block products up to 2^12 coefficients and the ones around that
edge, every pass structure above (tile splits, conversions of more than 2^16
coefficients, operands much shorter than the transform), squares, scratch
that is only 8-byte aligned, and batches with strides (the scanner's)."""
import numpy as np
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _product(engine, a, ab, b, bb, shift=0):
    F = engine.CudaFFT()
    F.init(engine.engine.fft_m_for(ab, bb))
    da = engine.DeviceBuffer.from_array(a)
    db = da if b is a else engine.DeviceBuffer.from_array(b)
    ow = engine.mul_out_words(ab, bb)
    out = engine.DeviceBuffer.from_array(np.full(ow, 0xEEEEEEEEEEEEEEEE, dtype=np.uint64))
    fa, fb = (engine.DeviceBuffer((8 << F.m) + 8) for _ in range(2))
    engine.gf2x_fft_mul_dev(F, da, ab, db, bb, out, fa.ptr + shift, fb.ptr + shift)
    got = out.to_numpy(ow)
    F.fini()
    return got


# chunks (a, b): exactly 2^k - 1, 2^k, 2^k + 1 in all; lone chunks; operands
# of 2^16 chunks and one more (the first with levels above 2^16)
CHUNKS = [(1, 1), (255, 257), (1024, 1), (1, 1023), (1025, 1025), (2048, 2049), (4000, 98),
          (4096, 4096), (4097, 4096), (1, 8192), (12000, 20000), (16384, 16384), (40000, 25000),
          (300, 120000), (65536, 65537), (65537, 70000), (200, 260000), (150000, 130000),
          (300000, 70000), (7, 500000)]


@pytest.mark.parametrize("ca,cb", CHUNKS)
def test_products_at_pass_edges(engine, oracle, ca, cb):
    ab, bb = 32 * ca - (ca * 7) % 32, 32 * cb - (cb * 5) % 32
    a, b = W.random_bits(ab, ca + 1), W.random_bits(bb, cb + 2)
    want = oracle.fft_mul(a, ab, b, bb)
    got = _product(engine, a, ab, b, bb)
    assert (got[: want.size] == want).all() and not got[want.size:].any()


@pytest.mark.parametrize("bits", [31, 70000, 140001, 600000])
def test_squares_and_unaligned_scratch(engine, oracle, bits):
    a = W.random_bits(bits, bits)
    want = oracle.fft_mul(a, bits, a, bits)
    for shift in (0, 8):
        got = _product(engine, a, bits, a, bits, shift)
        assert (got[: want.size] == want).all() and not got[want.size:].any(), shift


def test_products_of_sparse_and_full_operands(engine, oracle):
    # zero, one bit at either end, all ones
    bits = 200_003
    n = (bits + 63) // 64
    ones = np.full(n, 0xFFFFFFFFFFFFFFFF, dtype=np.uint64)
    ones[-1] = np.uint64((1 << (bits % 64)) - 1)
    low, high, zero = (np.zeros(n, dtype=np.uint64) for _ in range(3))
    low[0] = 1
    high[-1] = np.uint64(1 << ((bits - 1) % 64))
    for x in (ones, low, high, zero):
        for y in (ones, high):
            want = oracle.fft_mul(x, bits, y, bits)
            got = _product(engine, x, bits, y, bits)
            assert (got[: want.size] == want).all() and not got[want.size:].any()


@pytest.mark.parametrize("r", [60_013, 135_007, 528_001])
def test_strided_batches_through_the_running_product(engine, oracle, r):
    # the scanner multiplies all resident s at once: one degree at a time must
    # agree with blocks of 2 on every result line
    s = [5, 77, 1000, 30_001]
    a = engine.scan(r, s, 2, 10, L0=8, batch=4)
    assert a == engine.scan(r, s, 2, 10, L0=8, batch=4, block=2)
    assert len(a) == len(s)
