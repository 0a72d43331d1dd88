"""gf2e_mul where the second scratch buffer also holds the first operand or the
output, or is the first one (a square, which has no use for it): on each side
of the sizes where products change their form, against the oracle.  A square
leaves an operand in it as it was."""
import numpy as np
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 2^14 (cluster product), 2^15 and 2^16 (no rows above 2^16), 2^17 and 2^19
@pytest.mark.parametrize("ab,bb", [(200_001, 300_000), (400_001, 500_000), (1_000_001, 900_000),
                                   (2_500_001, 1_500_000), (6_000_001, 7_000_003)])
@pytest.mark.parametrize("shared", ["out", "a", "square", "square a", "square out"])
def test_second_buffer_shared(engine, oracle, ab, bb, shared):
    E = engine.engine
    square = shared.startswith("square")
    if square:
        bb = ab
    a, b = W.random_bits(ab, 1), W.random_bits(bb, 2)
    if square:
        b = a
    m = E.fft_m_for(ab, bb)
    F = engine.CudaFFT()
    F.init(m)
    ow = E.mul_out_words(ab, bb)
    fa, fb = engine.DeviceBuffer(8 << m), engine.DeviceBuffer(8 << m)
    da, out = engine.DeviceBuffer.from_array(a), engine.DeviceBuffer(8 * ow)
    if shared.endswith(" a") or shared == "a":
        fb.upload(a, offset_bytes=64)
        da = fb.ptr + 64
    if shared.endswith("out"):
        assert ow <= 1 << m
        out = fb
    if shared == "square":
        fb = fa
    db = da if square else engine.DeviceBuffer.from_array(b)
    E.gf2x_fft_mul_dev(F, da, ab, db, bb, out, fa, fb)
    want = oracle.fft_mul(a, ab, b, bb)
    assert (out.to_numpy(ow)[: want.size] == want).all()
    if shared == "square a":
        assert (fb.to_numpy(a.size, offset_bytes=64) == a).all()
