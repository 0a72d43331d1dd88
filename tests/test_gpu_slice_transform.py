"""Single transforms through the bit-sliced passes (csrc/slicefft.cu): every
size they serve up to 2^19 and the ones around its edges against the oracle's
transform, the inverse, random words and single nonzero words (whose
transforms show each twiddle), and a buffer on 8 bytes only, which takes the
word passes, at the largest sizes both against each other."""
import numpy as np
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _run(engine, m, f, shift=0):
    F = engine.CudaFFT()
    F.init(m)
    d = engine.DeviceBuffer((8 << m) + 8)
    d.upload(f, offset_bytes=shift)
    F.fwd(d.ptr + shift)
    got = d.to_numpy(1 << m, offset_bytes=shift)
    F.inv(d.ptr + shift)
    assert (d.to_numpy(1 << m, offset_bytes=shift) == f).all(), ("inverse", m, shift)
    return got


@pytest.mark.parametrize("m", list(range(9, 20)))
def test_transforms_against_oracle(engine, oracle, m):
    f = W.splitmix64(40 + m, 1 << m)
    assert (_run(engine, m, f) == oracle.fft_fwd(f, m)).all()
    one = np.zeros(1 << m, dtype=np.uint64)
    one[(5 << (m - 3)) | 1] = np.uint64(0x8000000000000001)
    assert (_run(engine, m, one) == oracle.fft_fwd(one, m)).all()


@pytest.mark.parametrize("m", [13, 18, 20, 21, 22, 23, 24])
def test_sliced_and_word_passes_agree(engine, m):
    f = W.splitmix64(90 + m, 1 << m)
    assert (_run(engine, m, f) == _run(engine, m, f, 8)).all()
