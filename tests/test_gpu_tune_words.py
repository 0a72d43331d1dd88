"""The FFT autotuner times and checks the word passes, which its knobs act on,
and not the bit-sliced ones, which have none; and transforms and products under
non-default tunings through the word passes (buffers and scratch on 8 bytes
only), against the oracle."""
import numpy as np
import pytest

from kernel_names import kernel_counts, launched
from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu

TUNINGS = [
    dict(fft_tile_log=11, fft_cmin=2, fft_taylor_lv=1, fft_bfly_lv=1),
    dict(fft_tile_log=13, fft_cmin=16, fft_taylor_lv=2, fft_bfly_lv=2),
    dict(fft_tile_log=13, fft_cmin=4, fft_taylor_lv=3, fft_bfly_lv=1),
]


@pytest.fixture
def tuner(engine):
    from mersenne_trinomial_b200 import autotune as A
    saved = A.tune_get()
    yield A
    A.tune_set(**saved)


@pytest.mark.parametrize("m", [10, 14, 18])
def test_autotuner_runs_the_word_passes(tuner, m):
    got = []
    names = kernel_counts(lambda: got.append(tuner.fft_autotune(m, reps=1)))
    res = got[-1]
    assert launched(names, "k_fft_pass") > 0, names
    assert not launched(names, "k_bfly") and not launched(names, "k_slice"), names
    assert all(c["status"] == "ok" for c in res["candidates"])
    assert tuner.tune_get() == res["best"]


@pytest.mark.parametrize("tune", TUNINGS)
def test_word_passes_under_tuning(engine, oracle, tuner, tune):
    tuner.tune_set(**tune)
    E = engine.engine
    for m in (11, 15, 18):
        f = W.splitmix64(700 + m, 1 << m)
        F = engine.CudaFFT()
        F.init(m)
        d = engine.DeviceBuffer((8 << m) + 8)
        d.upload(f, offset_bytes=8)
        F.fwd(d.ptr + 8)
        assert (d.to_numpy(1 << m, offset_bytes=8) == oracle.fft_fwd(f, m)).all(), (tune, m)
        F.inv(d.ptr + 8)
        assert (d.to_numpy(1 << m, offset_bytes=8) == f).all(), (tune, m)
        F.fini()
    ab, bb = 2**20 + 3, 2**19 + 1                   # above the cluster product's 2^14
    a, b = W.random_bits(ab, ab), W.random_bits(bb, bb + 1)
    m = E.fft_m_for(ab, bb)
    F = engine.CudaFFT()
    F.init(m)
    ow = E.mul_out_words(ab, bb)
    fa, fb = engine.DeviceBuffer((8 << m) + 8), engine.DeviceBuffer((8 << m) + 8)
    out = engine.DeviceBuffer(8 * ow)
    E.gf2x_fft_mul_dev(F, engine.DeviceBuffer.from_array(a), ab, engine.DeviceBuffer.from_array(b),
                       bb, out, fa.ptr + 8, fb.ptr + 8)
    want = oracle.fft_mul(a, ab, b, bb)
    assert (out.to_numpy(ow)[: want.size] == want).all()
