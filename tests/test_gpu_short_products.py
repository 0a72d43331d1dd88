"""Batches of short products (product_batch in csrc/cantor.cu) on both sides of
the line between the cluster product and the word passes: which kernels run,
the same scan results as with few s at a time, and single products of every
size around the line against the oracle."""
import numpy as np
import pytest
import torch

from kernel_names import kernel_counts, launched
from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


# transforms of 2^4 (r = 129), 2^7, 2^8, 2^9 and 2^10 coefficients; a wave of the
# cluster product is half as many products as there are SMs
@pytest.mark.parametrize("r,waves", [(129, 1), (1279, 1), (2281, 2), (4423, 3), (9689, 30)])
def test_route_and_results_of_many_resident_s(engine, monkeypatch, r, waves):
    monkeypatch.setenv("GF2E_SCAN_GRAPHS", "0")           # the kernels by themselves
    wave = torch.cuda.get_device_properties(0).multi_processor_count // 2
    E = engine.engine
    for slots in (waves * wave, waves * wave + 1):
        if slots > min((r - 1) // 2, 512):
            continue
        S = E.Scanner(r, slots)
        S.submit(np.arange(1, slots + 1), 2, 10**6, 10**5, 10**5)
        S.step(1)
        torch.cuda.synchronize()
        names = kernel_counts(lambda: S.step(2))
        S.close()
        words = slots > waves * wave
        assert (launched(names, "k_fft_pass") > 0) == words, (slots, names)
        assert (launched(names, "k_small_mul") > 0) != words, (slots, names)
    slots = min((r - 1) // 2, waves * wave + 1, 300)
    s = np.arange(1, slots + 1)
    assert E.scan(r, s, 2, 40, L0=8, batch=slots) == E.scan(r, s, 2, 40, L0=8, batch=16)


@pytest.mark.parametrize("bits", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 8191, 8193,
                                  16383, 16385])
def test_single_products_around_the_line(engine, oracle, bits):
    for other in (1, bits):
        a, b = W.random_bits(bits, bits), W.random_bits(other, 7)
        want = oracle.comb_mul(a, bits, b, other)
        got = engine.gf2x_fft_mul(a, bits, b, other)
        assert (got[: want.size] == want).all() and not got[want.size:].any(), other
    E = engine.engine                                   # a square: one operand
    m = E.fft_m_for(bits, bits)
    F = engine.CudaFFT()
    F.init(m)
    ow = E.mul_out_words(bits, bits)
    d, out = engine.DeviceBuffer.from_array(a), engine.DeviceBuffer(8 * ow)
    fa, fb = engine.DeviceBuffer(8 << m), engine.DeviceBuffer(8 << m)
    E.gf2x_fft_mul_dev(F, d, bits, d, bits, out, fa, fb)
    want = oracle.comb_mul(a, bits, a, bits)
    assert (out.to_numpy(ow)[: want.size] == want).all()
