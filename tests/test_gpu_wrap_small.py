"""Wrapped products where the transforms are cluster products or just above
(2^11 .. 2^16 points, csrc/wrapmul.cu): chunk counts from one past a power of
two to a quarter past it and beyond, balanced and uneven, against the oracle."""
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [12, 13, 14, 15, 16, 17])
def test_wrapped_products_by_value(engine, oracle, m):
    E = engine.engine
    half = 1 << (m - 1)
    jobs, want = [], []
    for extra in (1, 2, 17, half // 8 + 1, half // 4 - 1, half // 4, half // 4 + 1):
        for share in (0.5, 0.11):
            ca = int((half + extra + 1) * share)
            cb = half + extra + 1 - ca
            for ab, bb in ((32 * ca, 32 * cb), (32 * ca - 31, 32 * cb - 5)):
                a, b = W.random_bits(ab, len(jobs)), W.random_bits(bb, 1000 + len(jobs))
                jobs.append((engine.DeviceBuffer.from_array(a), ab, engine.DeviceBuffer.from_array(b),
                             bb, engine.DeviceBuffer(8 * E.mul_out_words(ab, bb))))
                want.append(oracle.fft_mul(a, ab, b, bb))
    engine.mul_batch_dev(jobs)
    for (_, ab, _, bb, out), w in zip(jobs, want):
        got = out.to_numpy(E.mul_out_words(ab, bb))
        assert (got[: w.size] == w).all() and not got[w.size:].any(), (ab, bb)
