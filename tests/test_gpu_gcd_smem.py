"""Quadratic gcds in shared memory (csrc/lehmer.cuh without the matrix) against
the oracle's Euclid at the sizes where they can go wrong: one word and less,
word edges, zero and equal operands, factors of x, very uneven operands (large
quotients) and the largest operands that fit, and one word more, which takes
the kernel for larger ones."""
import numpy as np
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _gcd(engine, pairs, cap):
    bufs = [(engine.DeviceBuffer.from_array(a), ab, engine.DeviceBuffer.from_array(b), bb)
            for a, ab, b, bb in pairs]
    return engine.engine.gcd_batch(bufs, g_cap_words=cap)


def _poly(bits, seed):
    w = W.random_bits(bits, seed)
    w[(bits - 1) >> 6] |= np.uint64(1 << ((bits - 1) & 63))
    return w


def test_small_and_degenerate_pairs(engine, oracle):
    pairs = []
    for i, (ab, bb) in enumerate([(1, 1), (1, 64), (64, 64), (65, 64), (128, 1), (129, 3), (63, 200),
                                  (700, 7), (4097, 65), (4096, 4096), (5000, 4)]):
        pairs.append((_poly(ab, i + 1), ab, _poly(bb, i + 50), bb))
    z = np.zeros(3, dtype=np.uint64)
    x = _poly(150, 9)
    pairs += [(z, 150, x, 150), (x, 150, z, 150), (z, 150, z, 150), (x, 150, x, 150)]
    low = np.zeros(5, dtype=np.uint64)          # x^200 and x^130 + x^77
    low[200 >> 6] = np.uint64(1 << (200 & 63))
    two = np.zeros(5, dtype=np.uint64)
    two[130 >> 6] |= np.uint64(1 << (130 & 63))
    two[77 >> 6] |= np.uint64(1 << (77 & 63))
    pairs.append((low, 201, two, 131))
    degs, gs = _gcd(engine, pairs, 80)
    for (a, ab, b, bb), d, g in zip(pairs, degs, gs):
        want = oracle.poly_gcd(a, b)
        assert int(d) == want[0], (ab, bb)
        w = np.asarray(want[1], dtype=np.uint64)
        n = min(w.size, g.size)
        assert (g[:n] == w[:n]).all() and not g[n:].any(), (ab, bb)


@pytest.mark.parametrize("bits,other,common", [(20_000, 19_999, 700), (99_767, 50_001, 65),
                                                (60_000, 900, 400), (408_000, 407_000, 130),
                                                (409_537, 409_500, 130)])
def test_planted_factors_up_to_the_limit(engine, oracle, bits, other, common):
    c = _poly(common, 3)
    pair = []
    for n, seed in ((bits, 4), (other, 5)):
        q = _poly(n - common + 1, seed)
        pair += [oracle.fft_mul(q, n - common + 1, c, common)[: (n + 63) // 64], n]
    degs, gs = _gcd(engine, [tuple(pair)], 64)
    d, g = int(degs[0]), gs[0]
    assert d >= common - 1
    if d == common - 1:
        assert (g[: c.size] == c).all() and not g[c.size:].any()
    else:                       # a further common factor by chance: c divides the gcd
        q = engine.engine.gcd_batch([(engine.DeviceBuffer.from_array(g), d + 1,
                                      engine.DeviceBuffer.from_array(c), common)])[0]
        assert int(q[0]) == common - 1
