"""Fused squaring passes (csrc/frobenius.cu) where windows end inside a warp
tile, and the groups of the host-buffer call (csrc/trinomial.cu), against the
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one word to a few tiles (8192 bits of output a lane row, 16384 a warp tile),
# sizes around their multiples, s at both ends and in the middle
@pytest.mark.parametrize("r", [5, 63, 65, 127, 129, 4095, 4423, 16383, 16385, 32769, 49153])
def test_small_states(engine, oracle, r):
    half = (r - 1) // 2
    s = sorted({1, 2, min(3, half), max(1, half // 2), max(1, half - 1), half})
    nw = (r + 63) // 64
    stride = nw + (nw & 1)
    rng = np.random.default_rng(r)
    st = np.zeros((len(s), stride), dtype=np.uint64)
    st[:, :nw] = rng.integers(0, 1 << 64, size=(len(s), nw), dtype=np.uint64)
    if r % 64:
        st[:, nw - 1] &= np.uint64((1 << (r % 64)) - 1)
    a = engine.DeviceBuffer.from_array(st.reshape(-1))
    b = engine.DeviceBuffer(st.nbytes)
    ds = engine.DeviceBuffer.from_array(np.array(s, dtype=np.uint64))
    for k in (2, 4, 7):
        engine.trin_square_batch(a, b, stride, len(s), r, ds, k)
    got = a.to_numpy(st.size).reshape(st.shape)
    for i, si in enumerate(s):
        assert (got[i, :nw] == oracle.trin_square_k(st[i, :nw].copy(), r, si, 13)).all(), si


# single squarings: a word a thread up to 2^15 words, warp tiles above
@pytest.mark.parametrize("r", [5, 65, 129, 4423, 44687, 2097151, 2097153])
def test_single_squarings(engine, oracle, r):
    half = (r - 1) // 2
    nw = (r + 63) // 64
    stride = nw + (nw & 1)
    for s in sorted({1, 2, min(64, half), max(1, half // 3), max(1, half - 1), half}):
        st = np.zeros((1, stride), dtype=np.uint64)
        st[0, :nw] = np.random.default_rng(r + s).integers(0, 1 << 64, size=nw, dtype=np.uint64)
        if r % 64:
            st[0, nw - 1] &= np.uint64((1 << (r % 64)) - 1)
        a, b = engine.DeviceBuffer.from_array(st.reshape(-1)), engine.DeviceBuffer(st.nbytes)
        engine.trin_square_batch(a, b, stride, 1, r,
                                 engine.DeviceBuffer.from_array(np.array([s], dtype=np.uint64)), 1)
        want = oracle.trin_square_k(st[0, :nw].copy(), r, s, 1)
        assert (a.to_numpy(stride)[:nw] == want).all(), s


# whole batches in one group (below 48 MB), equal groups with a remainder,
# groups of one state, and shrinking groups (k > 128, 16 states and more);
# ends in either buffer (k odd, k/2 even and odd)
@pytest.mark.parametrize("r,n,k", [(20000003, 19, 5), (20000003, 21, 6), (20000003, 23, 131),
                                   (136279841, 3, 9), (300000007, 2, 4), (99767, 30, 129)])
def test_host_groups(engine, r, n, k):
    rng = np.random.default_rng(n)
    s = rng.integers(1, (r - 1) // 2 + 1, size=n).astype(np.uint64)
    nw = (r + 63) // 64
    got = engine.frobenius_host(r, s, k)
    # the same from resident states, whose passes are compared with the oracle above
    stride = nw + (nw & 1)
    st = np.zeros((1, stride), dtype=np.uint64)
    for i in {0, n // 2, n - 2, n - 1}:
        st[:] = 0
        st[0, 0] = 2
        a, b = engine.DeviceBuffer.from_array(st.reshape(-1)), engine.DeviceBuffer(st.nbytes)
        engine.trin_square_batch(a, b, stride, 1, r,
                                 engine.DeviceBuffer.from_array(s[i:i + 1].copy()), k)
        assert (got[i] == a.to_numpy(stride)[:nw]).all(), i
