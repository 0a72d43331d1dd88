"""Fused squaring passes (csrc/frobenius.cu) below the L2 size, and states on 8
bytes only, which keep the one-squaring kernel, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("r,n", [(30011, 64), (30011, 70), (99767, 24), (999961, 3), (2100001, 1)])
def test_small_batches(engine, oracle, r, n, shift):
    rng = np.random.default_rng(r + n)
    nw = (r + 63) // 64
    stride = nw + (nw & 1)
    st = np.zeros((n, stride), dtype=np.uint64)
    st[:, :nw] = rng.integers(0, 1 << 64, size=(n, nw), dtype=np.uint64)
    st[:, nw - 1] &= np.uint64((1 << (r % 64)) - 1)
    s = rng.integers(1, (r - 1) // 2 + 1, size=n).astype(np.uint64)
    a, b = engine.DeviceBuffer(st.nbytes + 16), engine.DeviceBuffer(st.nbytes + 16)
    a.upload(st.reshape(-1), offset_bytes=shift)
    ds = engine.DeviceBuffer.from_array(s)
    for k in (2, 5):
        engine.trin_square_batch(a.ptr + shift, b.ptr + shift, stride, n, r, ds, k)
    got = a.to_numpy(n * stride, offset_bytes=shift).reshape(n, stride)
    for i in range(0, n, max(1, n // 7)):
        assert (got[i, :nw] == oracle.trin_square_k(st[i, :nw].copy(), r, int(s[i]), 7)).all(), i
