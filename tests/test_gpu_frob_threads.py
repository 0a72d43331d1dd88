"""Chained squaring passes (csrc/frobenius.cu) of two threads on one stream: the
launch before a pass need not be of the same call, whose states it must still
find finished."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,n,k", [(4423, 5, 40), (99767, 24, 24), (999961, 3, 21)])
def test_two_threads_on_one_stream(engine, oracle, r, n, k):
    nw = (r + 63) // 64
    stride = nw + (nw & 1)
    half = (r - 1) // 2
    stream = torch.cuda.Stream()
    sets = []
    for t in range(2):
        rng = np.random.default_rng(r + t)
        st = np.zeros((n, stride), dtype=np.uint64)
        st[:, :nw] = rng.integers(0, 1 << 64, size=(n, nw), dtype=np.uint64)
        st[:, nw - 1] &= np.uint64((1 << (r % 64)) - 1)
        s = rng.integers(1, half + 1, size=n).astype(np.uint64)
        sets.append((st, s, engine.DeviceBuffer.from_array(st.reshape(-1)), engine.DeviceBuffer(st.nbytes),
                     engine.DeviceBuffer.from_array(s)))
    torch.cuda.synchronize()
    start, failed = threading.Barrier(2), []

    def work(t):
        try:
            _, _, a, b, ds = sets[t]
            start.wait(30)
            for _ in range(3):
                engine.trin_square_batch(a, b, stride, n, r, ds, k, stream=stream.cuda_stream)
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    torch.cuda.synchronize()
    for st, s, a, _, _ in sets:
        got = a.to_numpy(st.size).reshape(st.shape)
        for i in range(n):
            want = oracle.trin_square_k(st[i, :nw].copy(), r, int(s[i]), 3 * k)
            assert (got[i, :nw] == want).all(), i
