"""gf2e_gcd_batch with results put where operands are, a job's own or another
job's: operands are read before any result is written (csrc/gcd.cu), whatever
kernel the sizes call for."""
import ctypes as C

import numpy as np
import pytest

from mersenne_trinomial_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 64 jobs, and more than the SMs hold at a time; one result per operand place
@pytest.mark.parametrize("n,bits", [(64, 900), (700, 900), (200, 30_000)])
@pytest.mark.parametrize("shift", [0, 1, 5])
def test_results_over_operands(engine, oracle, n, bits, shift):
    from mersenne_trinomial_b200._lib import GcdJob, call
    words = (bits + 63) // 64
    rng = np.random.default_rng(bits)
    a = rng.integers(0, 1 << 64, size=(n, words), dtype=np.uint64)
    b = rng.integers(0, 1 << 64, size=(n, words), dtype=np.uint64)
    if bits % 64:
        a[:, -1] &= np.uint64((1 << (bits % 64)) - 1)
        b[:, -1] &= np.uint64((1 << (bits % 64)) - 1)
    da, db = engine.DeviceBuffer.from_array(a.reshape(-1)), engine.DeviceBuffer.from_array(b.reshape(-1))
    jobs = (GcdJob * n)()
    for i in range(n):                       # job i's result over job (i + shift)'s a
        g = da.ptr + 8 * words * ((i + shift) % n)
        jobs[i] = GcdJob(da.ptr + 8 * words * i, bits, db.ptr + 8 * words * i, bits, g, words)
    need = C.c_size_t()
    call("gf2e_gcd_workspace_size", jobs, n, C.byref(need))
    ws = engine.DeviceBuffer(need.value)
    degs = np.zeros(n, dtype=np.int64)
    call("gf2e_gcd_batch", jobs, n, degs.ctypes.data, ws.ptr, ws.nbytes, None)
    got = da.to_numpy(n * words).reshape(n, words)
    for i in range(0, n, max(1, n // 40)):
        d, g = oracle.poly_gcd(a[i], b[i])
        assert int(degs[i]) == d, i
        assert (got[(i + shift) % n] == np.asarray(g, dtype=np.uint64)[:words]).all(), i
