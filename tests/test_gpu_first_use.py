"""The first calls of a process, which make their plans: the twiddle tables are
on the device before a kernel on any stream reads them.  Transforms of one pass
and products by word passes, whose first kernel reads them, on the batch's own
streams and on a caller's non-blocking one, against the oracle."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
sys.path.insert(0, %(root)r)
import numpy as np
import torch
import mersenne_trinomial_b200 as M
from mersenne_trinomial_b200 import engine as E
from mersenne_trinomial_b200 import workloads as W
from oracle import oracle as O
torch.zeros(1, device="cuda")
stream = torch.cuda.Stream()                     # non-blocking
buf = M.DeviceBuffer.from_array
sizes = [(40 << m, 21 << m) for m in range(10)]
ops = [(W.random_bits(a, a), W.random_bits(b, b + 1)) for a, b in sizes]
dev = [(buf(x), buf(y), M.DeviceBuffer(8 * M.mul_out_words(a, b)))
       for (a, b), (x, y) in zip(sizes, ops)]
f = [W.splitmix64(m, 1 << m) for m in range(2, 11)]
df = [buf(x) for x in f]
torch.cuda.synchronize()
M.mul_batch_dev([(x, a, y, b, o) for (x, y, o), (a, b) in zip(dev, sizes)])
def check(what):
    torch.cuda.synchronize()
    for (a, b), (x, y), d in zip(sizes, ops, dev):
        want = O.comb_mul(x, a, y, b)
        assert (d[2].to_numpy(M.mul_out_words(a, b))[: want.size] == want).all(), (what, a, b)
        d[2].upload(np.zeros(M.mul_out_words(a, b), dtype=np.uint64))
check("batch")
for x, d in zip(f, df):
    F = M.CudaFFT()
    F.init(x.size.bit_length() - 1)
    F.fwd(d, stream=stream.cuda_stream)
    torch.cuda.synchronize()
    assert (d.to_numpy(x.size) == O.fft_fwd(x, x.size.bit_length() - 1)).all(), x.size
a, b = sizes[0]
assert M.lib().gf2e_mul_noalloc(dev[0][0].ptr, a, dev[0][1].ptr, b, dev[0][2].ptr,
                                stream.cuda_stream) == 0
torch.cuda.synchronize()
want = O.comb_mul(ops[0][0], a, ops[0][1], b)
assert (dev[0][2].to_numpy(M.mul_out_words(a, b))[: want.size] == want).all()
print("ok")
"""


@pytest.mark.parametrize("run", range(3))
@pytest.mark.parametrize("words", [False, True])
def test_first_calls_of_a_process(run, words):
    env = dict(os.environ)
    if words:
        env["GF2E_FFT_TAYLOR"] = "cascade"              # every product by word passes
    out = subprocess.run([sys.executable, "-c", SCRIPT % {"root": ROOT}], env=env,
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("ok")
