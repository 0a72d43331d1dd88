"""Device memory a batch of half-gcds draws from its pool (csrc/hgcd.cu), against
what a scanner's footprint counts for one: 90 words a member and operand word.
The pool keeps what it has drawn, so a process that has run one batch shows its
most."""
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
from mersenne_trinomial_b200 import workloads as W
bits, n = %(bits)d, %(n)d
def operand(b, seed):
    x = W.random_bits(b, seed)
    x[(b - 1) >> 6] |= np.uint64(1 << ((b - 1) & 63))
    return M.DeviceBuffer.from_array(x)
pairs = [(operand(bits, 2 * k + 1), bits, operand(bits - 1, 2 * k + 2), bits - 1) for k in range(n)]
small = [(operand(100000, 1), 100000, operand(99999, 2), 99999)]
M.engine.gcd_large(small, max_parallel=1)            # kernels loaded, the pool made
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
degs, _, st = M.engine.gcd_large(pairs, max_parallel=n)
torch.cuda.synchronize()
print((before - torch.cuda.mem_get_info()[0]) / 8 / ((bits + 63) // 64) / n)
"""


# sizes where a batch draws the most of what it may
@pytest.mark.parametrize("bits,n", [(1_600_183, 64), (16_000_183, 16)])
def test_words_a_member(bits, n):
    out = subprocess.run([sys.executable, "-c", SCRIPT % {"root": ROOT, "bits": bits, "n": n}],
                         capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stdout + out.stderr
    assert 20 < float(out.stdout) < 90, out.stdout
