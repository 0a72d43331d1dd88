"""GF2E_FFT_TAYLOR gives products the word passes of the plan it forces, as it
does single transforms, at every size: gf2e_mul then leaves the product's
coefficients in its first scratch buffer (the sliced transform and the cluster
product leave something else there), half-gcds use the same plans, and
products and gcds agree with the oracle.  Plans are cached per process, so each
setting runs in its own."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
sys.path[:0] = [%(root)r, %(root)r + "/tests"]
import numpy as np
from kernel_names import kernel_counts, launched
import mersenne_trinomial_b200 as M
from mersenne_trinomial_b200 import engine as E
from mersenne_trinomial_b200 import workloads as W
from oracle import oracle as O
for ab, bb in %(sizes)r:
    a, b = W.random_bits(ab, 3), W.random_bits(bb, 4)
    m = E.fft_m_for(ab, bb)
    F = M.CudaFFT()
    F.init(m)
    ow = E.mul_out_words(ab, bb)
    da, db = M.DeviceBuffer.from_array(a), M.DeviceBuffer.from_array(b)
    out, fa, fb = M.DeviceBuffer(8 * ow), M.DeviceBuffer(8 << m), M.DeviceBuffer(8 << m)
    E.gf2x_fft_mul_dev(F, da, ab, db, bb, out, fa, fb)
    got, f = out.to_numpy(ow), fa.to_numpy(1 << m)
    want = O.fft_mul(a, ab, b, bb)
    assert (got[: want.size] == want).all(), ("mul", ab, bb)
    words = np.zeros((1 << m) + 2, dtype=np.uint32)          # 32-bit words of the sum
    words[: 1 << m] = (f & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    words[1 : (1 << m) + 1] ^= (f >> np.uint64(32)).astype(np.uint32)
    n = min(words.size, 2 * ow) // 2 * 2
    assert (words[:n].view(np.uint64) == got[: n // 2]).all(), ("coefficients", ab, bb)
    F.fini()
pairs, plain = [], []
for k in (1, 2):
    bits = 150000 + k
    a, b = W.random_bits(bits, k), W.random_bits(bits - 7, 10 + k)
    plain.append((a, b))
    pairs.append((M.DeviceBuffer.from_array(a), bits, M.DeviceBuffer.from_array(b), bits - 7))
got = []
names = kernel_counts(lambda: got.append(E.gcd_large(pairs, g_cap_words=8, max_parallel=2)))
assert launched(names, "k_hgcd_base"), names
assert not launched(names, "k_bfly") and not launched(names, "k_slice"), names
for (a, b), d in zip(plain, got[0][0]):
    assert int(d) == O.poly_gcd(a, b)[0]
print("ok")
"""

SIZES = [(700, 5), (5000, 4900), (200_000, 199_000), (3_000_000, 1_000_000)]


@pytest.mark.parametrize("plan", ["tau", "cascade"])
def test_products_take_the_forced_plan(plan):
    env = dict(os.environ, GF2E_FFT_TAYLOR=plan)
    out = subprocess.run([sys.executable, "-c", SCRIPT % {"root": ROOT, "sizes": SIZES}], env=env,
                         capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("ok")
