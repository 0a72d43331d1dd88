"""The bodies of the bit-sliced product's kernels
(mersenne_trinomial_b200/csrc/slicefft.cuh) on the host, compiled with address
and undefined-behaviour checks where the compiler has them, against the
oracle's products: separate launches of 2^10 .. 2^19 coefficients (no rows, and
2 to 8 rows of 2^16; tops and low passes of each kind) and the cluster product
of 2^10 .. 2^14, with balanced, uneven and tiny operands and the first chunk
flipped as the scanner's running product does."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from mersenne_trinomial_b200 import workloads as W

CSRC = os.path.join(ROOT, "mersenne_trinomial_b200", "csrc")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = os.path.join(tmp_path_factory.mktemp("slice"), "slicefft_driver")
    base = ["g++", "-O1", "-std=c++17", "-Wno-unknown-pragmas", "-I", CSRC, "-o", exe,
            os.path.join(ROOT, "tests", "slicefft_driver.cpp")]
    checked = base + ["-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
    if subprocess.run(checked, capture_output=True, timeout=900).returncode != 0:
        subprocess.run(base, check=True, timeout=900)
    return exe


def _run(driver, tmp, jobs):
    """jobs: (kind, m, plog, abits, bbits, xor0); the products of random operands."""
    recs, words = [], []
    for i, (kind, m, plog, ab, bb, xor0) in enumerate(jobs):
        a, b = W.random_bits(ab, 100 + i), W.random_bits(bb, 200 + i)
        ca, cb, ow = (ab + 31) // 32, (bb + 31) // 32, ((ab + bb + 63) >> 6) + 1
        assert ca + cb - 1 <= 1 << m
        recs.append(np.concatenate([np.array([kind, m, plog, ca, cb, xor0, ow], dtype=np.uint64), a, b]))
        words.append(ow)
    np.concatenate(recs).tofile(os.path.join(tmp, "in"))
    subprocess.run([driver, os.path.join(tmp, "in"), os.path.join(tmp, "out")], check=True, timeout=900)
    got = np.fromfile(os.path.join(tmp, "out"), dtype=np.uint64)
    at = 0
    for ow in words:
        yield got[at:at + ow]
        at += ow
    assert at == got.size


def _check(oracle, driver, tmp, jobs):
    for (kind, m, plog, ab, bb, xor0), got, i in zip(jobs, _run(driver, tmp, jobs), range(len(jobs))):
        a, b = W.random_bits(ab, 100 + i), W.random_bits(bb, 200 + i)
        a[0] ^= np.uint64(xor0)
        w = oracle.fft_mul(a, ab, b, bb) if ab * bb > 10**8 else oracle.comb_mul(a, ab, b, bb)
        assert (got[: w.size] == w).all() and not got[w.size:].any(), (kind, m, plog, ab, bb)


def _sizes(m):
    n = 32 << m
    return [(n // 2 - 5, n // 2 - 40), (9000, n - 9100) if m > 10 else (3000, n - 3100), (n - 100, 33),
            (1, 1), (100, 77)]


@pytest.mark.parametrize("m", [10, 11, 12, 13, 14])
def test_cluster_products(oracle, driver, tmp_path, m):
    _check(oracle, driver, tmp_path, [(1, m, 0, ab, bb, x) for ab, bb in _sizes(m) for x in (0, 2)
                                      if ab > 1 or not x])


@pytest.mark.parametrize("m,plogs", [(10, (2, 3)), (13, (2, 3)), (14, (3,)), (15, (2, 3)), (16, (3,)),
                                     (17, (2, 3))])
def test_separate_launches(oracle, driver, tmp_path, m, plogs):
    _check(oracle, driver, tmp_path, [(0, m, p, ab, bb, 2 if ab > 1 else 0) for ab, bb in _sizes(m)
                                      for p in plogs])


@pytest.mark.parametrize("m", [18, 19])
def test_rows_above_2_16(oracle, driver, tmp_path, m):
    n = 32 << m
    _check(oracle, driver, tmp_path, [(0, m, 3, n // 2 - 5, n // 2 - 40, 0),
                                      (0, m, 3, 32 * 70_000, n - 32 * 70_000 - 11, 2)])
