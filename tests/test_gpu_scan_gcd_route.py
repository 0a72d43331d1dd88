"""Interval gcds of many resident s at r from 150000 bits on
(csrc/scanner.cu): the quadratic kernel where its waves are shorter than the
half-gcd's parts, the half-gcd else; the same results either way."""
import numpy as np
import pytest

from kernel_names import kernel_counts, launched

pytestmark = pytest.mark.gpu


def _gcd_kernels(engine, monkeypatch, r, slots):
    monkeypatch.setenv("GF2E_HGCD_STREAMS", "1")         # half-gcds from this thread
    S = engine.engine.Scanner(r, slots)
    S.submit(r // 3 + np.arange(slots), 30, 10**6, 1, 1)       # residues of full degree
    names = kernel_counts(lambda: S.step(1))
    S.close()
    return launched(names, "k_hgcd_base") > 0, launched(names, "k_gcd_smem") > 0


# below 150000 bits always quadratic; 409536 bits are the most that fit
@pytest.mark.parametrize("r,slots,half", [(149999, 3, False), (150001, 3, True), (160001, 64, True),
                                          (160001, 65, False), (300001, 65, False),
                                          (399999, 65, False), (400001, 65, True),
                                          (400001, 129, False), (409537, 129, True)])
def test_route(engine, monkeypatch, r, slots, half):
    # (the half-gcd ends with quadratic gcds of what it leaves)
    got = _gcd_kernels(engine, monkeypatch, r, slots)
    assert got[0] == half, got
    assert half or got[1]


def test_same_results(engine):
    E = engine.engine
    r, s = 160001, 50000 + np.arange(100)
    many = E.scan(r, s, 30, 37, L0=4, batch=100)
    assert many == E.scan(r, s, 30, 37, L0=4, batch=25)
    assert any(" p" in line for line in many)
