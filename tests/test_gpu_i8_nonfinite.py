"""Infinities and NaN in c and among the integrals, through the digit product
(jci_fci_i8.cu, engine 128) beside the floating product engine 16: they reach
the elements of sigma that H connects to them, and no others.  Bars of the
other sigma tests for the others: FP64 1e-12, FP32 2e-6 of the largest |sigma|.
"""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}
PLANS = [(5, 128, 16, 1), (5, 128, 128, 1), (7, 1, 128, 5)]


def _index(p, q):  # packed pairs of 1-based orbitals, and of pairs
    p, q = max(p, q), min(p, q)
    return p * (p - 1) // 2 + q - 1


def _eri(i, j, k, l):
    a, b = _index(i, j), _index(k, l)
    a, b = max(a, b), min(a, b)
    return a * (a + 1) // 2 + b


def _setup():
    from oracle.oracle import OracleSpace
    s = jb.Space(8, 9)  # 126 x 126 strings, three chunks
    ints = make_integrals(9, 9, 31)
    m1, m2 = ints.packed()
    return s, OracleSpace(s.na, s.nb, s.norb), m1, m2


def _sigma(s, v, prec):
    import torch
    dt = torch.float64 if prec == jb.FP64 else torch.float32
    x = torch.as_tensor(v).to(device="cuda", dtype=dt)
    y = torch.full_like(x, 7.0)
    s.sigma_device(x.data_ptr(), y.data_ptr(), 1, s.ndets, prec, 0)
    torch.cuda.synchronize()
    return y.double().cpu().numpy()


def _check(y, hit, ref, prec, what):
    assert 0 < hit.sum() < len(hit)
    assert not np.isfinite(y[hit]).any(), what
    assert np.abs(y[~hit] - ref[~hit]).max() <= BAR[prec] * np.abs(ref).max(), what


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_integral(value, prec):
    s, o, m1, m2 = _setup()
    v = np.random.default_rng(6).standard_normal(s.ndets)
    t = _eri(2, 7, 4, 9)  # four orbitals: doubles only
    ref = o.sigma(m1, m2, v[None, :])[0]
    other = m2.copy()
    other[t] += 1.0
    hit = o.sigma(m1, other, v[None, :])[0] != ref
    other[t] = value
    s.set_integrals(m1, other, 0.0, 0.0)
    for plan in PLANS:
        s.set_sigma_plan(prec, *plan)
        _check(_sigma(s, v, prec), hit, ref, prec, plan)
    # and the same tables again with numbers
    s.set_integrals(m1, m2, 0.0, 0.0)
    for plan in PLANS:
        s.set_sigma_plan(prec, *plan)
        assert np.abs(_sigma(s, v, prec) - ref).max() <= BAR[prec] * np.abs(ref).max(), plan
    s.close()


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_element(value, prec):
    s, o, m1, m2 = _setup()
    v = np.random.default_rng(6).standard_normal(s.ndets)
    d = 3 * s.nbstr + 60
    v[d] = 0.0
    ref = o.sigma(m1, m2, v[None, :])[0]
    e = np.zeros((1, s.ndets))
    e[0, d] = 1.0
    hit = o.sigma(m1, m2, e)[0] != 0
    v[d] = value
    s.set_integrals(m1, m2, 0.0, 0.0)
    for plan in PLANS:
        s.set_sigma_plan(prec, *plan)
        _check(_sigma(s, v, prec), hit, ref, prec, plan)
    s.close()
