"""Elements of sigma, one by one, for vectors whose elements lie decades apart:
the 8-bit digit product (jci_fci_i8.cu, engine 128) beside the floating
product engine 16.

A floating sum of sigma_i = sum_j H_ij c_j has an error of a few roundings of
sum_j |H_ij| |c_j|, however small that is beside the largest |sigma|; digits cut
relative to the largest element of a whole column do not.  The bars are 1e-13
(FP64) and 1e-5 (FP32) of sum_j |H_ij| |c_j|: some thousand terms at one
rounding each, 1000 x 1.1e-16 and 170 x 6e-8.  Rows that the large elements
do not reach are the ones at stake: there the digits of a column once left
1e-7 (FP64, elements 1e-10 of the large ones) and 2e-4 (FP32, 1e-6).
"""
import functools

import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-13, jb.FP32: 1e-5}
GENERAL = {"many chunks": (8, 9, 0, 0, 9, 0, 0),      # 126 x 126 strings, 20 singles
           "two steps": (5, 16, 0, 0, 16, 0, 0)}      # 560 x 120, 39 singles
ROWS = {"many chunks": 80, "two steps": 24}


@functools.lru_cache(maxsize=None)
def _rows(name):
    """Sampled rows of H (exact to the oracle's rounding of each element)."""
    from oracle.oracle import OracleSpace
    s = jb.Space(*GENERAL[name])
    ints = make_integrals(s.norb, s.norb, 31)
    m1, m2 = ints.packed()
    o = OracleSpace(s.na, s.nb, s.norb)
    rng = np.random.default_rng(12)
    rows = np.sort(rng.choice(s.ndets, ROWS[name], replace=False))
    H = np.zeros((len(rows), s.ndets))
    for k, i in enumerate(rows):
        e = np.zeros((1, s.ndets))
        e[0, i] = 1.0
        H[k] = o.sigma(m1, m2, e)[0]  # H is symmetric
    return s, m1, m2, rows, H


def _vector(s, H, kind, prec):
    rng = np.random.default_rng(13)
    g = rng.standard_normal(s.ndets)
    if kind == "spikes":  # three large elements
        w = (1e-10 if prec == jb.FP64 else 1e-6) * g
        w[rng.integers(0, s.ndets, 3)] = 1.0
    elif kind == "strings":  # every alpha and beta string a weight of its own, as in a CI vector
        w = (g.reshape(s.nastr, s.nbstr) * 10.0 ** -rng.uniform(0, 5, s.nastr)[:, None]
             * 10.0 ** -rng.uniform(0, 5, s.nbstr)[None, :]).ravel()
    else:  # every element a weight of its own
        w = g * 10.0 ** -rng.uniform(0, 10, s.ndets)
    return w if prec == jb.FP64 else w.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("kind", ["spikes", "strings", "elements"])
@pytest.mark.parametrize("name", list(GENERAL))
def test_small_elements(name, kind, prec):
    import torch
    s, m1, m2, rows, H = _rows(name)
    v = _vector(s, H, kind, prec)
    ref = (H.astype(np.longdouble) * v).sum(axis=1).astype(np.float64)
    scale = (np.abs(H) * np.abs(v)).sum(axis=1)
    if kind == "spikes":
        large = np.abs(v) == 1.0
        assert (~(H[:, large] != 0).any(axis=1)).sum() > len(rows) // 4
    sp = jb.Space(*GENERAL[name])
    ints = make_integrals(sp.norb, sp.norb, 31)
    sp.set_integrals(m1, m2, ints.e_nuc, 0.0)
    dt = torch.float64 if prec == jb.FP64 else torch.float32
    x = torch.as_tensor(v).to(device="cuda", dtype=dt)
    ran = 0
    for plan in ((5, 128, 16, 1), (5, 128, 128, 1), (5, 1, 128, 1), (7, 1, 128, 5)):
        try:
            sp.set_sigma_plan(prec, *plan)
        except jb.JciError as e:
            assert e.status == 1 and (plan[2] != 128 or plan[0] == 7)
            continue
        y = torch.full_like(x, float("nan"))
        sp.sigma_device(x.data_ptr(), y.data_ptr(), 1, sp.ndets, prec, 0)
        torch.cuda.synchronize()
        got = y.double().cpu().numpy()[rows]
        worst = (np.abs(got - ref) / scale).max()
        print(f"{name} {kind} {plan} {worst:.2e}")
        assert worst <= BAR[prec], (plan, worst)
        ran += 1
    assert ran >= 3
    sp.close()
