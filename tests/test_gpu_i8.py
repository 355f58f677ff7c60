"""The alpha-single x beta-single product on the integer tensor cores
(jci_fci_i8.cu, product engine 128) and the plan that splits the singles
between the hole-string products and k_coulomb (plan 7, threads 1).

Against the oracle's sigma at the edges of their tiles: spaces of one and of
many 48-column chunks, with the last chunk nearly empty or full, one and two
32-wide steps of singles, panel rows in one to four quarters of tensor
memory, alpha and beta spaces of different size, rows of odd length (no
16-byte copies), orbitals common to every string.  Bars of the other sigma
tests: FP64 1e-12, FP32 2e-6 of the largest |sigma|.
"""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}
PLANS = [(5, 128, 128, 1), (7, 1, 128, 5), (7, 1, 128, 6)]
# general: electrons, orbitals, nfrozen, ndocc, nactive, nfrzvirt, xlevel
SPACES = [(6, 6, 0, 0, 6, 0, 0),      # 20 x 20: one chunk, 9 singles
          (7, 7, 0, 0, 7, 0, 0),      # odd electrons
          (8, 9, 0, 0, 9, 0, 0),      # 126 strings
          (13, 9, 0, 0, 9, 0, 0),     # more electrons than orbitals
          (10, 10, 0, 0, 10, 0, 0),   # 252 strings, 25 singles
          (11, 11, 0, 0, 11, 0, 0),   # 462 x 462, 30 singles: one 32-wide step
          (10, 10, 0, 2, 6, 0, 0),    # orbitals of every string
          (7, 13, 0, 0, 13, 0, 0)]    # 715 x 286: 36 singles, 78 pairs


def _space(general, seed=31):
    from oracle.oracle import OracleSpace
    s = jb.Space(*general)
    ints = make_integrals(s.norb, s.norb, seed)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    o = OracleSpace(s.na, s.nb, s.norb, ndocc=general[3], nactv=general[4])
    return s, o, m1, m2


def _sigma(s, v, prec):
    import torch
    dt = torch.float64 if prec == jb.FP64 else torch.float32
    x = torch.as_tensor(v).to(device="cuda", dtype=dt)
    y = torch.full_like(x, float("nan"))
    s.sigma_device(x.data_ptr(), y.data_ptr(), 1, s.ndets, prec, 0)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def _plans(s, prec):
    """The plans of PLANS that the space can run (at least the split one)."""
    ok = []
    for p in PLANS:
        try:
            s.set_sigma_plan(prec, *p)
            ok.append(p)
        except jb.JciError as e:
            assert e.status == 1
    assert ok
    return ok


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("general", SPACES)
def test_i8_against_oracle(general, prec):
    s, o, m1, m2 = _space(general)
    rng = np.random.default_rng(5)
    v = rng.standard_normal(s.ndets)
    # a few large elements: chunks whose columns keep exponents of their own
    w = 1e-7 * rng.standard_normal(s.ndets)
    w[rng.integers(0, s.ndets, 3)] = 1.0
    for x in (v, w):
        ref = o.sigma(m1, m2, x[None, :])[0]
        for plan in _plans(s, prec):
            s.set_sigma_plan(prec, *plan)
            y = _sigma(s, x, prec)
            assert np.abs(y.astype(np.float64) - ref).max() <= BAR[prec] * np.abs(ref).max(), plan
            assert np.array_equal(_sigma(s, x, prec), y), plan
    s.close()


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
def test_i8_special_vectors(prec):
    """A zero vector, one unit vector, a vector with an infinity and a NaN."""
    s, o, m1, m2 = _space((8, 9, 0, 0, 9, 0, 0))
    n, nb = s.ndets, s.nbstr
    unit = np.zeros(n)
    unit[7 * nb + 50] = 1.0
    bad = np.random.default_rng(6).standard_normal(n)
    bad[3 * nb + 60], bad[90 * nb + 2] = np.inf, np.nan
    ref = o.sigma(m1, m2, unit[None, :])[0]
    for plan in _plans(s, prec):
        s.set_sigma_plan(prec, *plan)
        assert not _sigma(s, np.zeros(n), prec).any(), plan
        y = _sigma(s, unit, prec).astype(np.float64)
        assert np.abs(y - ref).max() <= BAR[prec] * np.abs(ref).max(), plan
        # every element that the Hamiltonian connects to them is not finite
        y = _sigma(s, bad, prec)
        for d in (3 * nb + 60, 90 * nb + 2):
            e = np.zeros(n)
            e[d] = 1.0
            hit = np.abs(o.sigma(m1, m2, e[None, :])[0]) > 0
            assert not np.isfinite(y[hit]).any(), plan
    s.close()


def test_i8_plan_refused():
    """threads 1 needs the integer engine and the hole-string doubles."""
    s, _, _, _ = _space((8, 9, 0, 0, 9, 0, 0))
    for plan in ((7, 1, 16, 5), (7, 1, 128, 2), (6, 1, 0, 5)):
        with pytest.raises(jb.JciError):
            s.set_sigma_plan(jb.FP64, *plan)
    s.close()
