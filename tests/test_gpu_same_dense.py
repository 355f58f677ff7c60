"""The same-spin part of the one-group sigma as dense products
(jci_fci_dense.cu; plan 5, threads 1).

Against the oracle's sigma where a tile can go wrong: fewer strings than a
tile's rows, one string more than a tile, rows of odd length (no 16-byte
copies), alpha and beta spaces of different size, a spin without doubles,
orbitals common to every string, enough strings for the widest tile.  Bars of
the other sigma tests: FP64 1e-12, FP32 2e-6 of the largest |sigma|.
"""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}
# general: electrons, orbitals, nfrozen, ndocc, nactive, nfrzvirt, xlevel
SPACES = [(3, 6, 0, 0, 6, 0, 0),      # 15 x 6: less than a tile; beta has no doubles
          (7, 7, 0, 0, 7, 0, 0),      # 35 x 35: odd rows, a tile and a few
          (9, 9, 0, 0, 9, 0, 0),      # 126 x 126
          (13, 9, 0, 0, 9, 0, 0),     # more electrons than orbitals: 36 x 84
          (10, 10, 0, 2, 6, 0, 0),    # orbitals of every string
          (7, 13, 0, 0, 13, 0, 0),    # 715 x 286
          (11, 12, 0, 0, 12, 0, 0)]   # 924 x 792: the widest tile
ENGINES = (8, 16, 32, 64, 128)


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


def _engines(s, prec):
    ok = []
    for R in ENGINES:
        try:
            s.set_sigma_plan(prec, 5, 1, R, 1)
            ok.append(R)
        except jb.JciError as e:
            assert e.status == 1
    assert ok
    return ok


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("general", SPACES)
def test_same_dense_against_oracle(general, prec):
    s, o, m1, m2 = _space(general)
    x = np.random.default_rng(5).standard_normal(s.ndets)
    ref = o.sigma(m1, m2, x[None, :])[0]
    for R in _engines(s, prec):
        s.set_sigma_plan(prec, 5, 1, R, 1)
        y = _sigma(s, x, prec)
        assert np.abs(y.astype(np.float64) - ref).max() <= BAR[prec] * np.abs(ref).max(), R
        assert np.array_equal(_sigma(s, x, prec), y), R
    s.close()


def test_same_dense_follows_new_integrals():
    s, o, _, _ = _space((7, 7, 0, 0, 7, 0, 0))
    x = np.random.default_rng(7).standard_normal(s.ndets)
    s.set_sigma_plan(jb.FP64, 5, 1, 16, 1)
    _sigma(s, x, jb.FP64)
    ints = make_integrals(s.norb, s.norb, 32)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    s.set_sigma_plan(jb.FP64, 5, 1, 16, 1)
    ref = o.sigma(m1, m2, x[None, :])[0]
    assert np.abs(_sigma(s, x, jb.FP64) - ref).max() <= 1e-12 * np.abs(ref).max()
    s.close()


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
def test_same_dense_infinity_stays_with_its_neighbours(prec):
    """An infinity reaches the elements that the Hamiltonian connects to it, and
    no other through a product with zero."""
    s, o, m1, m2 = _space((9, 9, 0, 0, 9, 0, 0))
    x = np.random.default_rng(6).standard_normal(s.ndets)
    d = 3 * s.nbstr + 60
    x[d] = np.inf
    e = np.zeros(s.ndets)
    e[d] = 1.0
    hit = np.abs(o.sigma(m1, m2, e[None, :])[0]) > 0
    # the row and the column of the two dense products
    near = np.zeros((s.nastr, s.nbstr), bool)
    near[3], near[:, 60] = True, True
    y0 = x.copy()
    y0[d] = 0.0
    ref = o.sigma(m1, m2, y0[None, :])[0]
    for R in _engines(s, prec):
        if R == 128:  # its rows with an infinity are summed by another path
            continue
        s.set_sigma_plan(prec, 5, 1, R, 1)
        y = _sigma(s, x, prec).astype(np.float64)
        assert not np.isfinite(y[hit]).any(), R
        far = near.ravel() & ~hit
        assert far.any()
        assert np.abs(y[far] - ref[far]).max() <= BAR[prec] * np.abs(ref).max(), R
    s.close()
