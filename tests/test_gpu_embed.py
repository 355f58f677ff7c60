"""Truncated spaces large enough for sigma through the full CI space
(jci_embed.cu; which of the two ways a space takes is timed, both must be
right): several occupation groups per spin, odd electrons, a frozen core, one
and several vectors, and integrals set again after the first sigma, against
the oracle at the bars of the other sigma tests."""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}


@pytest.mark.parametrize("general", [(11, 12, 0, 1, 7, 0, 2),    # 117 600 of 731 808
                                     (12, 12, 1, 2, 6, 0, 2),    # frozen core, 2 DOCC
                                     (8, 12, 0, 1, 8, 0, 1)])    # 50 960 of 245 025
def test_truncated_space_through_full_space(general):
    from oracle.oracle import OracleSpace
    s = jb.Space(*general)
    assert s.ndets > 16384 and s.npq > 1
    o = OracleSpace(s.na, s.nb, s.norb, general[3], general[4], general[6])
    rng = np.random.default_rng(3)
    v = rng.standard_normal((3, s.ndets))
    for seed in (21, 22):  # the second set replaces the first in the same handle
        ints = make_integrals(s.norb, s.norb, seed)
        m1, m2 = ints.packed()
        s.set_integrals(m1, m2, ints.e_nuc, 0.0)
        ref = o.sigma(m1, m2, v)
        for prec in (jb.FP64, jb.FP32):
            y = s.sigma(v, prec)
            assert np.abs(y - ref).max() <= BAR[prec] * np.abs(ref).max()
            assert np.array_equal(s.sigma(v, prec), y)
    s.close()
