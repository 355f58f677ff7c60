"""The Davidson's captured iteration holds the addresses of sigma's scratch; a
solve after the plan was changed and changed back, with the scratch replaced
in between, must not run the old capture."""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu


def test_scratch_replaced_between_solves():
    s = jb.Space(10, 10)
    ints = make_integrals(10, 10, 43)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    v = np.random.default_rng(8).standard_normal((1, s.ndets))
    opts = dict(maxiter=300, krymin=4, krymax=16, nroots=2, refdim=8, restol=1e-9)
    blocks, wide = (6, 0, 2, 6), (6, 0, 2, 5)  # 64-column blocks of E; all columns at once
    s.set_sigma_plan(jb.FP64, *blocks)
    a = s.davidson(**opts)
    s.set_sigma_plan(jb.FP64, *wide)
    s.sigma(v)  # E grows
    s.set_sigma_plan(jb.FP64, *blocks)
    b = s.davidson(**opts)
    assert np.array_equal(a.energies, b.energies)
    assert np.array_equal(a.civec, b.civec)
    s.close()
