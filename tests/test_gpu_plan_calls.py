"""Pinning the sigma plan (jci_sigma_tuning -> jci_sigma_set_plan): the values
that one run reports are accepted by the next, and arguments that no plan has
are refused."""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu


def _space(*general):
    s = jb.Space(*general)
    ints = make_integrals(s.norb, s.norb, 41)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    return s


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("general", [(6, 6), (8, 8)])  # one dense product; a tuned plan
def test_reported_plan_can_be_pinned(general, prec):
    a, b = _space(*general), _space(*general)
    v = np.random.default_rng(4).standard_normal((2, a.ndets))
    ref = a.sigma(v, prec)
    plan = a.sigma_tuning(prec)[:4]
    assert (plan == (0, 0, 0, 0)) == (a.ndets <= 2048)
    b.set_sigma_plan(prec, *plan)
    assert np.array_equal(b.sigma(v, prec), ref)
    assert b.sigma_tuning(prec)[:4] == plan
    # another plan and back
    b.set_sigma_plan(prec, 0, 128, 1, 1)
    b.sigma(v, prec)
    b.set_sigma_plan(prec, *plan)
    assert np.array_equal(b.sigma(v, prec), ref)
    a.close()
    b.close()


@pytest.mark.parametrize("general", [(6, 6), (8, 8)])
def test_threads_that_no_plan_has(general):
    s = _space(*general)
    refused = [(m, t, 1, 1) for m in (0, 1, 2, 3, 4, 5) for t in (0, -128, 100)]
    refused += [(6, -1, 0, 1), (7, -1, 16, 1)]
    if s.ndets > 2048:
        refused.append((0, 0, 0, 0))
    for plan in refused:
        for prec in (jb.FP64, jb.FP32):
            with pytest.raises(jb.JciError) as ei:
                s.set_sigma_plan(prec, *plan)
            assert ei.value.status == 1, plan
    s.close()
