"""Autotuning with little device memory: a plan whose scratch finds no room is
dropped, and the first sigma takes another one instead of failing."""
import ctypes

import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
# none; the digits but not the transposes; the transposes but no large E block
@pytest.mark.parametrize("limit", [0, 9 << 20, 20 << 20])
def test_plans_without_room_are_dropped(limit, prec):
    ints = make_integrals(12, 12, 44)
    m1, m2 = ints.packed()
    v = np.random.default_rng(9).standard_normal((1, 924 * 924))
    ref = None
    for cap in (None, limit):
        s = jb.Space(12, 12)
        s.set_integrals(m1, m2, ints.e_nuc, 0.0)
        if cap is not None:
            assert jb.lib().jci_test_limit_scratch(s.h, ctypes.c_size_t(cap)) == 0
        y = s.sigma(v, prec)
        if ref is None:
            ref = y
        assert np.abs(y - ref).max() <= BAR[prec] * np.abs(ref).max()
        assert np.array_equal(s.sigma(v, prec), y)
        assert s.sigma_tuning(prec)[1] != 0 or s.sigma_tuning(prec)[0] in (6, 7)
        s.close()


def test_pinned_plan_without_room():
    """The digits of a pinned plan are refused as a lack of memory, not as a
    plan that does not exist, and the handle works as before."""
    s = jb.Space(10, 10)
    ints = make_integrals(10, 10, 44)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    assert jb.lib().jci_test_limit_scratch(s.h, ctypes.c_size_t(0)) == 0
    with pytest.raises(jb.JciError) as ei:
        s.set_sigma_plan(jb.FP64, 5, 128, 128, 1)
    assert ei.value.status == 3
    v = np.random.default_rng(9).standard_normal((1, s.ndets))
    y = s.sigma(v)
    assert jb.lib().jci_test_limit_scratch(s.h, ctypes.c_size_t(1 << 40)) == 0
    s.set_sigma_plan(jb.FP64, 5, 128, 128, 1)
    z = s.sigma(v)
    assert np.abs(z - y).max() <= 1e-12 * np.abs(y).max()
    s.close()
