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


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
def test_pinned_plan_on_a_callers_stream(prec):
    """The first sigma after jci_sigma_set_plan runs on a stream of the caller,
    which knows nothing of the handle's own: the plan's tables must be there.
    The bar is that of the other sigma tests."""
    import torch

    from oracle.oracle import OracleSpace
    ints = make_integrals(10, 10, 41)
    m1, m2 = ints.packed()
    o = OracleSpace(5, 5, 10)
    v = np.random.default_rng(5).standard_normal(252 * 252)
    ref = o.sigma(m1, m2, v[None, :])[0]
    bar = (1e-12 if prec == jb.FP64 else 2e-6) * np.abs(ref).max()
    x = torch.as_tensor(v).to(device="cuda",
                              dtype=torch.float64 if prec == jb.FP64 else torch.float32)
    torch.cuda.synchronize()
    ran = 0
    for plan in ((5, 1, 16, 1), (5, 1, 128, 1), (7, 1, 128, 5), (6, 0, 0, 5), (7, 128, 16, 3),
                 (6, 128, 66, 1), (6, 128, 18, 1)):
        s = jb.Space(10, 10)  # new tables for every plan
        s.set_integrals(m1, m2, ints.e_nuc, 0.0)
        try:
            s.set_sigma_plan(prec, *plan)
        except jb.JciError as e:
            assert e.status == 1
            s.close()
            continue
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            y = torch.full_like(x, float("nan"))
        s.sigma_device(x.data_ptr(), y.data_ptr(), 1, s.ndets, prec, st.cuda_stream)
        torch.cuda.synchronize()
        assert np.abs(y.double().cpu().numpy() - ref).max() <= bar, plan
        s.close()
        ran += 1
    assert ran >= 5
