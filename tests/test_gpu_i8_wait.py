"""The bounded waits of the digit product (jci_fci_i8.cu): a chunk that is
never handed over (jci_test_expire_next_wait) makes every role give up after
about a second; the kernel returns, the host reads JCI_ERR_TIMEOUT, and the
next sigma on the same space is right again."""
import ctypes
import time

import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}


def _space():
    s = jb.Space(10, 10)
    ints = make_integrals(10, 10, 46)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    f = jb.lib().jci_test_expire_next_wait
    f.argtypes = [ctypes.c_void_p]
    return s, lambda: f(s.h)


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("graded", [False, True])
def test_host_call(prec, graded):
    s, arm = _space()
    v = np.random.default_rng(2).standard_normal(s.ndets)
    if graded:  # the strings whose digits the product cuts itself
        v *= 1e-9
        v[::5003] = 1.0
    s.set_sigma_plan(prec, 5, 128, 16, 1)
    ref = s.sigma(v[None, :], prec)[0]
    s.set_sigma_plan(prec, 5, 128, 128, 1)
    bar = BAR[prec] * np.abs(ref).max()
    assert np.abs(s.sigma(v[None, :], prec)[0] - ref).max() <= bar
    assert arm() == 0
    t0 = time.time()
    with pytest.raises(jb.JciError) as e:
        s.sigma(v[None, :], prec)
    assert e.value.status == 10  # JCI_ERR_TIMEOUT
    assert 0.5 < time.time() - t0 < 60
    for _ in range(2):
        assert np.abs(s.sigma(v[None, :], prec)[0] - ref).max() <= bar
    s.close()


def test_device_call():
    """jci_sigma_device returns before its kernels have run; the next call on
    the handle reports the wait, without synchronising."""
    import torch
    s, arm = _space()
    x = torch.randn(s.ndets, dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(3))
    ref, y = torch.empty_like(x), torch.empty_like(x)
    s.set_sigma_plan(jb.FP64, 5, 128, 128, 1)

    def call(out):
        s.sigma_device(x.data_ptr(), out.data_ptr(), 1, s.ndets, jb.FP64, 0)

    call(ref)
    torch.cuda.synchronize()
    assert arm() == 0
    call(y)
    torch.cuda.synchronize()
    with pytest.raises(jb.JciError) as e:
        call(y)
    assert e.value.status == 10
    y.fill_(0)
    call(y)
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    s.close()
