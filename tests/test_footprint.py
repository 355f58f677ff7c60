"""Device memory that the solve server admits a request with
(jci_request_footprint): host arithmetic, and on a GPU what a solve really
takes."""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

TRUNCATED = (11, 12, 0, 1, 7, 0, 2)    # 117 600 determinants, 731 808 in the full space
LARGE = (12, 16, 0, 2, 10, 0, 2)       # 13 025 196 of 64 128 064
SPACES = [(6, 6, 0, 0, 6, 0, 0), (10, 10, 0, 0, 10, 0, 0), (12, 12, 0, 0, 12, 0, 0),
          (13, 13, 0, 0, 13, 0, 0), TRUNCATED, (8, 12, 0, 1, 8, 0, 1), (10, 10, 0, 2, 6, 0, 0)]


def test_full_space_is_counted():
    n, generic = jb.request_footprint(LARGE)
    assert not generic
    # the full space's vectors, transposes, digits and autotune vectors in FP64
    assert n > 64128064 * (16 + 16 + 16 + 7) + (4 << 30)
    assert jb.request_footprint(LARGE, precision=jb.MIXED)[0] > n + 64128064 * (8 + 8 + 4)


def test_one_group_plans_are_counted():
    # digits, both vectors of the autotuner, transposes, one E block
    n, _ = jb.request_footprint((14, 14, 0, 0, 14, 0, 0), krymax=8)
    assert n > 11778624 * (8 * 26 + 7 + 32) + (4 << 30)


def test_budgets():
    """Without room for the full space a truncated request keeps to the generic
    kernel; without room for the plans a request gets the whole budget; only
    panels and tables that exceed it are refused."""
    n, _ = jb.request_footprint(LARGE)
    small, generic = jb.request_footprint(LARGE, budget_bytes=n - 1)
    assert generic and small < n - 64128064 * 64
    assert jb.request_footprint(LARGE, budget_bytes=n) == (n, False)
    assert jb.request_footprint(LARGE, budget_bytes=small) == (small, True)
    with pytest.raises(jb.JciError) as ei:
        jb.request_footprint(LARGE, budget_bytes=small // 2)
    assert ei.value.status == 11
    one, _ = jb.request_footprint((14, 14, 0, 0, 14, 0, 0), krymax=8)
    assert jb.request_footprint((14, 14, 0, 0, 14, 0, 0), krymax=8,
                                budget_bytes=one - (1 << 30)) == (one - (1 << 30), False)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [jb.FP64, jb.MIXED])
@pytest.mark.parametrize("general", SPACES)
def test_solve_stays_within(general, precision):
    """What the device has less after a solve (and, for the larger spaces, while
    its plans were timed) is at most the footprint."""
    import torch
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    warm = jb.Space(4, 4)  # the library's own context and static arrays
    ints = make_integrals(4, 4, 1)
    m1, m2 = ints.packed()
    warm.set_integrals(m1, m2, ints.e_nuc, 0.0)
    warm.sigma(np.ones((1, warm.ndets)))
    free0, _ = torch.cuda.mem_get_info()
    s = jb.Space(*general)
    ints = make_integrals(s.norb, s.norb, 9)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    s.davidson(maxiter=12, krymin=4, krymax=24, nroots=1, refdim=8, restol=1e-12,
               precision=precision, block=True)
    torch.cuda.synchronize()
    used = free0 - torch.cuda.mem_get_info()[0]
    assert used <= jb.request_footprint(general, precision=precision)[0]
    s.close()
    warm.close()


@pytest.mark.gpu
def test_server_keeps_to_its_budget():
    """A budget without room for the full space: the request is admitted and
    solved, with the energies of one that has the room."""
    ints = make_integrals(12, 12, 9)
    m1, m2 = ints.packed()
    kw = dict(nroots=1, krymin=4, krymax=16, refdim=8, restol=1e-9)
    n, _ = jb.request_footprint(TRUNCATED, krymax=16)
    energies = []
    for budget in (n, n - 1):
        srv = jb.Server(budget_bytes=budget, slots=2)
        t = [srv.submit(TRUNCATED, m1, m2, ints.e_nuc, 0.0, **kw) for _ in range(2)]
        for k in t:
            r = srv.wait(k)
            assert r.status == 0 and r.converged
            energies.append(r.energies[0])
        srv.close()
    assert max(energies) - min(energies) < 1e-10
