"""Both routes of sigma for a truncated space (jci_sigma_route,
jci_sigma_set_route): each one forced, so that it is known which ran, against
the oracle at the bars of the other sigma tests; the reported route pinned in
another handle gives the same bits; a Davidson solve (captured iterations)
through the full space."""
import numpy as np
import pytest

import jayci_b200 as jb
from jayci_b200.synth import make_integrals

pytestmark = pytest.mark.gpu
BAR = {jb.FP64: 1e-12, jb.FP32: 2e-6}
GENERAL = (11, 12, 0, 1, 7, 0, 2)  # 117 600 of 731 808 determinants
GENERIC, FULL = 1, 2


def _space(general=GENERAL, seed=21):
    s = jb.Space(*general)
    ints = make_integrals(s.norb, s.norb, seed)
    m1, m2 = ints.packed()
    s.set_integrals(m1, m2, ints.e_nuc, 0.0)
    return s, m1, m2


@pytest.mark.parametrize("prec", [jb.FP64, jb.FP32])
@pytest.mark.parametrize("general", [GENERAL,
                                     (12, 12, 1, 2, 6, 0, 2),  # a frozen orbital, 2 DOCC
                                     (8, 12, 0, 1, 8, 0, 1)])  # 50 960 of 245 025
def test_each_route_against_oracle(general, prec):
    from oracle.oracle import OracleSpace
    s, m1, m2 = _space(general)
    o = OracleSpace(s.na, s.nb, s.norb, general[3], general[4], general[6])
    v = np.random.default_rng(3).standard_normal((2, s.ndets))
    ref = o.sigma(m1, m2, v)
    assert s.sigma_route(prec) == (0, 0, 0, 0, 0)
    s.sigma(v, prec)
    assert s.sigma_route(prec)[0] in (GENERIC, FULL)
    got = {}
    for route in (GENERIC, FULL, GENERIC):
        s.set_sigma_route(prec, route)
        y = s.sigma(v, prec)
        assert s.sigma_route(prec)[0] == route
        assert np.abs(y - ref).max() <= BAR[prec] * np.abs(ref).max(), route
        assert np.array_equal(s.sigma(v, prec), y), route
        assert route not in got or np.array_equal(got[route], y)
        got[route] = y
    # they sum in different orders, so equal bits would be one route run twice
    assert not np.array_equal(got[GENERIC], got[FULL])
    s.close()


@pytest.mark.parametrize("route", [GENERIC, FULL])
def test_reported_route_can_be_pinned(route):
    a, _, _ = _space()
    b, _, _ = _space()
    v = np.random.default_rng(4).standard_normal((1, a.ndets))
    a.set_sigma_route(jb.FP64, route)
    ref = a.sigma(v)
    r = a.sigma_route(jb.FP64)
    assert r[0] == route
    b.set_sigma_route(jb.FP64, *r)
    assert np.array_equal(b.sigma(v), ref)
    assert b.sigma_route(jb.FP64) == r
    a.close()
    b.close()


def test_davidson_through_each_route():
    """The captured iterations run the pinned route; changing it drops them."""
    s, _, _ = _space()
    opts = dict(maxiter=400, krymin=4, krymax=16, nroots=2, refdim=8, restol=1e-9)
    got = {}
    for route in (FULL, GENERIC, FULL):
        s.set_sigma_route(jb.FP64, route)
        r = s.davidson(**opts)
        assert s.sigma_route(jb.FP64)[0] == route
        if route in got:
            assert np.array_equal(got[route].energies, r.energies)
        got[route] = r
    assert np.abs(got[FULL].energies - got[GENERIC].energies).max() <= 1e-10
    ov = np.abs(np.einsum("ij,ij->i", got[FULL].civec, got[GENERIC].civec))
    assert (ov > 1 - 1e-9).all()
    s.close()


def test_routes_refused():
    s, _, _ = _space()
    for args in ((jb.MIXED, 1), (jb.FP64, 3), (jb.FP64, -1), (jb.FP64, 1, 0, 128, 1, 1),
                 (jb.FP64, 2, 8, 128, 1, 1), (jb.FP64, 2, 0, 100, 1, 1)):
        with pytest.raises(jb.JciError) as ei:
            s.set_sigma_route(*args)
        assert ei.value.status == 1, args
    s.close()
    one = jb.Space(8, 8)  # one group: plans, not routes
    with pytest.raises(jb.JciError) as ei:
        one.set_sigma_route(jb.FP64, 1)
    assert ei.value.status == 12  # before the integrals
    ints = make_integrals(8, 8, 3)
    m1, m2 = ints.packed()
    one.set_integrals(m1, m2, ints.e_nuc, 0.0)
    one.set_sigma_route(jb.FP64, 0)
    with pytest.raises(jb.JciError) as ei:
        one.set_sigma_route(jb.FP64, 1)
    assert ei.value.status == 1
    one.close()


def test_unused_full_space_is_let_go():
    """One precision on the generic kernel, the other never used: the full
    space's tables (over 100 MB here) do not stay with the handle."""
    import torch
    s, _, _ = _space()
    v = np.random.default_rng(6).standard_normal((1, s.ndets))
    s.set_sigma_route(jb.FP64, GENERIC)
    s.sigma(v)
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    s.set_sigma_route(jb.FP64, FULL)
    s.sigma(v)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] < free0 - (100 << 20)
    s.set_sigma_route(jb.FP64, GENERIC)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free0 - (16 << 20)
    s.close()


@pytest.mark.parametrize("route", [GENERIC, FULL])
@pytest.mark.parametrize("captured", [False, True])
def test_two_streams_of_one_handle(route, captured):
    """One thread queues sigmas of different vectors on two streams, as it could
    when every truncated sigma was the scratch-free kernel; also as replays of
    two captured graphs."""
    import torch
    s, _, _ = _space()
    s.set_sigma_route(jb.FP64, route)
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(6, s.ndets, generator=g, dtype=torch.float64, device="cuda")
    ref = torch.empty_like(x)
    for k in range(6):
        s.sigma_device(x[k].data_ptr(), ref[k].data_ptr(), 1, s.ndets, jb.FP64, 0)
    torch.cuda.synchronize()
    y = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def call(k, st):
        s.sigma_device(x[k].data_ptr(), y[k].data_ptr(), 1, s.ndets, jb.FP64, st.cuda_stream)

    if captured:
        graphs = []
        for k in range(6):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[k], stream=streams[k & 1]):
                call(k, streams[k & 1])
        for k in range(6):
            with torch.cuda.stream(streams[k & 1]):
                graphs[k].replay()
    else:
        for k in range(6):
            call(k, streams[k & 1])
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    s.close()
