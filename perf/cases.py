"""The calls that a determinant-CI program makes of this framework, as timed
cases: sigma = H c on device vectors over the range of spaces the engine
takes (CAS(6,6) to FCI(16,16), odd electron counts, partly filled and
truncated spaces), in FP64 and FP32, one vector and several; sigma through
host arrays; a bounded Davidson solve; Dyson orbitals.

A case is a dict: "op" names the call, the space is given by its &general
values, the integrals are the seeded synthetic ones of jayci_b200.synth with
rank = CI orbitals (the shapes of the repository's own workloads).
"""
import itertools
import math

import numpy as np
import torch

import jayci_b200 as jb
from jayci_b200.synth import make_integrals, unpack_integrals

GENERAL = ("electrons", "orbitals", "nfrozen", "ndocc", "nactive", "nfrzvirt", "xlevel")


def _case(name, op, electrons, orbitals, nfrozen=0, ndocc=0, nactive=None, nfrzvirt=0,
          xlevel=0, **more):
    if nactive is None:
        nactive = orbitals - nfrozen - nfrzvirt - ndocc
    c = dict(op=op, electrons=electrons, orbitals=orbitals, nfrozen=nfrozen, ndocc=ndocc,
             nactive=nactive, nfrzvirt=nfrzvirt, xlevel=xlevel, **more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest solves of a geometry scan: 400 determinants, every
        # sigma is launches and latency
        _case("sigma_cas6_6", "sigma", 6, 6, nvec=1, dtype="f64"),
        # an ordinary active space, the size most CASSCF steps use
        _case("sigma_cas10_10", "sigma", 10, 10, nvec=1, dtype="f64"),
        # the 12-orbital workload with its three roots, one call for all (the
        # sigma of a collapse or of start vectors)
        _case("sigma_fci12_12", "sigma", 12, 12, nvec=3, dtype="f64"),
        # the same space in the FP32 phase of a mixed-precision solve
        _case("sigma_fci12_12_f32", "sigma", 12, 12, nvec=1, dtype="f32"),
        # an odd electron count: alpha and beta string spaces differ
        _case("sigma_cas13_13", "sigma", 13, 13, nvec=1, dtype="f64"),
        # two frozen core orbitals, 11.8 million determinants: the space the
        # repository's solves are quoted on, in both precisions
        _case("sigma_fci14_14_fc2", "sigma", 18, 16, nfrozen=2, nvec=1, dtype="f64"),
        _case("sigma_fci14_14_fc2_f32", "sigma", 18, 16, nfrozen=2, nvec=1, dtype="f32"),
        # the benchmark's space: the largest that one GPU solves
        _case("sigma_fci16_16", "sigma", 16, 16, nvec=1, dtype="f64"),
        # a truncated space (9 x 9 occupation groups, excitation level 2):
        # the reference's DOCC / ACTV / VIRT expansions
        _case("sigma_trunc12_16_x2", "sigma", 12, 16, ndocc=2, nactive=10, xlevel=2, nvec=1,
              dtype="f64"),
        # sigma of host arrays (the drop-in call of a program that keeps its
        # vectors in host memory)
        _case("sigma_host_fci12_12", "sigma_host", 12, 12, nvec=1, dtype="f64"),
        # a CASSCF macro-iteration: new integrals, then a bounded number of
        # Davidson iterations on three roots
        _case("davidson_fci12_12", "davidson", 12, 12, nroots=3, iters=48),
        # Dyson orbitals between states of N + 1 and N electrons
        _case("dyson_13_12", "dyson", 13, 12, nstates=2),
    ]


def draw(rng):
    op = rng.choices(("sigma", "sigma_host", "davidson", "dyson"), (8, 1, 2, 1))[0]
    if op == "sigma":
        kind = rng.choices(("cas", "trunc"), (4, 1))[0]
        dtype = rng.choice(("f64", "f64", "f32"))
        nvec = rng.choice((1, 1, 2, 3, 4))
        if kind == "trunc":
            orb = rng.randint(9, 15)
            e = rng.randint(6, 11)
            docc = rng.randint(1, 2)
            actv = rng.randint(max(5, (e + 1) // 2 + 1 - docc), max(6, orb - docc - 2))
            return _case("", "sigma", e, orb, ndocc=docc, nactive=actv,
                         xlevel=rng.choice((1, 2)), nvec=1, dtype=dtype)
        orb = rng.randint(6, 15)
        e = min(max(4, orb + rng.choice((-3, -2, -1, 0, 0, 0, 1, 2))), 2 * orb - 2)
        fc = rng.choice((0, 0, 1, 2))
        return _case("", "sigma", e + 2 * fc, orb + fc, nfrozen=fc, nvec=nvec if orb < 14 else 1,
                     dtype=dtype)
    if op == "sigma_host":
        orb = rng.randint(8, 13)
        return _case("", op, orb + rng.choice((-1, 0, 1)), orb, nvec=rng.choice((1, 2)),
                     dtype="f64")
    if op == "davidson":
        orb = rng.randint(8, 13)
        return _case("", op, orb + rng.choice((-1, 0, 1)), orb, nroots=rng.randint(1, 4),
                     iters=rng.randint(24, 60))
    orb = rng.randint(9, 13)
    return _case("", op, orb + rng.choice((0, 1)), orb, nstates=rng.randint(1, 3))


# ---- what a program keeps -------------------------------------------------

_KEPT = {}  # the spaces of the last case: string tables, device tables and sigma plans


def _space(general):
    """The string space of these &general values.  A program makes it once
    and keeps it for every sigma, solve and geometry."""
    if general not in _KEPT:
        _KEPT[general] = jb.Space(*general)
    return _KEPT[general]


def _general(case, electrons=None):
    g = [case[k] for k in GENERAL]
    if electrons is not None:
        g[0] = electrons
    return tuple(g)


def _norb(case):
    return case["orbitals"] - case["nfrozen"] - case["nfrzvirt"]


def _integrals(case, seed):
    n = _norb(case)
    i = make_integrals(n, n, seed)
    return (*i.packed(), i.e_nuc)


# sigma's integrals belong to the kept space (a solve's vectors change from
# call to call, its integrals do not)
SIGMA_SEED = 104


def _vectors(nvec, ndets, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(nvec, ndets, generator=g, dtype=torch.float64, device="cuda")
    return v / v.norm(dim=1, keepdim=True)


def prepare(case, seed):
    general = _general(case)
    second = _general(case, case["electrons"] - 1) if case["op"] == "dyson" else None
    for g in [g for g in _KEPT if g not in (general, second)]:
        del _KEPT[g]
    known = general in _KEPT
    sp = _space(general)
    st = {"op": case["op"], "space": sp}
    if case["op"] in ("sigma", "sigma_host"):
        if not known:
            m1, m2, enuc = _integrals(case, SIGMA_SEED)
            sp.set_integrals(m1, m2, enuc)
        v = _vectors(case["nvec"], sp.ndets, seed)
        if case["op"] == "sigma_host":
            st["v"] = v.cpu().numpy()
            if not known:
                sp.sigma(st["v"])
            return st
        st["precision"] = jb.FP64 if case["dtype"] == "f64" else jb.FP32
        st["v"] = v if case["dtype"] == "f64" else v.float()
        del v
        st["s"] = torch.zeros_like(st["v"])
        if not known:  # the first call picks the space's plan
            run(st)
            torch.cuda.synchronize()
    elif case["op"] == "davidson":
        st["ints"] = _integrals(case, seed)
        st["opts"] = dict(maxiter=case["iters"], krymin=max(4, case["nroots"]), krymax=20,
                          nroots=case["nroots"], refdim=12, restol=1e-13)
        if not known:
            run(st)
    else:
        st["space1"] = _space(second)
        rng = np.random.default_rng(seed)
        for k, s in (("v0", sp), ("v1", st["space1"])):
            x = rng.standard_normal((case["nstates"], s.ndets))
            st[k] = x / np.linalg.norm(x, axis=1, keepdims=True)
        st["states"] = tuple(range(1, case["nstates"] + 1))
        if not known:
            for s, e in ((sp, 0), (st["space1"], 1)):
                m1, m2, enuc = _integrals(case, SIGMA_SEED + e)
                s.set_integrals(m1, m2, enuc)
            run(st)
    return st


def run(st):
    op, sp = st["op"], st["space"]
    if op == "sigma":
        v, s = st["v"], st["s"]
        sp.sigma_device(v.data_ptr(), s.data_ptr(), v.shape[0], v.shape[1], st["precision"],
                        torch.cuda.current_stream().cuda_stream)
        return s
    if op == "sigma_host":
        return sp.sigma(st["v"])
    if op == "davidson":
        sp.set_integrals(*st["ints"])
        r = sp.davidson(**st["opts"])
        return {"energies": r.energies, "civec": r.civec}
    return jb.dyson(sp, st["space1"], st["v0"], st["v1"], st["states"], st["states"])


# ---- what a pass cannot do without ----------------------------------------

def _strings(case, electrons):
    """Strings of each group (holes in DOCC, electrons in VIRT) of one spin."""
    n, nd, na = _norb(case), case["ndocc"], case["nactive"]
    nv = n - nd - na
    out = {}
    for h in range(min(case["xlevel"], nd) + 1):
        for p in range(min(case["xlevel"], nv) + 1):
            k = electrons - (nd - h) - p
            if 0 <= k <= na:
                out[h, p] = math.comb(nd, h) * math.comb(nv, p) * math.comb(na, k)
    return out


def _counts(case, electrons):
    """(determinants, alpha x beta double replacements of the average
    determinant, same-spin replacements of the average determinant)."""
    e = electrons - 2 * case["nfrozen"]
    ea, eb = (e + 1) // 2, e // 2
    ga, gb, x = _strings(case, ea), _strings(case, eb), case["xlevel"]
    dets = sum(m * k for (h, p), m in ga.items() for (i, q), k in gb.items()
               if h + i <= x and p + q <= x)
    n = _norb(case) - (case["ndocc"] if x == 0 else 0)
    n = n if x else min(n, case["nactive"])
    d = case["ndocc"] if x == 0 else 0
    full = math.comb(n, ea - d) * math.comb(n, eb - d)
    keep = dets / full  # share of a full space's replacements that stay in this one
    oa, ob = ea - d, eb - d
    sa, sb = oa * (n - oa), ob * (n - ob)
    same = sum(o * (n - o) + math.comb(o, 2) * math.comb(n - o, 2) for o in (oa, ob))
    return dets, sa * sb * math.sqrt(keep), same * math.sqrt(keep)


def work(case):
    op = case["op"]
    dets, ab, same = _counts(case, case["electrons"])
    n = _norb(case)
    e = case["electrons"] - 2 * case["nfrozen"]
    oa, ob = (e + 1) // 2, e // 2
    # alpha x beta part as one product per alpha string (singles x the pairs
    # that the beta strings reach), same-spin part one multiply-add an element
    need = min(ab, oa * (n - oa) * (1 + ob + ob * (n - ob))) + same
    if op in ("sigma", "sigma_host"):
        w = 8 if case["dtype"] == "f64" else 4
        return {"bytes": 2.0 * w * dets * case["nvec"], "flops": 2.0 * need * dets * case["nvec"]}
    if op == "davidson":
        m = max(4, case["nroots"])
        it = case["iters"]
        # sigma, and the basis and its sigma read once an iteration
        return {"bytes": 8.0 * dets * it * (2 + 2 * m), "flops": it * 2.0 * dets * (need + 4 * m)}
    dets1 = _counts(case, case["electrons"] - 1)[0]
    k = case["nstates"]
    return {"bytes": 8.0 * k * (dets + dets1), "flops": 2.0 * k * k * dets * max(oa, ob)}


# ---- the same values in 64 bits, by plain torch ----------------------------

def _full_strings(n, k):
    lists = np.array(list(itertools.combinations(range(n), k)), dtype=np.int64).reshape(-1, k)
    masks = (1 << lists).sum(1) if k else np.zeros(1, np.int64)
    return lists, masks.astype(np.int64)


def _replace(masks, p, q):
    """a+_p a_q of every string: (kept strings, their images, signs)."""
    src = np.nonzero((masks >> q) & 1)[0]
    m = masks[src] ^ (1 << q)
    free = ((m >> p) & 1) == 0
    src, m = src[free], m[free]
    lo, hi = min(p, q), max(p, q)
    between = (m & ((1 << hi) - 1)) >> (lo + 1) if hi > lo else m * 0
    par = np.zeros(len(m), np.int64)
    for b in range(hi - lo - 1 if hi > lo else 0):
        par ^= (between >> b) & 1
    order = np.argsort(masks)
    dst = order[np.searchsorted(masks[order], m | (1 << p))]
    return src, dst, 1.0 - 2.0 * par


def _same_spin(masks, h, eri, cuda):
    """Dense same-spin Hamiltonian over all strings of one spin."""
    n, ns = h.shape[0], len(masks)
    E = {}
    for p in range(n):
        for q in range(n):
            s, d, f = _replace(masks, p, q)
            E[p, q] = tuple(torch.as_tensor(x, device=cuda) for x in (s, d, f))
    H = torch.zeros(ns, ns, dtype=torch.float64, device=cuda)
    heff = h - 0.5 * np.einsum("prrq->pq", eri)
    G = torch.zeros(ns, ns, dtype=torch.float64, device=cuda)
    for p in range(n):
        for q in range(n):
            G.zero_()
            for r in range(n):
                for t in range(n):
                    s, d, f = E[r, t]
                    G.view(-1).index_add_(0, d * ns + s, f * (0.5 * eri[p, q, r, t]))
            s, d, f = E[p, q]
            H.index_add_(0, d, G.index_select(0, s) * f[:, None])
            H.view(-1).index_add_(0, d * ns + s, f * heff[p, q])
    return H


def _embed(case, electrons):
    """Positions of the space's determinants among all of
    (alpha string) x (beta string), both in lexical order."""
    n, nd, na, x = _norb(case), case["ndocc"], case["nactive"], case["xlevel"]
    groups, index = [], []
    for k in ((electrons + 1) // 2, electrons // 2):
        lists, masks = _full_strings(n, k)
        h = nd - (lists < nd).sum(1)
        p = (lists >= nd + na).sum(1)
        got = []
        for a in range(min(x, nd) + 1):
            for b in range(min(x, n - nd - na) + 1):
                sel = np.nonzero((h == a) & (p == b))[0]
                if len(sel):
                    got.append((a, b, sel))
        groups.append(got)
        index.append(masks)
    pos, nb = [], len(index[1])
    for a, b, sa in groups[0]:
        for c, d, sb in groups[1]:
            if a + c <= x and b + d <= x:
                pos.append((sa[:, None] * nb + sb[None, :]).reshape(-1))
    return index[0], index[1], np.concatenate(pos)


def _sigma64(case, v):
    cuda = "cuda"
    n = _norb(case)
    m1, m2, _ = _integrals(case, SIGMA_SEED)
    h, eri = unpack_integrals(m1, m2, n)
    ma, mb, pos = _embed(case, case["electrons"] - 2 * case["nfrozen"])
    A, B = len(ma), len(mb)
    whole = len(pos) == A * B
    pos = torch.as_tensor(pos, device=cuda)
    Ha = _same_spin(ma, h, eri, cuda)
    Hb = Ha if A == B and np.array_equal(ma, mb) else _same_spin(mb, h, eri, cuda)
    ea = [[_replace(ma, p, q) for q in range(n)] for p in range(n)]
    out = []
    for k in range(v.shape[0]):
        c = torch.zeros(A * B, dtype=torch.float64, device=cuda)
        c[pos] = v[k].double()
        c = c.view(A, B)
        s = Ha @ c + c @ Hb.T
        for r in range(n):
            for t in range(r + 1):
                y = torch.zeros_like(c)
                for p, q in {(r, t), (t, r)}:
                    src, dst, f = (torch.as_tensor(x, device=cuda) for x in _replace(mb, p, q))
                    y.index_add_(1, dst, c.index_select(1, src) * f[None, :])
                rows, cols, vals = [], [], []
                for p in range(n):
                    for q in range(n):
                        src, dst, f = ea[p][q]
                        rows.append(dst)
                        cols.append(src)
                        vals.append(f * eri[p, q, r, t])
                M = torch.sparse_coo_tensor(
                    torch.as_tensor(np.stack([np.concatenate(rows), np.concatenate(cols)]),
                                    device=cuda),
                    torch.as_tensor(np.concatenate(vals), device=cuda), (A, A)).to_sparse_csr()
                s += M @ y
        out.append(s.view(-1)[pos] if not whole else s.view(-1)[pos].clone())
    return torch.stack(out)


def _dyson64(case, v0, v1):
    """No phase: the reference's sum of v0(I) v1(I - orbital)."""
    n, e = _norb(case), case["electrons"] - 2 * case["nfrozen"]
    spin = 0 if e % 2 else 1
    k = [(e + 1) // 2, e // 2]
    m0 = [_full_strings(n, x)[1] for x in k]
    m1 = list(m0)
    m1[spin] = _full_strings(n, k[spin] - 1)[1]
    order = np.argsort(m1[spin])
    S = case["nstates"]
    x0 = v0.reshape(S, len(m0[0]), len(m0[1]))
    x1 = v1.reshape(S, len(m1[0]), len(m1[1]))
    out = np.zeros((S * S, case["orbitals"]))
    for o in range(n):
        src = np.nonzero((m0[spin] >> o) & 1)[0]
        dst = order[np.searchsorted(m1[spin][order], m0[spin][src] ^ (1 << o))]
        for j in range(S):
            a = x0[j][src] if spin == 0 else x0[j][:, src]
            for i in range(S):
                b = x1[i][dst] if spin == 0 else x1[i][:, dst]
                out[j * S + i, o] = np.sum(a * b)
    return out * math.sqrt(case["electrons"])


def exact(case, seed):
    if case["op"] == "davidson":  # a bounded number of iterations: no closed value
        return None
    if case["op"] == "dyson":
        st = prepare(case, seed)
        return _dyson64(case, st["v0"], st["v1"])
    e = case["electrons"] - 2 * case["nfrozen"]
    n = _norb(case)
    strings = max(math.comb(n, (e + 1) // 2), math.comb(n, e // 2))
    if strings > 13000:  # the dense same-spin Hamiltonians outgrow the card
        return None
    v = _vectors(case["nvec"], _counts(case, case["electrons"])[0], seed)
    s = _sigma64(case, v if case["dtype"] == "f64" else v.float())
    return s.cpu().numpy() if case["op"] == "sigma_host" else s
